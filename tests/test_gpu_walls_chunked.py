"""The chunked non-periodic solves (linesolve_walls.cu) at the lengths where a
chunk (16 points FP64, 32 FP32), a tile or a launch bound changes, against
the CPU oracle with the bars of test_gpu_bc.py: lines one point around whole
chunks (the last chunk holds one point, or the last two points lie in two
chunks), odd cross extents, lines that leave only the 8-line tiles and lines
that fall back to one thread each."""
import numpy as np
import pytest

from conftest import rel_err, seeded_field

pytestmark = pytest.mark.gpu

LEN = (2.0, 1.5, 3.0)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("direction", [0, 1, 2])
@pytest.mark.parametrize("n", [9, 16, 17, 18, 33, 34, 65, 129, 257, 514, 1030])
@pytest.mark.parametrize("ncl", [(1, 1), (2, 1), (2, 2)])
def test_wall_operators(oracle, torch_cuda, prec, direction, n, ncl):
    torch = torch_cuda
    from x3div_b200 import Context, to_device, to_host
    shape = [13, 9, 18]
    shape[direction] = n
    bc = [0] * 6
    bc[2 * direction:2 * direction + 2] = ncl
    ctx = Context(*shape, lengths=LEN, precision=prec, bc=bc)
    d = (ctx.dx, ctx.dy, ctx.dz)[direction]
    dt_ = torch.float64 if prec == "f64" else torch.float32
    tol = 1e-12 if prec == "f64" else 1e-5
    c = "xyz"[direction]
    u = to_device(seeded_field(shape, 3 + n, lengths=LEN, noise=1e-2), dt_)
    used = to_host(u).astype(np.float64)
    lead = (None,) if direction == 1 else ()
    for npaire, name in ((0, "der" + c), (1, "der" + c + "p")):
        t = torch.full_like(u, float("nan"))
        getattr(ctx, "der" + c)(t, u, ctx.op(name), *lead, *shape)
        ctx.sync()
        assert rel_err(to_host(t), oracle.der_np(direction, used, d, *ncl, npaire)) < tol, (name, n, ncl)
    less = list(shape)
    less[direction] -= 1
    p = to_device(np.asfortranarray(used[tuple(slice(0, k) for k in less)]), dt_)
    stag = [("inter" + c + "vp", "int" + c + "vp", "intvp", u, less, (n, n - 1)),
            ("inter" + c + "pv", "int" + c + "pv", "intpv", p, shape, (n - 1, n))]
    if direction != 1:
        stag.append(("der" + c + "vp", "der" + c + "vp", "dervp", u, less, (n, n - 1)))
    for routine, name, kind, src, out, pair in stag:
        t = torch.full(out[::-1], float("nan"), dtype=dt_, device="cuda")
        ext = list(shape)
        ext[direction:direction + 1] = pair
        getattr(ctx, routine)(t, src, ctx.op(name), *ext)
        ctx.sync()
        want = oracle.stag_np(kind, direction, to_host(src).astype(np.float64), d, *ncl, 1)
        assert rel_err(to_host(t), want) < tol, (routine, n, ncl)
    ctx.close()


def test_fp32_staggered_derivative_rounding(oracle, torch_cuda):
    """The 2-norm error of derxvp between walls on a smooth field with a little
    noise, which varies by less than 1 % from field to field: 4.99e-8, and
    5.54e-8 with the larger product of the backward sweep rounded first (one
    thread a line: 4.70e-8)."""
    torch = torch_cuda
    from x3div_b200 import Context, to_device, to_host
    shape = (256, 33, 64)
    ctx = Context(*shape, lengths=(np.pi, 2 * np.pi, 2 * np.pi), precision="f32", bc=(2, 2, 0, 0, 0, 0))
    errs = []
    for seed in range(3):
        u = to_device(seeded_field(shape, seed, lengths=(2 * np.pi,) * 3, noise=1e-2), torch.float32)
        t = torch.full((64, 33, 255), float("nan"), dtype=torch.float32, device="cuda")
        ctx.derxvp(t, u, ctx.op("derxvp"), 256, 255, 33, 64)
        ctx.sync()
        want = oracle.stag_np("dervp", 0, to_host(u).astype(np.float64), ctx.dx, 2, 2, 1)
        errs.append(float(np.linalg.norm((to_host(t) - want).ravel()) / np.linalg.norm(want.ravel())))
    ctx.close()
    assert np.mean(errs) < 5.2e-8, errs
