"""The chunked stage kernels on grids whose rows are not whole 16-byte units
and on fields at unaligned addresses (linesolve_any.cu), against the CPU
oracle with the bars of test_gpu_ops.py: tiles with a partial last column or
row, lines one point around a multiple of the chunk (16 points FP64, 32
FP32), an odd number of chunks, lines that need more than 256 threads a
tile, and lines that leave only the 8-line tiles."""
import numpy as np
import pytest

from conftest import rel_err, seeded_field
from test_gpu_ops import ROUTINES, X, Y, Z, call

pytestmark = pytest.mark.gpu

LEN = (2 * np.pi, 1.5, 3.0)


def _all_routines(oracle, ctx, u_d, make_out, shape, prec):
    from x3div_b200 import to_host
    used = to_host(u_d).astype(np.float64)
    d = {X: ctx.dx, Y: ctx.dy, Z: ctx.dz}
    tol = 1e-12 if prec == "f64" else 1e-5
    for routine, opname, kind, direction, style in ROUTINES:
        t_d = make_out()
        call(ctx, routine, style, t_d, u_d, ctx.op(opname), shape)
        ctx.sync()
        assert ctx.last_kernel() in (0, 3), (routine, ctx.last_kernel())
        err = rel_err(to_host(t_d), oracle.apply(kind, direction, used, d[direction]))
        assert err < tol, (routine, opname, shape, prec, err)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(17, 33, 31), (33, 16, 65), (49, 97, 32), (15, 300, 10), (271, 9, 12),
                                   (9, 12, 1000), (1001, 8, 9)])
def test_routines_on_odd_extents(oracle, torch_cuda, shape, prec):
    torch = torch_cuda
    from x3div_b200 import Context, to_device
    ctx = Context(*shape, lengths=LEN, precision=prec)
    u_d = to_device(seeded_field(shape, seed=sum(shape), noise=1e-2), torch.float64 if prec == "f64" else torch.float32)
    _all_routines(oracle, ctx, u_d, lambda: torch.full_like(u_d, float("nan")), shape, prec)
    ctx.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_routines_on_unaligned_fields(oracle, torch_cuda, prec):
    """Input and output one element into their allocations."""
    torch = torch_cuda
    from x3div_b200 import Context, to_device
    shape = (32, 24, 40)
    ctx = Context(*shape, lengths=LEN, precision=prec)
    u = to_device(seeded_field(shape, seed=5, noise=1e-2), torch.float64 if prec == "f64" else torch.float32)

    def shifted():
        return torch.full((u.numel() + 1,), float("nan"), dtype=u.dtype, device="cuda")[1:].view(u.shape)

    u_d = shifted()
    u_d.copy_(u)
    _all_routines(oracle, ctx, u_d, shifted, shape, prec)
    ctx.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(17, 12, 10), (34, 33, 18), (45, 16, 33), (9, 290, 12)])
def test_stages_on_odd_extents(oracle, torch_cuda, shape, prec):
    """divergence, gradp, momentum_rhs_eq and an Euler step in three fused
    launches a stage, with the bars of test_gpu_stages.py (FP32: an
    interpolation alone is about 6e-6 and a stage chains three operators)."""
    torch = torch_cuda
    from x3div_b200 import Context, to_device, to_host
    ctx = Context(*shape, lengths=LEN, precision=prec)
    dt_ = torch.float64 if prec == "f64" else torch.float32
    tol = 1e-12 if prec == "f64" else 1e-4
    u = [to_device(seeded_field(shape, s, lengths=LEN, noise=1e-2), dt_) for s in (1, 2, 3)]
    uh = [to_host(a).astype(np.float64) for a in u]
    h = (ctx.dx, ctx.dy, ctx.dz)
    p = torch.empty(shape[::-1], dtype=torch.float64, device="cuda")
    n0 = ctx.launch_count()
    ctx.divergence(p, *u)
    assert ctx.launch_count() - n0 == 3
    assert rel_err(to_host(p), oracle.divergence(*uh, *h)) < tol
    ph = seeded_field(shape, 30, kind="rand", lengths=LEN, noise=0)
    pd = to_device(ph)
    g, du = ([torch.empty_like(u[0]) for _ in range(3)] for _ in range(2))
    ctx.gradp(*g, pd)
    assert ctx.launch_count() - n0 == 6
    ctx.momentum_rhs_eq(*du, *u)
    assert ctx.launch_count() - n0 == 9
    ctx.sync()
    for got, want in zip(g, oracle.gradp(ph, *h)):
        assert rel_err(to_host(got), want) < tol
    for got, want in zip(du, oracle.momentum_rhs(*uh, *h)):
        assert rel_err(to_host(got), want) < tol
    ctx.euler_step(*u, *du, p, *g, 1e-3)
    ctx.sync()
    oracle.euler_step(*uh, 1e-3, lengths=LEN)
    # the divergence carries the unit roundoff times the interpolation's
    # condition (99) times the largest wavenumber (2 / h), and the projection
    # divides it by the smallest one (2 pi / L): on (9, 290, 12) the cells are
    # a hundred times flatter than long, and FP32 gives 2.3e-3
    bound = 99 * 2 / min(h) * max(LEN) / (2 * np.pi) * (2.0**-53 if prec == "f64" else 2.0**-24)
    for got, want in zip(u, uh):
        assert rel_err(to_host(got), want) < max(bound, 1e-11 if prec == "f64" else 1e-4)
    ctx.close()


# (32, 112, 256) is an extent whose divergence along z an untuned FP32 context
# solves in packed pairs (configuration 14), which store the FP64 result two
# points at a time
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape,cfg", [((32, 112, 256), -1), ((64, 24, 32), 12), ((64, 24, 32), 14),
                                       ((64, 24, 32), 15), ((64, 24, 32), -1)])
@pytest.mark.parametrize("off_u,off_p", [(0, 1), (1, 0), (1, 1)])
def test_stages_on_unaligned_fields(oracle, torch_cuda, shape, cfg, prec, off_u, off_p):
    """The velocity and its work arrays off_u, the FP64 pressure off_p
    elements into their allocations."""
    torch = torch_cuda
    from x3div_b200 import Context, to_device, to_host
    ctx = Context(*shape, lengths=LEN, precision=prec)
    ctx.set_kernel(cfg)
    dt_ = torch.float64 if prec == "f64" else torch.float32
    tol = 1e-12 if prec == "f64" else 1e-4

    def new(dtype, off):
        n = shape[0] * shape[1] * shape[2]
        return torch.full((n + off,), float("nan"), dtype=dtype, device="cuda")[off:].view(shape[::-1])

    u = [new(dt_, off_u).copy_(to_device(seeded_field(shape, s, lengths=LEN, noise=1e-2), dt_)) for s in (1, 2, 3)]
    uh = [to_host(a).astype(np.float64) for a in u]
    h = (ctx.dx, ctx.dy, ctx.dz)
    p = new(torch.float64, off_p)
    g, du = ([new(dt_, off_u) for _ in range(3)] for _ in range(2))
    ctx.divergence(p, *u)
    ctx.momentum_rhs_eq(*du, *u)
    ctx.sync()
    assert rel_err(to_host(p), oracle.divergence(*uh, *h)) < tol
    for got, want in zip(du, oracle.momentum_rhs(*uh, *h)):
        assert rel_err(to_host(got), want) < tol
    ph = seeded_field(shape, 30, kind="rand", lengths=LEN, noise=0)
    p.copy_(to_device(ph))
    ctx.gradp(*g, p)
    ctx.sync()
    for got, want in zip(g, oracle.gradp(ph, *h)):
        assert rel_err(to_host(got), want) < tol
    ctx.close()


# an extent of own x transforms, one of cuFFT's (x, y) plane and fused z
# transforms, and one of its 3-D transform
@pytest.mark.parametrize("shape", [(32, 20, 16), (20, 12, 24), (18, 12, 10)])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_pressure_one_element_into_its_allocation(oracle, torch_cuda, shape, prec):
    """The periodic solve alone, inside a step and inside a captured step."""
    torch = torch_cuda
    from x3div_b200 import Context, X3DError, to_device, to_host
    stream = torch.cuda.Stream()
    ctx = Context(*shape, lengths=LEN, precision=prec, stream=stream)
    dt_ = torch.float64 if prec == "f64" else torch.float32
    n = shape[0] * shape[1] * shape[2]

    def new(off):
        return torch.full((n + off,), float("nan"), dtype=torch.float64, device="cuda")[off:].view(shape[::-1])

    rhs = seeded_field(shape, 21, kind="rand", lengths=LEN, noise=0)
    p = new(1).copy_(to_device(rhs))
    torch.cuda.synchronize()
    ctx.poisson(p)
    ctx.sync()
    assert rel_err(to_host(p), oracle.poisson(rhs, *LEN)) < 1e-12
    u0 = [to_device(seeded_field(shape, s, lengths=LEN, noise=1e-2), dt_) for s in (1, 2, 3)]
    uh = [to_host(a).astype(np.float64) for a in u0]
    bound = 99 * 2 / min(ctx.dx, ctx.dy, ctx.dz) * max(LEN) / (2 * np.pi) * (2.0**-53 if prec == "f64" else 2.0**-24)

    def state():
        u = [a.clone() for a in u0]
        return u, [torch.empty_like(a) for a in u], new(1), [torch.empty_like(a) for a in u]

    eager, captured = state(), state()
    torch.cuda.synchronize()
    u, du, q, g = eager
    ctx.euler_step(*u, *du, q, *g, 1e-3)
    ctx.close()
    ctx = Context(*shape, lengths=LEN, precision=prec, stream=stream)  # nothing allocated yet
    u, du, q, g = captured
    ctx.step_capture(*u, *du, q, *g, 1e-3)
    ctx.step_launch()
    ctx.sync()
    assert torch.equal(eager[2], captured[2])
    for a, b in zip(eager[0] + eager[3], captured[0] + captured[3]):
        assert torch.equal(a, b)
    oracle.euler_step(*uh, 1e-3, lengths=LEN)
    for a, want in zip(u, uh):  # the bound of test_stages_on_odd_extents
        assert rel_err(to_host(a), want) < max(bound, 1e-11 if prec == "f64" else 1e-4)
    with pytest.raises(X3DError):  # a complex array has no such address
        ctx.poisson_zpencil(new(1), 1, 0, 1, 0)
    ctx.close()


# x_tile_lines: 8 lines a tile, 16, and (FP32) 32
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(17, 12, 10), (17, 160, 130), (17, 300, 260), (33, 20, 30), (9, 130, 150)])
def test_short_x_lines(oracle, torch_cuda, shape, prec):
    """Periodic and walled x operators on lines of one or two chunks."""
    torch = torch_cuda
    from x3div_b200 import Context, to_device, to_host
    dt_ = torch.float64 if prec == "f64" else torch.float32
    tol = 1e-12 if prec == "f64" else 1e-5
    u = to_device(seeded_field(shape, 3, lengths=LEN, noise=1e-2), dt_)
    used = to_host(u).astype(np.float64)
    ctx = Context(*shape, lengths=LEN, precision=prec)
    names = [("derx", "der"), ("derxx", "der2"), ("derxvp", "dervp"), ("derxpv", "derpv"), ("intxvp", "intvp"),
             ("intxpv", "intpv")]
    outs = [torch.full_like(u, float("nan")) for _ in names]
    one = torch.full_like(u, float("nan"))
    ctx.apply_batch([(ctx.op(n), u, o) for (n, _), o in zip(names, outs)])
    ctx.derx(one, u, ctx.op("derx"), *shape)
    ctx.sync()
    for (_, kind), o in zip(names, outs):
        assert rel_err(to_host(o), oracle.apply(kind, X, used, ctx.dx)) < tol, kind
    assert rel_err(to_host(one), oracle.apply("der", X, used, ctx.dx)) < tol
    ctx.close()
    n = shape[0]
    ctx = Context(*shape, lengths=LEN, precision=prec, bc=(2, 1, 0, 0, 0, 0))
    t = torch.full_like(u, float("nan"))
    ctx.derx(t, u, ctx.op("derx"), *shape)
    s = torch.full((shape[2], shape[1], n - 1), float("nan"), dtype=dt_, device="cuda")
    ctx.interxvp(s, u, ctx.op("intxvp"), n, n - 1, *shape[1:])
    ctx.sync()
    assert rel_err(to_host(t), oracle.der_np(X, used, ctx.dx, 2, 1, 0)) < tol
    assert rel_err(to_host(s), oracle.stag_np("intvp", X, used, ctx.dx, 2, 1, 1)) < tol
    ctx.close()
