"""The configurations an untuned context picks (default_cfgs): fields on both
sides of the rule's 24 MiB line in either precision, small ones where the wave
model decides, lines that rule out the first picks (odd chunk counts, long
lines); plain programs of one and six operators and the fused stages, which
accumulate, take several inputs or an FP64 one.  The picked kernel agrees with
the oracle and is one of the non-persistent ones, and above the line it is the
one the rule names."""
import numpy as np
import pytest

from conftest import rel_err, seeded_field
from test_gpu_ops import ROUTINES, X, Y, Z

pytestmark = pytest.mark.gpu

PERSISTENT = {6, 7, 8, 9, 10, 11, 12, 13, 15, 17, 18}
LARGE = 24 << 20  # bytes of a field above which the order of configurations is fixed

SMALL_F64 = [(16, 24, 40), (96, 80, 64), (128, 112, 96), (64, 1024, 36), (1040, 64, 20), (160, 128, 153)]
LARGE_F64 = [(160, 128, 154), (256, 128, 128)]
SMALL_F32 = [(16, 24, 40), (96, 80, 64), (160, 96, 144), (64, 1024, 36), (1040, 64, 20), (184, 184, 184)]
LARGE_F32 = [(184, 184, 186), (192, 192, 192)]
BOXES = [("f64", s) for s in SMALL_F64 + LARGE_F64] + [("f32", s) for s in SMALL_F32 + LARGE_F32]


def _large(prec, shape):
    return shape[0] * shape[1] * shape[2] * (4 if prec == "f32" else 8) > LARGE


def test_boxes_lie_on_their_side_of_the_line():
    assert not any(_large("f64", s) for s in SMALL_F64) and all(_large("f64", s) for s in LARGE_F64)
    assert not any(_large("f32", s) for s in SMALL_F32) and all(_large("f32", s) for s in LARGE_F32)


def _context(torch, prec, shape):
    from x3div_b200 import Context
    return (Context(*shape, lengths=(2 * np.pi,) * 3, precision=prec),
            torch.float64 if prec == "f64" else torch.float32)


@pytest.mark.parametrize("prec,shape", BOXES)
def test_default_picks_match_oracle(oracle, torch_cuda, shape, prec):
    torch = torch_cuda
    from x3div_b200 import to_device, to_host
    ctx, dt = _context(torch, prec, shape)
    u = to_device(seeded_field(shape, seed=sum(shape), noise=1e-2), dt)
    used = to_host(u).astype(np.float64)
    d = {X: ctx.dx, Y: ctx.dy, Z: ctx.dz}
    tol = 1e-12 if prec == "f64" else 1e-5
    for direction in (X, Y, Z):
        rows = [(n, k) for _, n, k, dd, _ in ROUTINES if dd == direction and not n.endswith("p")]
        rows = [r for r in rows if r[0] not in ("derxp", "deryp", "derzp")][:6]
        outs = [torch.full_like(u, float("nan")) for _ in rows]
        ctx.apply_batch([(ctx.op(n), u, o) for (n, _), o in zip(rows, outs)])
        ctx.sync()
        picked = {ctx.last_kernel()}
        refs = [oracle.apply(k, direction, used, d[direction]) for _, k in rows]
        for (n, _), o, ref in zip(rows, outs, refs):
            assert rel_err(to_host(o), ref) < tol, (n, shape, prec)
            ctx.apply(ctx.op(n), u, o)
            ctx.sync()
            picked.add(ctx.last_kernel())
            assert rel_err(to_host(o), ref) < tol, (n, shape, prec)
        assert not picked & PERSISTENT
        if _large(prec, shape):  # their chunk counts suit 19 or, where odd multiples of 2, only 20
            assert picked <= {19, 20}, (direction, picked)
    ctx.close()


@pytest.mark.parametrize("prec,shape", [b for b in BOXES if max(b[1]) < 300] + [("f32", (32, 112, 256))])
def test_default_picks_of_the_stages(oracle, torch_cuda, shape, prec):
    torch = torch_cuda
    from x3div_b200 import to_device, to_host
    ctx, dt = _context(torch, prec, shape)
    tol = 1e-12 if prec == "f64" else 1e-4
    u = [to_device(seeded_field(shape, s, noise=1e-2), dt) for s in (1, 2, 3)]
    uh = [to_host(a).astype(np.float64) for a in u]
    h = (ctx.dx, ctx.dy, ctx.dz)
    p = torch.empty(shape[::-1], dtype=torch.float64, device="cuda")
    g, du = ([torch.empty_like(u[0]) for _ in range(3)] for _ in range(2))
    last = {}
    ctx.momentum_rhs_eq(*du, *u)  # its last launch: six accumulated operators along z
    last["transeq_z"] = ctx.last_kernel()
    ctx.divergence(p, *u)  # two accumulated ones along z, FP64 out
    last["div_z"] = ctx.last_kernel()
    ph = seeded_field(shape, 30, kind="rand", noise=0)
    ctx.gradp(*g, to_device(ph))  # three plain ones on three inputs along x
    last["gradp_x"] = ctx.last_kernel()
    ctx.sync()
    for got, want in zip([p] + du, [oracle.divergence(*uh, *h)] + list(oracle.momentum_rhs(*uh, *h))):
        assert rel_err(to_host(got), want) < tol
    for got, want in zip(g, oracle.gradp(ph, *h)):
        assert rel_err(to_host(got), want) < tol
    assert not set(last.values()) & PERSISTENT, last
    if _large(prec, shape):
        assert last["transeq_z"] == (14 if prec == "f32" else 0), last
        assert last["div_z"] == 0, last
        assert last["gradp_x"] in ((5, 19) if prec == "f32" else (19, 20)), last
    if shape == (32, 112, 256):  # the packed pairs with FP64 output
        assert last["div_z"] == 14, last
    ctx.close()
