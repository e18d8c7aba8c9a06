"""The configurations an untuned context picks (default_cfgs): on both sides
of each line of the rule, along every direction and for one and six
operators, the picked kernel agrees with the oracle on every operator and is
one of the non-persistent ones."""
import numpy as np
import pytest

from conftest import rel_err, seeded_field
from test_gpu_ops import ROUTINES, X, Y, Z

pytestmark = pytest.mark.gpu

PERSISTENT = {6, 7, 8, 9, 10, 11, 12, 13, 15, 17, 18}


# fields of at most 4 MiB, at most 16 MiB and more, in either precision, and
# lines that rule out the first picks (odd chunk counts, long lines)
@pytest.mark.parametrize("shape", [(16, 24, 40), (96, 80, 64), (128, 112, 96), (160, 96, 144), (264, 136, 128),
                                   (64, 1024, 36), (1040, 64, 20)])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_default_picks_match_oracle(oracle, torch_cuda, shape, prec):
    torch = torch_cuda
    from x3div_b200 import Context, to_device, to_host
    ctx = Context(*shape, lengths=(2 * np.pi,) * 3, precision=prec)
    dt = torch.float64 if prec == "f64" else torch.float32
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
        assert ctx.last_kernel() not in PERSISTENT
        for (n, k), o in zip(rows, outs):
            ref = oracle.apply(k, direction, used, d[direction])
            assert rel_err(to_host(o), ref) < tol, (n, shape, prec)
            ctx.apply(ctx.op(n), u, o)
            ctx.sync()
            assert ctx.last_kernel() not in PERSISTENT
            assert rel_err(to_host(o), ref) < tol, (n, shape, prec)
    ctx.close()
