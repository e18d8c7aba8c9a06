"""derpv and interpv written as the shifted second output of dervp's and
intervp's solve (shifted_twin): every subset order a work-list can name them
in, on aligned and odd extents, one-chunk lines and short last chunks, along
each direction and through the batch kernel's x output forms, against the
oracle with the bars of test_gpu_ops.py."""
import itertools

import numpy as np
import pytest

from conftest import rel_err, seeded_field

pytestmark = pytest.mark.gpu

NAMES = {0: ("derxvp", "derxpv", "intxvp", "intxpv"), 1: ("deryvp", "derypv", "intyvp", "intypv"),
         2: ("derzvp", "derzpv", "intzvp", "intzpv")}
KINDS = ("dervp", "derpv", "intvp", "intpv")


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(64, 48, 32), (16, 12, 10), (17, 33, 15), (100, 36, 20), (258, 9, 31), (8, 140, 129)])
@pytest.mark.parametrize("cfg", [-1, 0, 6, 12, 14, 19, 20])
def test_work_lists_with_twins(oracle, torch_cuda, shape, prec, cfg):
    torch = torch_cuda
    from x3div_b200 import Context, to_device, to_host
    ctx = Context(*shape, lengths=(2 * np.pi, 1.5, 3.0), precision=prec)
    ctx.set_kernel(cfg)
    u = to_device(seeded_field(shape, seed=sum(shape), noise=1e-2), torch.float64 if prec == "f64" else torch.float32)
    used = to_host(u).astype(np.float64)
    tol = 1e-12 if prec == "f64" else 1e-5
    for d in range(3):
        h = (ctx.dx, ctx.dy, ctx.dz)[d]
        ref = [oracle.apply(k, d, used, h) for k in KINDS]
        for order in ((0, 1), (1, 0), (3, 1, 0, 2), (1, 3), (0, 1, 2, 3, 1), (2, 3, 3)):
            outs = [torch.full_like(u, float("nan")) for _ in order]
            ctx.apply_batch([(ctx.op(NAMES[d][k]), u, o) for k, o in zip(order, outs)])
            ctx.sync()
            for k, o in zip(order, outs):
                assert rel_err(to_host(o), ref[k]) < tol, (d, order, k)
    ctx.close()


def test_an_output_named_twice_keeps_the_last_write(oracle, torch_cuda):
    torch = torch_cuda
    from x3div_b200 import Context, to_device, to_host
    shape = (64, 48, 32)
    ctx = Context(*shape, lengths=(2 * np.pi,) * 3)
    u = to_device(seeded_field(shape, seed=1, noise=1e-2))
    out = torch.full_like(u, float("nan"))
    for d, a, b in itertools.product(range(3), (0, 1), (0, 1)):
        if a == b:
            continue
        ctx.apply_batch([(ctx.op(NAMES[d][a]), u, out), (ctx.op(NAMES[d][b]), u, out)])
        ctx.sync()
        assert rel_err(to_host(out), oracle.apply(KINDS[b], d, to_host(u), (ctx.dx, ctx.dy, ctx.dz)[d])) < 1e-12
    ctx.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("tuned", [False, True])
def test_batch_sweep(oracle, torch_cuda, prec, tuned):
    torch = torch_cuda
    from x3div_b200 import Batch, to_device, to_host
    boxes = [(64, 48, 32), (100, 36, 20), (40, 8, 140), (16, 130, 12)]
    dt = torch.float64 if prec == "f64" else torch.float32
    fields = [[to_device(seeded_field(b, seed=i, noise=1e-2), dt)] for i, b in enumerate(boxes)]
    outs = [[[[torch.full_like(fs[0], float("nan")) for _ in range(6)] for _ in range(3)]] for fs in fields]
    batch = Batch(boxes, precision=prec)
    batch.bind_sweep(fields, outs)
    if tuned:
        batch.autotune()
    batch.run()
    batch.sync()
    tol = 1e-12 if prec == "f64" else 1e-5
    for b, fs, os_ in zip(boxes, fields, outs):
        used = to_host(fs[0]).astype(np.float64)
        for d in range(3):
            for k, kind in enumerate(("der", "der2", "dervp", "derpv", "intvp", "intpv")):
                ref = oracle.apply(kind, d, used, 2 * np.pi / b[d])
                assert rel_err(to_host(os_[0][d][k]), ref) < tol, (b, d, kind)
    batch.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("tuned", [False, True])
def test_batch_jobs_of_one_shape_with_different_twins(oracle, torch_cuda, prec, tuned):
    """Every other field sends the families its caller does not want (derpv
    and interpv) to one dump array per job, so that only the others' solves
    have shifted outputs: jobs of one box shape and direction then differ in
    the operators they solve, and a CTA goes from one kind to the other many
    times over the 24 fields."""
    torch = torch_cuda
    from x3div_b200 import Batch, to_device, to_host
    boxes = [(48, 32, 40), (32, 24, 16)]
    nfields = 24
    dt = torch.float64 if prec == "f64" else torch.float32
    fields = [[to_device(seeded_field(b, seed=100 * i + f, noise=1e-2), dt) for f in range(nfields)]
              for i, b in enumerate(boxes)]
    outs = []
    for fs in fields:
        per_field = []
        for f, u in enumerate(fs):
            per_dir = []
            for _ in range(3):
                row = [torch.full_like(u, float("nan")) for _ in range(6)]
                if f % 2:
                    row[5] = row[3]
                per_dir.append(row)
            per_field.append(per_dir)
        outs.append(per_field)
    batch = Batch(boxes, precision=prec)
    batch.bind_sweep(fields, outs)
    if tuned:
        batch.autotune()
    batch.run()
    batch.sync()
    tol = 1e-12 if prec == "f64" else 1e-5
    for b, fs, os_ in zip(boxes, fields, outs):
        for f, u in enumerate(fs):
            used = to_host(u).astype(np.float64)
            for d in range(3):
                for k, kind in enumerate(("der", "der2", "dervp", "derpv", "intvp", "intpv")):
                    if f % 2 and k in (3, 5):
                        continue
                    ref = oracle.apply(kind, d, used, 2 * np.pi / b[d])
                    assert rel_err(to_host(os_[f][d][k]), ref) < tol, (b, f, d, kind)
    batch.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("tuned", [False, True])
@pytest.mark.parametrize("nops", [1, 3, 4, 5])
def test_batch_of_fewer_families(oracle, torch_cuda, prec, nops, tuned):
    """Lists without a twin run the batch kernel without the shifted outputs
    (1 and 3 families), lists with one the kernel with them."""
    torch = torch_cuda
    from x3div_b200 import Batch, to_device, to_host
    boxes = [(64, 48, 32), (100, 36, 20), (40, 8, 140)]
    dt = torch.float64 if prec == "f64" else torch.float32
    fields = [[to_device(seeded_field(b, seed=i, noise=1e-2), dt)] for i, b in enumerate(boxes)]
    outs = [[[[torch.full_like(fs[0], float("nan")) for _ in range(6)] for _ in range(3)]] for fs in fields]
    batch = Batch(boxes, precision=prec)
    batch.bind_sweep(fields, outs, nops)
    if tuned:
        batch.autotune()
    batch.run()
    batch.sync()
    tol = 1e-12 if prec == "f64" else 1e-5
    for b, fs, os_ in zip(boxes, fields, outs):
        used = to_host(fs[0]).astype(np.float64)
        for d in range(3):
            for k, kind in enumerate(("der", "der2", "dervp", "derpv", "intvp", "intpv")):
                got = to_host(os_[0][d][k])
                if k < nops:
                    assert rel_err(got, oracle.apply(kind, d, used, 2 * np.pi / b[d])) < tol, (b, d, kind)
                else:
                    assert np.isnan(got).all()
    batch.close()
