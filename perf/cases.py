"""The work a program has this library do, as measurable cases.

A case is a dict of plain values with a `family`:

  operator  one routine of x3d_derive or x3d_staggered on one field, the
            smallest call a driver makes (test=1 style checks, post-processing);
  sweep     every operator family along every direction on one field, as one
            work-list (x3d_apply_batch): the derivative benchmark;
  walls     the non-periodic branches: first derivatives of both parities and
            the staggered interpolations and derivatives along walled
            directions, one routine call each, as the channel (Dirichlet y)
            and free-slip Taylor-Green set-ups need them;
  boxes     many independent uneven boxes in one persistent launch (Batch);
  poisson   the spectral pressure solve in place, periodic or with walls;
  step      one Euler step from a kept velocity: the whole time loop body, as
            one call (`calls` false) or as the reference driver's sequence of
            routines (`calls` true).

`tuned` cases call x3d_autotune once per box, as the benchmark does and the
integration notes advise for long runs; the others use the library as created.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from x3div_b200 import Batch, Context

TWO_PI = 2.0 * math.pi
KINDS = ("der", "der2", "dervp", "derpv", "intvp", "intpv")
PERIODIC = (0, 0, 0, 0, 0, 0)

# (operator instance, kind) per direction, in the order of the derivative sweep
SWEEP = [[("derx", "der"), ("derxx", "der2"), ("derxvp", "dervp"), ("derxpv", "derpv"), ("intxvp", "intvp"),
          ("intxpv", "intpv")],
         [("dery", "der"), ("deryy", "der2"), ("deryvp", "dervp"), ("derypv", "derpv"), ("intyvp", "intvp"),
          ("intypv", "intpv")],
         [("derz", "der"), ("derzz", "der2"), ("derzvp", "dervp"), ("derzpv", "derpv"), ("intzvp", "intvp"),
          ("intzpv", "intpv")]]

# box shapes of the batching workload
BOX_SHAPES = [(96, 96, 96), (128, 256, 64), (200, 100, 150), (256, 256, 256), (64, 512, 64)]


def listed():
    def case(name, family, shape, precision, **more):
        c = dict(name=name, family=family, nx=shape[0], ny=shape[1], nz=shape[2], precision=precision, bc="000000",
                 tuned=False)
        c.update(more)
        return c

    return [
        # one derivative of the 64^3 box of the reference's own run
        case("operator_64_f64", "operator", (64, 64, 64), "f64", direction=1, kind="der"),
        # the reference's run itself: 64^3, FP64, the driver's routines one by one
        case("step_64_f64", "step", (64, 64, 64), "f64", calls=True),
        # the derivative benchmark, FP32-mixed and FP64
        case("sweep_512_f32", "sweep", (512, 512, 512), "f32", tuned=True),
        case("sweep_384_f64", "sweep", (384, 384, 384), "f64", tuned=True),
        # boxes whose x extent is odd, or gives rows that are not whole 16 bytes
        case("sweep_odd_f64", "sweep", (171, 129, 150), "f64"),
        case("sweep_odd_f32", "sweep", (250, 171, 129), "f32"),
        # channel flow: walls along y; free-slip walls all round
        case("walls_channel_f64", "walls", (256, 129, 128), "f64", bc="002200"),
        case("walls_slip_f32", "walls", (193, 193, 193), "f32", bc="111111"),
        # eight of the batching workload's boxes
        case("boxes_f32", "boxes", (8, 0, 0), "f32", pick=48),
        # the pressure solve at the benchmark's size, and in a channel (walls along y)
        case("poisson_512", "poisson", (512, 512, 512), "f64"),
        case("poisson_channel", "poisson", (256, 129, 128), "f64", bc="001100"),
        # the time step of the benchmark
        case("step_512_f32", "step", (512, 512, 512), "f32", tuned=True, calls=False),
    ]


def _size(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    family = rng.choice(["operator", "sweep", "sweep", "walls", "boxes", "poisson", "step"])
    precision = rng.choice(["f64", "f32"])
    c = dict(family=family, precision=precision, bc="000000", tuned=False)
    if family == "boxes":
        c.update(nx=rng.randint(3, 12), ny=0, nz=0, pick=rng.randint(1, 1 << 30))
        return c
    # three sizes of the whole range; half the draws snap to a multiple of 8
    high = {"operator": 200, "sweep": 320, "walls": 220, "poisson": 320, "step": 320}[family]
    shape = [_size(rng, 16, high) for _ in range(3)]
    if family in ("poisson", "step"):  # boxes of equal sides: cells not far from cubes
        n = _size(rng, 16, 200)
        shape = [max(16, round(n * rng.uniform(0.6, 1.6))) for _ in range(3)]
    if rng.random() < 0.5:
        shape = [max(16, n // 8 * 8) for n in shape]
    if family == "operator":
        c.update(direction=rng.randrange(3), kind=rng.choice(KINDS))
    elif family == "walls":
        c["bc"] = rng.choice(["002200", "111111", "220000", "000011", "121212", "001100"])
    elif family == "poisson":
        c["precision"] = "f64"
        c["bc"] = rng.choice(["000000", "000000", "001100", "220000", "111111"])
        if c["bc"] == "111111":
            shape = [max(16, n // 2) for n in shape]
    elif family == "step":
        c.update(calls=rng.random() < 0.5, tuned=rng.random() < 0.3)
    elif family == "sweep":
        c["tuned"] = rng.random() < 0.3
    c.update(nx=shape[0], ny=shape[1], nz=shape[2])
    return c


# ---- geometry ---------------------------------------------------------------


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _bc(case):
    return tuple(int(ch) for ch in case["bc"])


def _walled(case, d):
    return _bc(case)[2 * d] != 0


def _lengths(case):
    # 2 pi, and pi between walls: the lowest mode of either has wavenumber 1
    return tuple(math.pi if _walled(case, d) else TWO_PI for d in range(3))


def _spacing(case, d):
    n = _shape(case)[d]
    return _lengths(case)[d] / (n - 1 if _walled(case, d) else n)


def _dtype(case):
    return torch.float32 if case["precision"] == "f32" else torch.float64


def _boxes(case):
    rng = np.random.default_rng(case["pick"])
    return [BOX_SHAPES[i] for i in rng.integers(0, len(BOX_SHAPES), size=case["nx"])]


# ---- inputs -----------------------------------------------------------------


def _noise(gen, shape, amplitude):
    return amplitude * torch.randn(shape[::-1], generator=gen, device="cuda", dtype=torch.float64)


def _velocity(case, shape, seed):
    """Taylor-Green velocity plus Gaussian noise, (nz, ny, nx) FP64 tensors."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nx, ny, nz = shape
    ax = [torch.arange(n, device="cuda", dtype=torch.float64) * (TWO_PI / n) for n in (nx, ny, nz)]
    x, y, z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    u = torch.sin(x) * torch.cos(y) * torch.cos(z) + _noise(gen, shape, 1e-2)
    v = -torch.cos(x) * torch.sin(y) * torch.cos(z) + _noise(gen, shape, 1e-2)
    w = _noise(gen, shape, 1e-2)
    return [a.to(_dtype(case)).contiguous() for a in (u, v, w)]


_kept = {}


def _context(case):
    """The program's context for this box (tuned where the case says so): made
    once and used for every set of fields, as a time loop does."""
    key = (_shape(case), case["precision"], case["bc"], case["tuned"])
    if key not in _kept:
        for old in _kept.values():
            old.close()
        _kept.clear()
        ctx = Context(*_shape(case), lengths=_lengths(case), precision=case["precision"],
                      bc=None if _bc(case) == PERIODIC else _bc(case))
        if case["tuned"]:
            ctx.autotune(6)
        _kept[key] = ctx
    return _kept[key]


def _wall_calls(case):
    """(routine, operator instance, kind, npaire, direction) of the walled directions."""
    out = []
    for d in range(3):
        if not _walled(case, d):
            continue
        c = "xyz"[d]
        out += [("der" + c, "der" + c, "der", 0, d), ("der" + c, "der" + c + "p", "der", 1, d),
                ("inter" + c + "vp", "int" + c + "vp", "intvp", 1, d),
                ("inter" + c + "pv", "int" + c + "pv", "intpv", 1, d)]
        if d != 1:
            out.append(("der" + c + "vp", "der" + c + "vp", "dervp", 1, d))
    return out


def _grid(shape, d, less):
    s = list(shape)
    s[d] -= less
    return s


def _empty(case, shape):
    return torch.empty(tuple(shape)[::-1], dtype=_dtype(case), device="cuda")


def prepare(case, seed):
    shape = _shape(case)
    family = case["family"]
    if family == "boxes":
        boxes = _boxes(case)
        fields = [_velocity(case, b, seed + 1000 * i) for i, b in enumerate(boxes)]
        # one array of outputs per box: [field][direction][operator family]
        outs = [torch.empty((3, 3, 6) + b[::-1], dtype=_dtype(case), device="cuda") for b in boxes]
        batch = Batch(boxes, precision=case["precision"])
        batch.bind_sweep(fields, outs)
        return dict(case=case, batch=batch, fields=fields, outs=outs)
    ctx = _context(case)
    st = dict(case=case, ctx=ctx)
    if family == "poisson":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        ps = [n - 1 if _walled(case, d) else n for d, n in enumerate(shape)]
        st["p"] = _noise(gen, ps, 1.0)
        return st
    vel = _velocity(case, shape, seed)
    if family == "operator":
        st.update(u=vel[0], out=torch.empty_like(vel[0]))
    elif family == "sweep":
        u = vel[0]
        outs = [torch.empty_like(u) for _ in range(18)]
        ops = [ctx.op(name) for row in SWEEP for name, _ in row]
        st.update(u=u, outs=outs, items=[(op, u, o) for op, o in zip(ops, outs)])
    elif family == "walls":
        calls = _wall_calls(case)
        # the velocity on the velocity grid, and on each walled direction's pressure grid
        pv = {d: vel[2].narrow(2 - d, 0, shape[d] - 1).contiguous() for d in range(3) if _walled(case, d)}
        outs = []
        for _, _, kind, _, d in calls:
            outs.append(_empty(case, _grid(shape, d, 1 if kind.endswith("vp") else 0)))
        st.update(u=vel[0], pv=pv, outs=outs, calls=[(c, ctx.op(c[1])) for c in calls])
    else:  # step
        new = lambda: [torch.empty_like(vel[0]) for _ in range(3)]  # noqa: E731
        st.update(u0=vel, u=new(), du=new(), g=new(),
                  p=torch.empty(shape[::-1], dtype=torch.float64, device="cuda"))
    return st


STEP_DT = 1e-3


def _operator(ctx, direction, kind, out, u, shape):
    nx, ny, nz = shape
    c = "xyz"[direction]
    if kind in ("der", "der2"):
        name = "der" + c * (2 if kind == "der2" else 1)
        args = (None, nx, ny, nz) if name == "dery" else (nx, ny, nz)
        getattr(ctx, name)(out, u, ctx.op(name), *args)
        return
    stag = ("der" if kind.startswith("der") else "inter") + c + kind[-2:]
    op = ctx.op(("der" if kind.startswith("der") else "int") + c + kind[-2:])
    ext = [nx, ny, nz]
    ext.insert(direction, shape[direction])
    lead = (None,) if stag in ("deryvp", "derypv") else ()
    getattr(ctx, stag)(out, u, op, *lead, *ext)


def _wall_call(ctx, call, op, u, pv, out, shape):
    routine, _, kind, _, d = call
    nx, ny, nz = shape
    if kind == "der":
        lead = (None,) if d == 1 else ()
        getattr(ctx, routine)(out, u, op, *lead, nx, ny, nz)
        return
    n = shape[d]
    pair = (n, n - 1) if kind.endswith("vp") else (n - 1, n)
    ext = [nx, ny, nz]
    ext[d:d + 1] = pair
    getattr(ctx, routine)(out, u if kind.endswith("vp") else pv[d], op, *ext)


def run(state):
    case = state["case"]
    family = case["family"]
    if family == "boxes":
        state["batch"].run()
        return state["outs"]
    ctx = state["ctx"]
    if family == "operator":
        _operator(ctx, case["direction"], case["kind"], state["out"], state["u"], _shape(case))
        return state["out"]
    if family == "sweep":
        ctx.apply_batch(state["items"])
        return state["outs"]
    if family == "walls":
        for (call, op), out in zip(state["calls"], state["outs"]):
            _wall_call(ctx, call, op, state["u"], state["pv"], out, _shape(case))
        return state["outs"]
    if family == "poisson":
        ctx.poisson(state["p"])
        return state["p"]
    u, du, g, p = state["u"], state["du"], state["g"], state["p"]
    for a, b in zip(u, state["u0"]):
        a.copy_(b)
    if case["calls"]:
        ctx.momentum_rhs_eq(*du, *u)
        ctx.int_time(*u, *du, STEP_DT)
        ctx.solve_poisson(p, *g, *u)
        ctx.cor_vel(*u, *g)
    else:
        ctx.euler_step(*u, *du, p, *g, STEP_DT)
    return dict(u=u, du=du, p=p, g=g)


def work(case):
    es = 4 if case["precision"] == "f32" else 8
    family = case["family"]
    if family == "boxes":
        pts = sum(a * b * c for a, b, c in _boxes(case))
        return dict(bytes=pts * 3 * 19 * es, flops=pts * 54 * 12)
    n = case["nx"] * case["ny"] * case["nz"]
    if family == "operator":
        return dict(bytes=2 * n * es, flops=12 * n)
    if family == "sweep":
        return dict(bytes=19 * n * es, flops=18 * 12 * n)
    if family == "walls":
        calls = len(_wall_calls(case))
        walls = sum(_walled(case, d) for d in range(3))
        return dict(bytes=(calls + 1 + walls) * n * es, flops=12 * calls * n)
    if family == "poisson":
        return dict(bytes=16 * n, flops=5.0 * n * math.log2(n))
    return dict(bytes=(12 * es + 8) * n, flops=(18 + 16) * 12 * n + 5.0 * n * math.log2(n))


def tolerance(case):
    """Several times the error measured against `exact` (largest over the
    outputs): the interpolations divide by 1 + 0.98 cos w, which lifts the
    unit roundoff about a hundredfold, and a step's pressure starts from the
    divergence, a difference of interpolated fields."""
    f32 = case["precision"] == "f32"
    family = case["family"]
    if family == "step":
        return dict(rel=1e-3 if f32 else 4e-12)
    if family == "poisson":
        return dict(rel=4e-14)
    return dict(rel=5e-6 if f32 else 4e-14)


# ---- 64-bit results in plain torch --------------------------------------------


def _scalars(kind, d):
    """alpha and (a, b, c) of an operator's stencil."""
    if kind == "der":
        return 1 / 3, (7 / 9 / d, 1 / 36 / d, 0.0)
    if kind == "der2":
        return 2 / 11, (12 / 11 / d**2, 3 / 44 / d**2, 0.0)
    if kind in ("dervp", "derpv"):
        return 9 / 62, (63 / 62 / d, 17 / 62 / 3 / d, 0.0)
    al = 0.49
    return al, ((75 + 70 * al) / 128, (126 * al - 25) / 256, (3 - 10 * al) / 256)


def _terms(kind, d):
    """The explicit stencil as (offset, weight) pairs."""
    a, b, c = _scalars(kind, d)[1]
    if kind == "der":
        return [(1, a), (-1, -a), (2, b), (-2, -b)]
    if kind == "der2":
        return [(1, a), (0, -2 * a), (-1, a), (2, b), (0, -2 * b), (-2, b)]
    if kind == "dervp":
        return [(1, a), (0, -a), (2, b), (-1, -b)]
    if kind == "derpv":
        return [(0, a), (-1, -a), (1, b), (-2, -b)]
    s = 1 if kind == "intvp" else 0
    return [(s, a), (s - 1, a), (s + 1, b), (s - 2, b), (s + 2, c), (s - 3, c)]


def _matrix(kind, n, d):
    """Dense M^-1 A of a periodic operator: rows of the stencil over the
    cyclic (alpha, 1, alpha) matrix.  (A transfer function on the modes would
    round the high ones' share of the field into the result.)"""
    al = _scalars(kind, d)[0]
    one = np.eye(n)
    lhs = one + al * (np.roll(one, 1, axis=1) + np.roll(one, -1, axis=1))
    rhs = sum(wt * np.roll(one, off, axis=1) for off, wt in _terms(kind, d))
    return torch.from_numpy(np.linalg.solve(lhs, rhs)).cuda()


def _along(mat, direction, u):
    axis = 2 - direction
    return torch.movedim(torch.tensordot(mat, u, dims=([1], [axis])), 0, axis).contiguous()


def _apply(kind, direction, u, d):
    return _along(_matrix(kind, u.shape[2 - direction], d), direction, u)


def _modes(kind, direction, u, d):
    """The periodic operator as its transfer function: used inside the step,
    whose divergence cancels the smooth part of the field, where a dense
    matrix's rounded row sums would show."""
    axis = 2 - direction
    n = u.shape[axis]
    w = TWO_PI * torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64) / n
    h = sum(wt * torch.exp(1j * off * w) for off, wt in _terms(kind, d))
    h = (h / (1 + 2 * _scalars(kind, d)[0] * torch.cos(w))).reshape([-1 if k == axis else 1 for k in range(3)])
    return torch.fft.irfft(torch.fft.rfft(u, dim=axis) * h, n=n, dim=axis)


def _wall_matrix(kind, n, d, ncl1, ncln, npaire):
    """Dense M^-1 A of a non-periodic operator for n velocity points."""
    al, (a, b, _) = _scalars(kind, d)
    if kind == "der":
        m = k = n
        up, lo, diag = np.full(n - 1, al), np.full(n - 1, al), np.ones(n)
        rhs = np.zeros((n, n))
        for i in range(2, n - 2):
            for off, wt in _terms(kind, d):
                rhs[i, i + off] += wt
        for end, ncl in ((0, ncl1), (1, ncln)):
            # row r and its neighbours counted from the wall; sg: orientation
            at = (lambda i: i) if end == 0 else (lambda i: n - 1 - i)
            sg = 1.0 if end == 0 else -1.0
            out_, in_ = (up, lo) if end == 0 else (lo, up)  # wall row's, then second row's wall side
            j = 0 if end == 0 else n - 2
            if ncl == 1:
                even = npaire == 1
                out_[j] = 0.0 if even else 2 * al
                if not even:
                    rhs[at(0), at(1)] += 2 * a * sg
                    rhs[at(0), at(2)] += 2 * b * sg
                rhs[at(1), at(2)] += a * sg
                rhs[at(1), at(0)] -= a * sg
                rhs[at(1), at(3)] += b * sg
                rhs[at(1), at(1)] += (-b if even else b) * sg
            else:
                out_[j] = 2.0
                in_[j] = 0.25
                (up if end == 0 else lo)[1 if end == 0 else n - 3] = 0.25
                for i, wt in ((0, -2.5 / d), (1, 2.0 / d), (2, 0.5 / d)):
                    rhs[at(0), at(i)] += wt * sg
                rhs[at(1), at(2)] += 0.75 / d * sg
                rhs[at(1), at(0)] -= 0.75 / d * sg
    else:
        vp = kind.endswith("vp")
        k, m = (n, n - 1) if vp else (n - 1, n)
        up, lo, diag = np.full(m - 1, al), np.full(m - 1, al), np.ones(m)
        if vp:
            diag[0] = diag[-1] = 1 + al
        else:
            up[0] = lo[-1] = 2 * al
        rhs = np.zeros((m, k))
        for i in range(m):
            for off, wt in _terms(kind, d):
                j = i + off
                if j < 0:
                    j = -j if vp else -1 - j
                elif j >= k:
                    j = 2 * (k - 1) - j if vp else 2 * k - 1 - j
                rhs[i, j] += wt
    lhs = np.diag(diag) + np.diag(up, 1) + np.diag(lo, -1)
    return torch.from_numpy(np.linalg.solve(lhs, rhs)).cuda()


def _waves(n, length):
    """Squared modified wavenumber and interpolation transfer function."""
    d = length / n
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    w = TWO_PI * torch.minimum(i, n - i) / n
    al, (a, b, _) = _scalars("dervp", d)
    wp = (2 * a * d * torch.sin(w / 2) + 2 * b * d * torch.sin(1.5 * w)) / (1 + 2 * al * torch.cos(w))
    al, (a, b, c) = _scalars("intvp", d)
    t = 2 * (a * torch.cos(w / 2) + b * torch.cos(1.5 * w) + c * torch.cos(2.5 * w)) / (1 + 2 * al * torch.cos(w))
    return (wp / d) ** 2, t


def _poisson(rhs, lengths):
    nz, ny, nx = rhs.shape
    (kx, tx), (ky, ty), (kz, tz) = (_waves(n, le) for n, le in zip((nx, ny, nz), lengths))
    h = nx // 2 + 1
    kx, tx = kx[:h][None, None, :], tx[:h][None, None, :]
    ky, ty = ky[None, :, None], ty[None, :, None]
    kz, tz = kz[:, None, None], tz[:, None, None]
    k = kx * (ty * tz) ** 2 + ky * (tx * tz) ** 2 + kz * (tx * ty) ** 2
    f = torch.where(k < 1e-16, torch.zeros_like(k), -1.0 / torch.clamp(k, min=1e-16))
    del k
    return torch.fft.irfftn(torch.fft.rfftn(rhs) * f, s=rhs.shape)


def _poisson_walls(case, rhs):
    lengths = list(_lengths(case))
    ext = rhs
    for d in range(3):
        if _walled(case, d):
            ext = torch.cat([ext, ext.flip(2 - d)], dim=2 - d)
            # the mirrored box of the n - 1 pressure points has twice the length
            lengths[d] *= 2
    out = _poisson(ext, lengths)
    return out[:rhs.shape[0], :rhs.shape[1], :rhs.shape[2]].contiguous()


def _step(case, u):
    d = [_spacing(case, k) for k in range(3)]
    ap = lambda kind, k, f: _modes(kind, k, f, d[k])  # noqa: E731
    du = [sum(ap("der", k, u[k] * uc) + u[k] * ap("der", k, uc) for k in range(3)) for uc in u]
    u = [a + STEP_DT * b for a, b in zip(u, du)]
    iv = lambda k, f: ap("intvp", k, f)  # noqa: E731
    div = iv(2, iv(1, ap("dervp", 0, u[0])) + ap("dervp", 1, iv(0, u[1]))) + ap("dervp", 2, iv(1, iv(0, u[2])))
    p = _poisson(div, _lengths(case))
    ip = lambda k, f: ap("intpv", k, f)  # noqa: E731
    pz = ip(2, p)
    g = [ap("derpv", 0, ip(1, pz)), ip(0, ap("derpv", 1, pz)), ip(0, ip(1, ap("derpv", 2, p)))]
    return dict(u=[a - b for a, b in zip(u, g)], du=du, p=p, g=g)


def exact(case, seed):
    shape = _shape(case)
    family = case["family"]
    if family == "boxes":
        out = []
        for i, b in enumerate(_boxes(case)):
            res = torch.empty((3, 3, 6) + b[::-1], dtype=torch.float64, device="cuda")
            for k, f in enumerate(_velocity(case, b, seed + 1000 * i)):
                for d in range(3):
                    for j, (_, kind) in enumerate(SWEEP[d]):
                        res[k, d, j] = _apply(kind, d, f.double(), TWO_PI / b[d])
            out.append(res)
        return out
    if family == "poisson":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        ps = [n - 1 if _walled(case, d) else n for d, n in enumerate(shape)]
        return _poisson_walls(case, _noise(gen, ps, 1.0))
    vel = [a.double() for a in _velocity(case, shape, seed)]
    if family == "operator":
        d = case["direction"]
        return _apply(case["kind"], d, vel[0], _spacing(case, d))
    if family == "sweep":
        return [_apply(kind, d, vel[0], _spacing(case, d)) for d in range(3) for _, kind in SWEEP[d]]
    if family == "walls":
        out = []
        bc = _bc(case)
        for _, _, kind, npaire, d in _wall_calls(case):
            mat = _wall_matrix(kind, shape[d], _spacing(case, d), bc[2 * d], bc[2 * d + 1], npaire)
            src = vel[2].narrow(2 - d, 0, shape[d] - 1) if kind.endswith("pv") else vel[0]
            out.append(_along(mat, d, src))
        return out
    return _step(case, vel)
