"""The work this framework is used for, as cases that can be timed and checked one by one.

Explicit assignments (the heat equation in both arithmetic modes, a variable-coefficient transport
equation, WENO5 advection, many grids at once) and implicit solves (one handler solved again and again,
one whole Solve call, a batch of Helmholtz problems, a served window of mixed requests), over the sizes
of the repository's own configurations and tests.  `exact` gives the same results in 64 bits without
the framework's code: torch expressions for the explicit cases, sine and cosine transforms (as dense
matrices) for the constant-coefficient solves, conjugate gradients preconditioned with them for the
variable-coefficient ones.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from opflow_gb300 import _capi as capi
from opflow_gb300 import api

F64 = torch.float64
DEV = "cuda"


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # one step per call on a small grid: what a time loop with other work between its steps pays
        dict(name="ftcs2d_65", kind="ftcs", nd=2, nx=65, ny=65, nz=1, mode="exact", steps=1),
        # the FTCS2D program's grid, part of its 1000 steps in one call, the reference's bits
        dict(name="ftcs2d_1025", kind="ftcs", nd=2, nx=1025, ny=1025, nz=1, mode="exact", steps=50),
        # the 512^3 heat run in the fixed-point mode
        dict(name="ftcs3d_512_fast", kind="ftcs", nd=3, nx=512, ny=512, nz=512, mode="fast", steps=50),
        # a 3D heat run in the reference's bits, odd extents and a spacing that is no power of two
        dict(name="ftcs3d_301_exact", kind="ftcs", nd=3, nx=301, ny=257, nz=333, mode="exact", steps=4),
        # advection-diffusion with a variable coefficient: any expression a user writes that is no FTCS step
        dict(name="transport2d_1000", kind="transport", nd=2, nx=1000, ny=702, nz=1, steps=4),
        # the WENO5-RK3 configuration's line length, a quarter of its lines
        dict(name="weno_exact_16384", kind="weno", lines=16384, n=4096, mode="exact", steps=1),
        # explicit steps of many uneven grids at once
        dict(name="ftcs_batch_64", kind="ftcs_batch", count=64, mix=11, steps=4),
        # the pressure equation of a time loop: one handler, its matrix kept, solved again
        dict(name="poisson2d_2048", kind="poisson", nd=2, nx=2048, ny=2048, nz=1, bc="neum", precision="mixed"),
        dict(name="poisson3d_256", kind="poisson", nd=3, nx=256, ny=256, nz=256, bc="neum", precision="mixed"),
        # one whole Solve call (assembly, set-up, solve) with a variable coefficient, all in float64
        dict(name="solve3d_expg_192", kind="expg", nd=3, nx=192, ny=192, nz=192, precision="fp64"),
        # many uneven Helmholtz problems solved together
        dict(name="helmholtz_batch_64", kind="helmholtz", count=64, mix=12),
        # a served window: one-shot Poisson requests and backward-Euler sessions, inputs resident
        dict(name="serve_24", kind="serve", count=24, mix=13),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _halving(n):
    """The nearest extent of the form (8 .. 15) * 2^k: one whose coarser grids halve evenly.  The singular
    (all-Neumann) problems are taken on such extents: elsewhere their iteration count varies with the
    right-hand side, and a few right-hand sides in a hundred never reach the tolerance."""
    k = max(0, n.bit_length() - 4)
    return max(8, int(round(n / (1 << k)))) << k


def draw(rng):
    kind = rng.choice(["ftcs2d", "ftcs3d", "transport", "weno", "ftcs_batch", "poisson2d", "poisson3d", "expg", "helmholtz", "serve"])
    if kind == "ftcs2d":
        return dict(kind="ftcs", nd=2, nx=_log_int(rng, 33, 2049), ny=_log_int(rng, 33, 2049), nz=1, mode=rng.choice(["exact", "fast"]),
                    steps=_log_int(rng, 1, 100))
    if kind == "ftcs3d":
        return dict(kind="ftcs", nd=3, nx=_log_int(rng, 17, 400), ny=_log_int(rng, 17, 400), nz=_log_int(rng, 17, 400),
                    mode=rng.choice(["exact", "fast"]), steps=_log_int(rng, 1, 20))
    if kind == "transport":
        nd = rng.choice([2, 3])
        hi = 1500 if nd == 2 else 130
        return dict(kind="transport", nd=nd, nx=_log_int(rng, 24, hi), ny=_log_int(rng, 24, hi), nz=_log_int(rng, 24, hi) if nd == 3 else 1,
                    steps=_log_int(rng, 1, 8))
    if kind == "weno":
        return dict(kind="weno", lines=_log_int(rng, 3, 16384), n=_log_int(rng, 40, 4096), mode=rng.choice(["exact", "fast"]),
                    steps=_log_int(rng, 1, 4))
    if kind == "ftcs_batch":
        return dict(kind="ftcs_batch", count=rng.randint(4, 64), mix=rng.randint(100, 100000), steps=rng.randint(1, 8))
    if kind in ("poisson2d", "poisson3d"):
        nd = 2 if kind == "poisson2d" else 3
        lo, hi = (48, 2048) if nd == 2 else (24, 256)
        a = _log_int(rng, lo, hi)
        # the extents of one problem stay within a factor: spacings are near each other, as in use
        ext = [a if rng.random() < 0.5 else max(lo, min(hi, int(a * rng.uniform(0.8, 1.25)))) for _ in range(nd)]
        bc = rng.choice(["neum", "dirc"])
        if bc == "neum":
            ext = [_halving(m) for m in ext]
        return dict(kind="poisson", nd=nd, nx=ext[0], ny=ext[1], nz=ext[2] if nd == 3 else 1, bc=bc,
                    precision=rng.choice(["mixed", "mixed", "fp64"]))
    if kind == "expg":
        nd = rng.choice([2, 3, 3])
        n = _halving(_log_int(rng, 48, 1024) if nd == 2 else _log_int(rng, 24, 192))
        return dict(kind="expg", nd=nd, nx=n, ny=n, nz=n if nd == 3 else 1, precision=rng.choice(["mixed", "fp64"]))
    if kind == "helmholtz":
        return dict(kind="helmholtz", count=rng.randint(2, 64), mix=rng.randint(100, 100000))
    return dict(kind="serve", count=rng.randint(2, 24), mix=rng.randint(100, 100000))


# ------------------------------------------------------------------------------------- views and inputs
class _Span:
    """A device buffer of the framework as a CUDA array; keeps the object that owns the buffer."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (int(ptr), False), "version": 3}


def _values(state, f, inner):
    """The field's current values as a tensor (no copy); `inner`: its assignable cells only."""
    p = f.device_ptr()
    views = state.setdefault("views", {})
    v = views.get(p)
    if v is None:
        v = torch.as_tensor(_Span(f, p, f.shape), device=DEV)
        views[p] = v = v[f.index_slices(f.assignableRange)] if inner else v
    return v


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _extents(case):
    return [case["nx"], case["ny"], case["nz"]][:case["nd"]]


def _outer(vs):
    """Product field of per-dim profiles vs[d] (x first), indexed [z, y, x]."""
    out = vs[0]
    for v in vs[1:]:
        out = v.reshape([-1] + [1] * out.dim()) * out
    return out


def _gaussians(n, seed):
    """8 Gaussians in the unit box on the nodes of an n[0] x n[1] (x n[2]) grid, 0 on its boundary."""
    g = _gen(seed)
    c = 0.2 + 0.6 * torch.rand(8, 3, generator=g, dtype=F64, device=DEV)
    w = 0.03 + 0.07 * torch.rand(8, generator=g, dtype=F64, device=DEV)
    a = 0.5 + 0.5 * torch.rand(8, generator=g, dtype=F64, device=DEV)
    u = None
    for k in range(8):
        vs = []
        for d, m in enumerate(n):
            x = torch.linspace(0, 1, m, dtype=F64, device=DEV)
            v = torch.exp(-((x - c[k, d]) / w[k]) ** 2)
            v[0] = v[-1] = 0
            vs.append(v)
        t = a[k] * _outer(vs)
        u = t if u is None else u + t
    return u


def _smooth(n, seed):
    """A smooth random field on cell centres (six low Fourier modes), standard deviation 1."""
    g = _gen(seed + 1000)
    out = None
    for _ in range(6):
        k = torch.randint(1, 4, (3,), generator=g, device=DEV)
        ph = 2 * math.pi * torch.rand(3, generator=g, dtype=F64, device=DEV)
        a = torch.randn(1, generator=g, dtype=F64, device=DEV)
        vs = [torch.cos(2 * math.pi * k[d] * (torch.arange(m, dtype=F64, device=DEV) + 0.5) / m + ph[d]) for d, m in enumerate(n)]
        t = a * _outer(vs)
        out = t if out is None else out + t
    return (out - out.mean()) / out.std()


def _mesh(nodes):
    b = api.MeshBuilder().newMesh(*nodes)
    for d in range(len(nodes)):
        b.setMeshOfDim(d, 0.0, 1.0)
    return b.build()


def _builder(mesh, loc, bc, ext):
    b = api.ExprBuilder().setMesh(mesh).setLoc(loc)
    if ext:
        b.setExt(ext)
    for d in range(mesh.ndim):
        b.setBC(d, api.DimPos.start, bc, 0.0).setBC(d, api.DimPos.end, bc, 0.0)
    return b


def _fill(f, values):
    """Uploads `values` (a tensor over the assignable cells) into the field."""
    a = np.zeros(f.shape)
    a[f.index_slices(f.assignableRange)] = values.cpu().numpy()
    f.upload(a)


def _cells(n, seed, zero_mean):
    v = torch.randn(tuple(reversed(n)), generator=_gen(seed + 2000), dtype=F64, device=DEV)
    return v - v.mean() if zero_mean else v


def _weno_u0(lines, n, seed):
    """Per line a square and a cosine pulse."""
    g = _gen(seed + 3000)

    def uni(lo, hi):
        return lo + (hi - lo) * torch.rand(lines, 1, generator=g, dtype=F64, device=DEV)
    x = ((torch.arange(n, dtype=F64, device=DEV) + 0.5) / n)[None, :]
    c1, w1, a1, c2, w2, a2 = uni(0.1, 0.4), uni(0.05, 0.15), uni(0.5, 1.0), uni(0.55, 0.85), uni(0.05, 0.12), uni(0.3, 0.8)
    u = torch.where((x - c1).abs() < w1, a1, torch.zeros_like(x))
    d = (x - c2) / w2
    return u + torch.where(d.abs() < 1.0, a2 * torch.cos(0.5 * math.pi * d) ** 2, torch.zeros_like(d))


def _batch_sides(case):
    """Sides of the explicit batch: LogU[65, 513]."""
    r = random.Random(case["mix"])
    return [_log_int(r, 65, 513) for _ in range(case["count"])]


def _helmholtz(case):
    """(side, k) of the Helmholtz batch: side LogU[65, 1025] rounded to 2^m + 1, k LogU[1e-4, 1]."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["count"]):
        k = math.exp(r.uniform(math.log(1e-4), 0.0))
        side = math.exp(r.uniform(math.log(65), math.log(1025)))
        out.append(((1 << int(round(math.log2(side - 1)))) + 1, k))
    return out


def _serve_mix(case):
    """The served mix: 70% one-shot Poisson solves (2D side LogU[129, 1025], 3D LogU[64, 160], Neumann or
    Dirichlet), 30% backward-Euler sessions of 10-100 steps (side LogU[129, 513], dt = 1/side)."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["count"]):
        if r.random() < 0.7:
            n = [_log_int(r, 129, 1025)] * 2 if r.random() < 0.5 else [_log_int(r, 64, 160)] * 3
            bc = r.choice(["neum", "dirc"])
            out.append(dict(n=[_halving(m) for m in n] if bc == "neum" else n, alpha=0.0, beta=1.0, bc=bc, steps=1))
        else:
            n = _log_int(r, 129, 513)
            out.append(dict(n=[n, n], alpha=1.0, beta=1.0 / n, bc="dirc", steps=r.randint(10, 100)))
    return out


def _serve_f(q, k, seed):
    return _cells(q["n"], seed + 97 * k, q["bc"] == "neum").reshape(-1)


_BC = {"neum": api.BCType.Neum, "dirc": api.BCType.Dirc}


def _params(case, **more):
    p = dict(tol=1e-10, maxIter=300, precision=case.get("precision", "mixed"), zeroGuess=True)
    p.update(more)
    return api.StructSolverParams(**p)


# ------------------------------------------------------------------------------------------ expressions
def _ftcs_s(n):
    return 0.15 * (1.0 / (max(n) - 1)) ** 2


def _transport_dt(n):
    return 0.02 * (1.0 / max(n)) ** 2


_VEL = (0.5, 0.3, 0.2)


def _transport_expr(u, K, n):
    """u + dt*(div(K grad u) - v . grad u), the gradient of the advection taken downwind"""
    D1 = (api.dx, api.dy, api.dz)
    rhs = None
    for d in range(len(n)):
        t = D1[d](api.d1IntpCenterToCorner(K, d) * D1[d](u)) - _VEL[d] * D1[d](u, api.D1FirstOrderBiasedDownwind)
        rhs = t if rhs is None else rhs + t
    return u + _transport_dt(n) * rhs


def _expg_equation(f, K, nd):
    D1 = (api.dx, api.dy, api.dz)

    def getter(e):
        lhs = None
        for d in range(nd):
            t = D1[d](api.d1IntpCenterToCorner(K, d) * D1[d](e))
            lhs = t if lhs is None else lhs + t
        return f == lhs
    return getter


def _poisson_equation(f, nd):
    D2 = (api.d2x, api.d2y, api.d2z)

    def getter(e):
        lhs = None
        for d in range(nd):
            lhs = D2[d](e) if lhs is None else lhs + D2[d](e)
        return f == lhs
    return getter


# ---------------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def _prepare_ftcs(case, seed):
    n = _extents(case)
    u = _builder(_mesh(n), api.LocOnMesh.Corner, api.BCType.Dirc, 0).build()
    u.upload(_gaussians(n, seed).cpu().numpy())
    D2 = (api.d2x, api.d2y, api.d2z)
    lap = D2[0](u)
    for d in range(1, len(n)):
        lap = lap + D2[d](u)
    return dict(case=case, u=u, expr=u + _ftcs_s(n) * lap)


def _prepare_transport(case, seed):
    n = _extents(case)
    b = _builder(_mesh([m + 1 for m in n]), api.LocOnMesh.Center, api.BCType.Neum, 1)
    u, K = b.build(), b.build()
    _fill(u, _smooth(n, seed + 1))
    _fill(K, torch.exp(0.5 * _smooth(n, seed)))
    return dict(case=case, u=u, K=K, expr=_transport_expr(u, K, n))


def _prepare_weno(case, seed):
    n, lines = case["n"], case["lines"]
    mesh = api.MeshBuilder().newMesh(n + 1, lines + 1).setMeshOfDim(0, 0.0, 1.0).setMeshOfDim(1, 0.0, lines / n).build()
    u = _builder(mesh, api.LocOnMesh.Center, api.BCType.Periodic, 3).build()
    _fill(u, _weno_u0(lines, n, seed))
    return dict(case=case, u=u, dt=0.5 / n, mode=capi.EVAL_FAST if case["mode"] == "fast" else capi.EVAL_EXACT)


def _prepare_ftcs_batch(case, seed):
    fields, work = [], []
    for k, n in enumerate(_batch_sides(case)):
        u = _builder(_mesh([n, n]), api.LocOnMesh.Corner, api.BCType.Dirc, 0).build()
        u.upload(_gaussians([n, n], seed + 31 * k).cpu().numpy())
        fields.append(u)
        work.append((u, u + 0.2 * (1.0 / (n - 1)) ** 2 * (api.d2x(u) + api.d2y(u))))
    return dict(case=case, fields=fields, work=work, state=[{} for _ in fields])


def _prepare_poisson(case, seed):
    n = _extents(case)
    b = _builder(_mesh([m + 1 for m in n]), api.LocOnMesh.Center, _BC[case["bc"]], 1)
    p, f = b.build(), b.build()
    neum = case["bc"] == "neum"
    _fill(f, _cells(n, seed, neum))
    h = api.makeEqnSolveHandler(_poisson_equation(f, len(n)), p, _params(case, pinValue=neum, staticMat=True))
    return dict(case=case, p=p, f=f, handler=h)


def _prepare_expg(case, seed):
    n = _extents(case)
    b = _builder(_mesh([m + 1 for m in n]), api.LocOnMesh.Center, api.BCType.Neum, 1)
    p, f, K = b.build(), b.build(), b.build()
    _fill(K, torch.exp(_smooth(n, seed)))
    _fill(f, _cells(n, seed, True))
    return dict(case=case, p=p, f=f, K=K, params=_params(case, pinValue=True), getter=_expg_equation(f, K, len(n)))


def _prepare_helmholtz(case, seed):
    probs = []
    for side, k in _helmholtz(case):
        h = 1.0 / (side - 1)
        probs.append(api.Problem([side, side], [h, h], alpha=1.0, beta=k, loc=api.LocOnMesh.Corner, bc=api.BCType.Dirc))
    B = api.Batch(probs, _params(case))
    out = []
    for i, p in enumerate(probs):
        m = p.n[0] - 2
        B.set(i, _cells([m, m], seed + 53 * i, False).cpu().numpy())
        x, cnt = C.c_void_p(), C.c_size_t(0)
        capi.check(capi.lib().opflow_batch_vectors(B.handle, i, C.byref(x), None, C.byref(cnt)))
        out.append(torch.as_tensor(_Span(B, x.value, (m, m)), device=DEV))
    return dict(case=case, batch=B, out=out)


def _prepare_serve(case, seed):
    reqs = []
    for k, q in enumerate(_serve_mix(case)):
        p = api.Problem(q["n"], [1.0 / m for m in q["n"]], alpha=q["alpha"], beta=q["beta"], loc=api.LocOnMesh.Center, bc=_BC[q["bc"]])
        f = _serve_f(q, k, seed)
        reqs.append((p, f, q["steps"], torch.empty_like(f)))
    torch.cuda.synchronize()  # the server's own threads read the tensors
    return dict(case=case, server=api.Server(_params(case), max_active=64), reqs=reqs)


_PREPARE = dict(ftcs=_prepare_ftcs, transport=_prepare_transport, weno=_prepare_weno, ftcs_batch=_prepare_ftcs_batch, poisson=_prepare_poisson,
                expg=_prepare_expg, helmholtz=_prepare_helmholtz, serve=_prepare_serve)


# -------------------------------------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ftcs":
        state["u"].assign(state["expr"], mode=case["mode"], steps=case["steps"])
        return _values(state, state["u"], False)
    if kind == "transport":
        state["u"].assign(state["expr"], steps=case["steps"])
        return _values(state, state["u"], True)
    if kind == "weno":
        api.weno_rk3(state["u"], state["dt"], case["steps"], mode=state["mode"])
        return _values(state, state["u"], True)
    if kind == "ftcs_batch":
        api.assign_batch(state["work"], steps=case["steps"])
        return [_values(s, u, False) for s, u in zip(state["state"], state["fields"])]
    if kind == "poisson":
        state["handler"].solve()
        return _values(state, state["p"], True)
    if kind == "expg":
        api.Solve(state["getter"], state["p"], state["params"])
        return _values(state, state["p"], True)
    if kind == "helmholtz":
        state["batch"].solve()
        return state["out"]
    ids = [state["server"].submit(p, f, steps=steps, out=out) for p, f, steps, out in state["reqs"]]
    for i in ids:
        r = state["server"].result(i)
        if r["status"] != capi.OK:
            raise RuntimeError("request %d: status %d" % (i, r["status"]))
    return [out for _, _, _, out in state["reqs"]]


# ------------------------------------------------------------------------------------------------- work
def work(case):
    """Bytes: every field read once and written once per call.  Operations: per cell and step what the
    update's formula holds, per solve one operator and the updates of one iteration (a solver that needs
    one iteration needs no more)."""
    kind = case["kind"]
    if kind in ("ftcs", "transport"):
        n = _extents(case)
        cells = math.prod(n)
        per = (5 * len(n) + 2) if kind == "ftcs" else 14 * len(n)
        return dict(bytes=(16 if kind == "ftcs" else 24) * cells, flops=per * cells * case["steps"])
    if kind == "weno":
        cells = case["n"] * case["lines"]
        return dict(bytes=16 * cells, flops=3 * 70 * cells * case["steps"])
    if kind == "ftcs_batch":
        cells = sum(n * n for n in _batch_sides(case))
        return dict(bytes=16 * cells, flops=12 * cells * case["steps"])
    if kind in ("poisson", "expg"):
        cells = math.prod(_extents(case))
        return dict(bytes=(16 if kind == "poisson" else 24) * cells, flops=60 * cells)
    if kind == "helmholtz":
        cells = sum((s - 2) ** 2 for s, _ in _helmholtz(case))
        return dict(bytes=16 * cells, flops=60 * cells)
    mix = _serve_mix(case)
    return dict(bytes=sum(16 * math.prod(q["n"]) for q in mix), flops=sum(60 * math.prod(q["n"]) * q["steps"] for q in mix))


# ------------------------------------------------------------------------------------------------ exact
def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def _lap_step(u, s, n):
    """u + s * Laplacian on the inner nodes, the boundary nodes kept."""
    nd = len(n)
    inner = (slice(1, -1),) * nd
    c = u[inner]
    lap = torch.zeros_like(c)
    for d in range(nd):
        ax = nd - 1 - d
        lo, hi = list(inner), list(inner)
        lo[ax], hi[ax] = slice(0, -2), slice(2, None)
        lap += (u[tuple(lo)] - 2 * c + u[tuple(hi)]) * float(n[d] - 1) ** 2
    out = u.clone()
    out[inner] = c + s * lap
    return out


def _exact_ftcs(case, seed):
    n = _extents(case)
    u = _gaussians(n, seed)
    for _ in range(case["steps"]):
        u = _lap_step(u, _ftcs_s(n), n)
    return u


def _exact_ftcs_batch(case, seed):
    out = []
    for k, n in enumerate(_batch_sides(case)):
        u = _gaussians([n, n], seed + 31 * k)
        for _ in range(case["steps"]):
            u = _lap_step(u, 0.2 * (1.0 / (n - 1)) ** 2, [n, n])
        out.append(u)
    return out


def _faces(v, ax):
    """v with its first and last cells repeated along ax (mirrored ghosts), differences and means at the faces"""
    n = v.shape[ax]
    g = torch.cat([v.narrow(ax, 0, 1), v, v.narrow(ax, n - 1, 1)], ax)
    a, b = g.narrow(ax, 0, n + 1), g.narrow(ax, 1, n + 1)
    return b - a, 0.5 * (a + b)


def _flux_div(u, K, n):
    out = torch.zeros_like(u)
    for d, m in enumerate(n):
        ax = len(n) - 1 - d
        flux = _faces(u, ax)[0] * _faces(K, ax)[1]
        out += (flux.narrow(ax, 1, m) - flux.narrow(ax, 0, m)) * float(m) ** 2
    return out


def _exact_transport(case, seed):
    n = _extents(case)
    u, K = _smooth(n, seed + 1), torch.exp(0.5 * _smooth(n, seed))
    for _ in range(case["steps"]):
        rhs = _flux_div(u, K, n)
        for d, m in enumerate(n):
            ax = len(n) - 1 - d
            rhs -= _VEL[d] * _faces(u, ax)[0].narrow(ax, 0, m) * m
        u = u + _transport_dt(n) * rhs
    return u


def _weno_rhs(u, h):
    w = [u.roll(3 - s, 1) for s in range(6)]
    d1, d2, d3, d4, d5 = [(w[s + 1] - w[s]) / h for s in range(5)]
    p1 = d1 / 3 - 7 * d2 / 6 + 11 * d3 / 6
    p2 = -d2 / 6 + 5 * d3 / 6 + d4 / 3
    p3 = d3 / 3 + 5 * d4 / 6 - d5 / 6
    s1 = 13 / 12 * (d1 - 2 * d2 + d3) ** 2 + (d1 - 4 * d2 + 3 * d3) ** 2 / 4
    s2 = 13 / 12 * (d2 - 2 * d3 + d4) ** 2 + (d2 - d4) ** 2 / 4
    s3 = 13 / 12 * (d3 - 2 * d4 + d5) ** 2 + (3 * d3 - 4 * d4 + d5) ** 2 / 4
    eps = 1e-6 * torch.stack([d1, d2, d3, d4, d5]).square().amax(0) + 1e-99
    a1, a2, a3 = .1 / (s1 + eps) ** 2, .6 / (s2 + eps) ** 2, .3 / (s3 + eps) ** 2
    return (a1 * p1 + a2 * p2 + a3 * p3) / (a1 + a2 + a3)


def _exact_weno(case, seed):
    u = _weno_u0(case["lines"], case["n"], seed)
    h, dt = 1.0 / case["n"], 0.5 / case["n"]
    for part in u.split(2048):
        v = part.clone()
        for _ in range(case["steps"]):
            v1 = v - dt * _weno_rhs(v, h)
            v2 = 0.75 * v + 0.25 * (v1 - dt * _weno_rhs(v1, h))
            v = v / 3 + 2.0 / 3.0 * (v2 - dt * _weno_rhs(v2, h))
        part.copy_(v)
    return u


def _modes(m, h, how):
    """Orthonormal eigenvectors [mode, cell] and eigenvalues of the 1D operator -d2 with spacing h:
    cell-centred Neumann ("neum") and Dirichlet ("dirc") cells, inner nodes between Dirichlet ends ("node")."""
    i = torch.arange(m, dtype=F64, device=DEV)
    if how == "neum":
        k = i.clone()
        q = torch.cos(math.pi * k[:, None] * (i[None, :] + 0.5) / m) * math.sqrt(2.0 / m)
        q[0] = 1.0 / math.sqrt(m)
        th = math.pi * k / (2 * m)
    elif how == "dirc":
        k = i + 1
        q = torch.sin(math.pi * k[:, None] * (i[None, :] + 0.5) / m) * math.sqrt(2.0 / m)
        q[m - 1] *= math.sqrt(0.5)
        th = math.pi * k / (2 * m)
    else:
        k = i + 1
        q = torch.sin(math.pi * k[:, None] * (i[None, :] + 1) / (m + 1)) * math.sqrt(2.0 / (m + 1))
        th = math.pi * k / (2 * (m + 1))
    return q, (2 * torch.sin(th) / h) ** 2


def _spectral(n, h, how):
    """(to modes, from modes, eigenvalues of -Laplacian over [z, y, x])"""
    qs, ls = zip(*[_modes(m, hh, how) for m, hh in zip(n, h)])
    lam = torch.zeros(tuple(reversed(n)), dtype=F64, device=DEV)
    for d in range(len(n)):
        lam += ls[d].reshape([-1] + [1] * d)

    def apply(v, inverse):
        for d in range(len(n)):
            ax = len(n) - 1 - d
            q = qs[d].T if inverse else qs[d]
            v = torch.movedim(torch.movedim(v, ax, -1) @ q.T, -1, ax)
        return v
    return (lambda v: apply(v, False)), (lambda v: apply(v, True)), lam


def _spectral_solve(f, n, h, how, alpha, beta, steps=1):
    """(alpha + beta * -Laplacian)^-steps f; of a singular operator the zero-mean solution"""
    to, back, lam = _spectral(n, h, how)
    m = alpha + beta * lam
    inv = torch.where(m == 0, torch.zeros_like(m), 1.0 / m)
    return back(to(f) * inv ** steps)


def _exact_poisson(case, seed):
    n = _extents(case)
    neum = case["bc"] == "neum"
    x = -_spectral_solve(_cells(n, seed, neum), n, [1.0 / m for m in n], case["bc"], 0.0, 1.0)
    return x - x.reshape(-1)[0] if neum else x


def _exact_expg(case, seed):
    """Conjugate gradients on -div(K grad p) = -f, preconditioned with the constant-coefficient inverse."""
    n = _extents(case)
    K, f = torch.exp(_smooth(n, seed)), _cells(n, seed, True)
    to, back, lam = _spectral(n, [1.0 / m for m in n], "neum")
    inv = torch.where(lam == 0, torch.zeros_like(lam), 1.0 / lam)
    scale = K.rsqrt()
    x = torch.zeros_like(f)
    r = -f
    stop = 1e-14 * float(r.norm())
    z = scale * back(to(scale * r) * inv)
    p, rz = z.clone(), float((r * z).sum())
    for _ in range(400):
        q = -_flux_div(p, K, n)
        al = rz / float((p * q).sum())
        x += al * p
        r -= al * q
        r -= r.mean()
        if float(r.norm()) <= stop:
            break
        z = scale * back(to(scale * r) * inv)
        rz, old = float((r * z).sum()), rz
        p = z + (rz / old) * p
    return x - x.reshape(-1)[0]


def _exact_helmholtz(case, seed):
    out = []
    for i, (side, k) in enumerate(_helmholtz(case)):
        m = side - 2
        out.append(_spectral_solve(_cells([m, m], seed + 53 * i, False), [m, m], [1.0 / (side - 1)] * 2, "node", 1.0, k))
    return out


def _exact_serve(case, seed):
    out = []
    for k, q in enumerate(_serve_mix(case)):
        f = _serve_f(q, k, seed).reshape(tuple(reversed(q["n"])))
        x = _spectral_solve(f, q["n"], [1.0 / m for m in q["n"]], q["bc"], q["alpha"], q["beta"], q["steps"]).reshape(-1)
        out.append(x - x[0] if q["bc"] == "neum" else x)
    return out


_EXACT = dict(ftcs=_exact_ftcs, transport=_exact_transport, weno=_exact_weno, ftcs_batch=_exact_ftcs_batch, poisson=_exact_poisson,
              expg=_exact_expg, helmholtz=_exact_helmholtz, serve=_exact_serve)
