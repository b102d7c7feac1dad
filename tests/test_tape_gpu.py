"""Scalar programs over cells (values formed once, tables along one direction, short divisions) against the
oracle, bit for bit: expressions of every operator on uniform and stretched meshes, with and without tables
(from 2^15 cells), divisors and factors of every kind, zeros and values over the exponent range; and the
assembled coefficients of inner cells (from 4096 of them) beside the shell's."""
import numpy as np
import pytest

import common as cm
import oracle_lib as orc
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu


def _uniform(rng, s):
    return rng.random(s) + 0.5


def _wild(rng, s):
    v = rng.standard_normal(s) * 2.0 ** rng.integers(-1030, 400, s)
    v[rng.random(s) < 0.1] = 0.0
    return v


def _mesh(dims, stretched):
    return cm.mesh_points([cm.stretched_points(n) for n in dims]) if stretched else cm.mesh_uniform(list(dims))


def _terms(u, K, n):
    return [(u + 0.01 * (q + 1)) * (K - 0.02 * (q + 1)) / (3.0 + q) for q in range(n)]


def _sum(ts):
    s = ts[0]
    for t in ts[1:]:
        s = s + t
    return s


EXPRS = {
    "transport": lambda u, K, d: u + 1e-5 * sum((api.d1(api.d1IntpCenterToCorner(K, q) * api.d1(u, q), q) for q in range(1, d)),
                                                api.d1(api.d1IntpCenterToCorner(K, 0) * api.d1(u, 0), 0)) - 0.3 * api.d1_biased_upwind(u, 0),
    "laplace": lambda u, K, d: u - (0.25 * api.d2(u, 0)) / K - api.d2(u, d - 1) / 3.0 + u / K,
    "constants": lambda u, K, d: ((u / 300.0 - 1.0 * K) / (1.0 / 300) + (-1.0) * u) / 0.125 + 8.0 * K / -7.0 + 1.0 / u,
    "logic": lambda u, K, d: api.conditional(api.logical_or(u > K, u < 0.7), u * K, api.conditional(u >= K, u / 2.0, -K)),
    "functions": lambda u, K, d: api.max(api.abs(u - K), api.sqrt(api.abs(K))) + api.d1IntpCenterToCorner(K, 0) - -u,
    "limiter": lambda u, K, d: api.d1(api.d1_flux_limiter_intp(api.d1IntpCenterToCorner(K, 0), u, 0, "Superbee"), 0),
}


@pytest.mark.parametrize("dims", [(9, 8), (70, 37), (260, 150), (12, 9, 11), (45, 33, 40)])
@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("name", sorted(EXPRS))
def test_expressions_match_the_oracle(ctx, dims, stretched, name):
    D = len(dims)
    mesh = _mesh(dims, stretched)
    fd = cm.field_desc(D, capi.CENTER, [(capi.BC_NEUM, capi.BC_DIRC)] * D, ext=3)
    for values in (_uniform, _wild):
        rng = np.random.default_rng(sum(dims))
        hu, hk = orc.HostField(mesh, fd), orc.HostField(mesh, fd)
        for h in (hu, hk):
            sl = h.slices(h.assignable())
            h.data[sl] = values(rng, h.data[sl].shape)
            h.update_padding()
        u, K = api.CartesianField(mesh, fd, ctx), api.CartesianField(mesh, fd, ctx)
        u.upload(hu.data, update_padding=False)
        K.upload(hk.data, update_padding=False)
        L = [cm.Leaf("u"), cm.Leaf("K")]
        nodes = api.serialize(EXPRS[name](L[0], L[1], D), L)[0]
        for op in (capi.ASSIGN_EQ, capi.ASSIGN_ADD, capi.ASSIGN_DIV):
            u.assign(EXPRS[name](u, K, D), op={capi.ASSIGN_EQ: "=", capi.ASSIGN_ADD: "+", capi.ASSIGN_DIV: "/"}[op])
            orc.assign(hu, nodes, [hu, hk], op)
            got, want = u.download(), hu.data
            assert np.array_equal(got, want, equal_nan=True), (values.__name__, op, np.nanmax(np.abs(got - want)))


LONG = {
    # more than a small launch's instructions, more than any launch's, and more values at once than places
    "long": lambda u, K: _sum(_terms(u, K, 50)),
    "too_long": lambda u, K: _sum(_terms(u, K, 190)),
    "too_many": lambda u, K: _sum(_terms(u, K, 60)) * _sum([t * K for t in _terms(u, K, 60)]),
}


@pytest.mark.parametrize("dims", [(70, 37), (45, 33, 40)])
@pytest.mark.parametrize("name", sorted(LONG))
def test_long_expressions_match_numpy(ctx, dims, name):
    # (element by element: numpy's IEEE operations in the same order)
    mesh = _mesh(dims, False)
    fd = cm.field_desc(len(dims), capi.CENTER, [(capi.BC_NEUM, capi.BC_NEUM)] * len(dims), ext=1)
    u, K = api.CartesianField(mesh, fd, ctx), api.CartesianField(mesh, fd, ctx)
    sl = u.index_slices(u.assignableRange)
    vals = []
    for f in (u, K):
        a = f.download()
        a[sl] = _uniform(np.random.default_rng(len(vals)), a[sl].shape)
        f.upload(a)
        vals.append(a[sl].copy())
    u.assign(LONG[name](u, K))
    assert np.array_equal(u.download()[sl], LONG[name](*vals))


@pytest.mark.parametrize("n,stretched", [([80, 70], False), ([80, 70], True), ([260, 150], True), ([20, 21, 22], False), ([36, 33, 40], True)])
@pytest.mark.parametrize("bc,pin", [("neum", True), ("neum", False), ("dirc", False)])
def test_assembled_inner_cells_match_the_oracle(ctx, n, stretched, bc, pin):
    D = len(n)
    BC = {"neum": capi.BC_NEUM, "dirc": capi.BC_DIRC}[bc]
    mesh = _mesh([m + 1 for m in n], stretched)
    fd = cm.field_desc(D, capi.CENTER, [(BC, BC)] * D, [(0.3, -0.2)] * D, ext=1)
    rng = np.random.default_rng(sum(n))
    hosts = [orc.HostField(mesh, fd) for _ in range(3)]
    for h in hosts[1:]:
        sl = h.slices(h.assignable())
        h.data[sl] = rng.random(h.data[sl].shape) + 0.5
        h.update_padding()
    dev = [api.CartesianField(mesh, fd, ctx) for _ in hosts]
    for a, h in zip(dev, hosts):
        a.upload(h.data, update_padding=False)

    def eq(p, K, f):
        t = 0.5 * (K * p)
        for d in range(D):
            t = t - api.d1(api.d1IntpCenterToCorner(K, d) * api.d1(p, d), d) + api.d2(p, d) / 3.0
        return api.Eq(t, f / K + 2.0)
    off, coef, rhs = api.assemble(lambda e: eq(e, dev[1], dev[2]), dev[0], pin=pin)
    L = [cm.Leaf(x) for x in "pKf"]
    nodes = api.serialize(eq(*L).residual_expr(), L)[0]
    want_off, want_coef, want_rhs = orc.assemble(hosts[0], nodes, hosts, 0, int(pin))
    got = {tuple(o): np.asarray(coef)[:, q] for q, o in enumerate(np.asarray(off).tolist())}
    for q, o in enumerate(want_off.tolist()):
        assert np.array_equal(got[tuple(o)], want_coef[:, q]), (o, np.abs(got[tuple(o)] - want_coef[:, q]).max())
    assert np.array_equal(rhs, want_rhs)


@pytest.mark.parametrize("n", [[80, 70], [300, 260], [40, 33, 20], [50, 44, 42]])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_infinite_and_nan_coefficients_reach_the_right_hand_side(ctx, n, bad):
    # the bias of a pad is always there, and 0 times an infinite factor is NaN
    D = len(n)
    mesh = cm.mesh_uniform([m + 1 for m in n])
    fd = cm.field_desc(D, capi.CENTER, [(capi.BC_DIRC, capi.BC_DIRC)] * D, [(0.3, -0.2)] * D, ext=1)
    rng = np.random.default_rng(sum(n))
    hosts = [orc.HostField(mesh, fd) for _ in range(3)]
    for h in hosts[1:]:
        sl = h.slices(h.assignable())
        v = rng.random(h.data[sl].shape) + 0.5
        if h is hosts[1]:
            v.flat[rng.integers(0, v.size, 40)] = bad
        h.data[sl] = v
        h.update_padding()
    dev = [api.CartesianField(mesh, fd, ctx) for _ in hosts]
    for a, h in zip(dev, hosts):
        a.upload(h.data, update_padding=False)

    def eq(p, K, f):
        t = 2.0 * p
        for d in range(D):
            t = t - api.d1(api.d1IntpCenterToCorner(K, d) * api.d1(p, d), d)
        return api.Eq(t, f)
    L = [cm.Leaf(x) for x in "pKf"]
    nodes = api.serialize(eq(*L).residual_expr(), L)[0]
    want = orc.assemble(hosts[0], nodes, hosts, 0, 0)[2]
    rhs = api.assemble(lambda e: eq(e, dev[1], dev[2]), dev[0])[2]
    assert np.isnan(want).any() and not np.isnan(want).all()
    assert np.array_equal(rhs, want, equal_nan=True)


@pytest.mark.parametrize("n", [[80, 70], [40, 33, 20]])
def test_coefficients_that_become_infinite_reach_a_kept_matrix_s_right_hand_side(ctx, n):
    # staticMat: the right-hand side alone is formed again, with the factors of the fields written since
    D = len(n)
    fd = cm.field_desc(D, capi.CENTER, [(capi.BC_DIRC, capi.BC_DIRC)] * D, ext=1)
    mesh = cm.mesh_uniform([m + 1 for m in n])
    p, K, f = (api.CartesianField(mesh, fd, ctx) for _ in range(3))
    K.assign(1.5 + 0.0 * f)
    f.assign(0.0 * K + 1.0)

    def eq(e):
        t = 2.0 * e
        for d in range(D):
            t = t - 1e-3 * api.d1(api.d1IntpCenterToCorner(K, d) * api.d1(e, d), d)
        return api.Eq(t, f)
    s = api.EqnSolveHandler(eq, p, api.StructSolverParams(tol=1e-8, maxIter=30, precision="mixed", staticMat=True))
    assert s.solve().converged and s.solve().converged
    f.assign(0.0 * K + 2.0)
    assert s.solve().converged
    a = K.download()
    a[tuple(m // 2 for m in reversed(n))] = np.inf
    K.upload(a)
    st = s.solve()
    assert not st.converged and np.isnan(st.relerr)


@pytest.mark.parametrize("n,stretched", [([300, 260], False), ([300, 260], True), ([50, 44, 42], False), ([50, 44, 42], True), ([258, 258], False), ([256, 259], True)])
@pytest.mark.parametrize("bc,pin", [("neum", True), ("neum", False), ("dirc", False)])
def test_assembled_inner_cells_of_larger_boxes(ctx, n, stretched, bc, pin):
    # (from 65536 inner cells the coefficients come from the scalar program: 256 x 256 of 258 x 258, 254 x 257 of 256 x 259)
    test_assembled_inner_cells_match_the_oracle(ctx, n, stretched, bc, pin)
