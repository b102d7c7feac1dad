"""The Krylov vector kernels: the residual of what they converge to, formed apart by the expression kernels,
over extents and boundaries that reach every branch of the operator's march (1D to 3D, constant and array
coefficients, periodic, rows longer and shorter than a chunk, single rows and planes), and values for which
a float32 copy of the residual is subnormal, zero or infinite."""
import numpy as np
import pytest

import common as cm
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu

BC = {"neum": capi.BC_NEUM, "dirc": capi.BC_DIRC, "per": capi.BC_PERIODIC}
TOL = 1e-9


def _solve(ctx, n, bc, array, prec, scale=1.0, guess=True, tol=TOL, A=1.0):
    D = len(n)
    mesh = cm.mesh_uniform([m + 1 for m in n])
    fd = cm.field_desc(D, capi.CENTER, [(BC[bc], BC[bc])] * D, ext=1)
    p, f, w, c = (api.CartesianField(mesh, fd, ctx) for _ in range(4))
    sl = f.index_slices(f.assignableRange)
    rng = np.random.default_rng(sum(n))
    for x, v in ((f, rng.standard_normal), (p, rng.standard_normal), (c, lambda s: 1.0 + rng.random(s))):
        a = x.download()
        a[sl] = v(a[sl].shape) * (A if x is c else scale)
        x.upload(a)
    d2 = [api.d2x, api.d2y, api.d2z][:D]

    def op(e):
        t = c * e if array else 1.0 * e
        for d, m in zip(d2, n):
            t = t - A * 0.2 / m ** 2 * d(e)
        return t
    par = api.StructSolverParams(tol=tol, maxIter=60, precision=prec, zeroGuess=not guess)
    st = api.Solve(lambda e: api.Eq(op(e), f), p, par)
    w.assign(op(p))
    fa, wa = f.download()[sl], w.download()[sl]
    return st, np.linalg.norm(fa - wa) / np.linalg.norm(fa), p.download()[sl]


@pytest.mark.parametrize("n,bc", [
    ([5], "neum"), ([1000], "per"), ([9001], "dirc"),
    ([7, 5], "dirc"), ([300, 17], "neum"), ([9000, 5], "per"), ([33, 513], "per"), ([257, 130], "dirc"),
    ([6, 5, 4], "neum"), ([40, 33, 19], "per"), ([300, 10, 9], "dirc"), ([24, 50, 70], "neum"),
])
@pytest.mark.parametrize("array", [False, True])
def test_the_residual_formed_apart_meets_the_tolerance(ctx, n, bc, array):
    for prec in ("mixed", "fp64"):
        st, res, _ = _solve(ctx, n, bc, array, prec)
        # the recurrence's residual meets the tolerance; the true one differs by rounding (condition < 10)
        assert st.converged and res <= 1.001 * TOL, (prec, st, res)


@pytest.mark.parametrize("n", [[200, 130], [60, 50, 40]])
def test_scaling_by_a_power_of_two_changes_no_bit(ctx, n):
    want = _solve(ctx, n, "dirc", False, "mixed", guess=False)
    for k in (-60, 70):
        got = _solve(ctx, n, "dirc", False, "mixed", scale=2.0 ** k, guess=False)
        assert got[0].niter == want[0].niter
        assert np.array_equal(got[2], want[2] * 2.0 ** k)


@pytest.mark.parametrize("n", [[200, 130], [60, 50, 40]])
def test_residuals_that_are_subnormal_in_float32(ctx, n):
    # values around 2^-130 in float32: 19 bits and fewer, still a preconditioner
    st, res, _ = _solve(ctx, n, "dirc", False, "mixed", scale=2.0 ** -130, guess=False, tol=1e-2)
    assert st.converged and res <= 1.001e-2, (st, res)


@pytest.mark.parametrize("n", [[130], [70, 50], [40, 33, 19]])
@pytest.mark.parametrize("k", [-900, 900])
def test_array_levels_scaled_to_the_ends_of_the_range(ctx, n, k):
    # the diagonal's exponent leaves the range of the six-operation quotient: IEEE divisions, the same bits
    want = _solve(ctx, n, "dirc", True, "fp64", guess=False)
    got = _solve(ctx, n, "dirc", True, "fp64", guess=False, A=2.0 ** k)
    assert got[0].niter == want[0].niter
    assert np.array_equal(got[2], want[2] * 2.0 ** -k)


@pytest.mark.parametrize("n,bc", [
    ([9, 1], "per"), ([1, 9], "per"), ([300, 1], "per"), ([1, 1], "per"),
    ([9, 1, 8], "per"), ([1, 8, 9], "per"), ([40, 9, 1], "per"), ([70, 1, 50], "per"), ([7, 1, 1], "per"),
    ([9, 1], "neum"), ([1, 9], "neum"), ([9, 1, 8], "neum"), ([40, 9, 1], "dirc"),
])
@pytest.mark.parametrize("array", [False, True])
def test_directions_of_one_cell(ctx, n, bc, array):
    # a periodic direction of one cell: the cell is its own neighbour on both sides
    for prec in ("mixed", "fp64"):
        st, res, _ = _solve(ctx, n, bc, array, prec)
        assert st.converged and res <= 1.001 * TOL, (prec, st, res)
