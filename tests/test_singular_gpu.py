"""Singular (all-Neumann and periodic) problems on extents whose coarser grids do not halve evenly: every
right-hand side of many converges, in a bounded number of iterations, and its residual formed apart meets the
tolerance."""
import numpy as np
import pytest

import common as cm
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu

TOL = 1e-9


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,bc", [([129, 129], "NN"), ([257, 257], "NN"), ([333, 333], "NN"), ([257, 130], "NP"), ([66, 257], "PN"), ([65, 49, 41], "NNN"),
                                  ([33, 66, 65], "NPN")])
def test_every_right_hand_side_converges(ctx, n, bc, precision):
    D = len(n)
    kinds = {"N": (capi.BC_NEUM, capi.BC_NEUM), "P": (capi.BC_PERIODIC, capi.BC_PERIODIC)}
    fd = cm.field_desc(D, capi.CENTER, [kinds[b] for b in bc], ext=1)
    mesh = cm.mesh_uniform([m + 1 for m in n])
    p, f, w = (api.CartesianField(mesh, fd, ctx) for _ in range(3))
    sl = f.index_slices(f.assignableRange)
    lap = lambda e: sum((api.d2(e, d) for d in range(1, D)), api.d2(e, 0))
    solver = api.EqnSolveHandler(lambda e: f == lap(e), p, api.StructSolverParams(tol=TOL, maxIter=60, precision=precision, zeroGuess=True))
    for seed in range(40):
        a = f.download()
        v = np.random.default_rng(seed).standard_normal(a[sl].shape)
        a[sl] = v - v.mean()
        f.upload(a)
        st = solver.solve()
        assert st.converged, (seed, st.niter, st.relerr)
        if seed % 12 == 0:
            # (values of p around 1e4 times the equation's rounding: far below the tolerance)
            w.assign(lap(p))
            fa, wa = f.download()[sl], w.download()[sl]
            assert np.linalg.norm(fa - wa) <= 1.01 * TOL * np.linalg.norm(fa)
