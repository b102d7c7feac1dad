"""The register-marching 2D multigrid strips against the chunked V-cycle, bit for bit, where strips can go
wrong: extents around a strip's width (56 columns, 54 on node-centred levels) and height, odd rows and
columns, levels a strip covers alone, every sweep count, boundary rows that differ in their centre
coefficient only (cell-centred, Dirichlet nodes) or in others too (Neumann nodes), mixed batches."""
import numpy as np
import pytest

import common as cm
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu

BC = {"neum": capi.BC_NEUM, "dirc": capi.BC_DIRC, "per": capi.BC_PERIODIC}


def _solve(ctx, monkeypatch, n, bc, loc, sweeps, chunked):
    for k in ("OPFLOW_MG_TILES", "OPFLOW_MG_BOTTOM"):
        if chunked:
            monkeypatch.setenv(k, "0")
        else:
            monkeypatch.delenv(k, raising=False)
    center = loc == capi.CENTER
    mesh = cm.mesh_uniform([m + 1 if center or bc == "per" else m for m in n])
    fd = cm.field_desc(2, loc, [(BC[bc], BC[bc])] * 2, ext=1 if center or bc == "neum" else 0)
    p, f = api.CartesianField(mesh, fd, ctx), api.CartesianField(mesh, fd, ctx)
    a = f.download()
    sl = f.index_slices(f.assignableRange)
    v = np.random.default_rng(n[0] * 7 + n[1]).standard_normal(a[sl].shape)
    a[sl] = v
    f.upload(a)
    # a Helmholtz operator: every boundary condition gives a regular system
    getter = lambda e: f == e - 0.01 * (api.d2x(e) + api.d2y(e))
    st = api.Solve(getter, p, api.StructSolverParams(tol=1e-9, maxIter=6, precision="mixed", preSweeps=sweeps[0], postSweeps=sweeps[1],
                                                     zeroGuess=True))
    return st.niter, st.relerr, p.download()


@pytest.mark.parametrize("n,bc,loc,sweeps", [
    ([56, 40], "neum", capi.CENTER, (2, 2)),
    ([57, 41], "dirc", capi.CENTER, (2, 2)),
    ([113, 31], "dirc", capi.CENTER, (2, 2)),
    ([40, 300], "neum", capi.CENTER, (2, 2)),
    ([301, 263], "dirc", capi.CENTER, (1, 1)),
    ([170, 129], "neum", capi.CENTER, (3, 3)),
    ([170, 129], "dirc", capi.CENTER, (4, 4)),
    ([170, 129], "dirc", capi.CENTER, (1, 3)),
    ([128, 96], "per", capi.CENTER, (2, 2)),
    ([65, 65], "dirc", capi.CORNER, (2, 2)),
    ([129, 257], "dirc", capi.CORNER, (3, 2)),
    ([129, 129], "neum", capi.CORNER, (2, 2)),
    ([257, 65], "neum", capi.CORNER, (1, 1)),
])
def test_strips_match_the_chunked_v_cycle(ctx, monkeypatch, n, bc, loc, sweeps):
    want = _solve(ctx, monkeypatch, n, bc, loc, sweeps, True)
    got = _solve(ctx, monkeypatch, n, bc, loc, sweeps, False)
    assert got[0] == want[0] and got[1] == want[1]
    assert np.array_equal(got[2], want[2]), np.abs(got[2] - want[2]).max()
