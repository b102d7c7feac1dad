"""The fused 3D multigrid steps (a CTA marching a 64 x 32 patch along z) against the chunked V-cycle, bit
for bit: extents around a patch's own 56 x 24 cells, odd and small ones, one and two sweeps, Dirichlet and
Neumann, and batches that mix such levels with others."""
import numpy as np
import pytest

import common as cm
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu

BC = {"neum": capi.BC_NEUM, "dirc": capi.BC_DIRC}


def _solve(ctx, monkeypatch, n, bc, sweeps, chunked):
    if chunked:
        monkeypatch.setenv("OPFLOW_MG_ZMARCH", "0")
    else:
        monkeypatch.delenv("OPFLOW_MG_ZMARCH", raising=False)
    mesh = cm.mesh_uniform([m + 1 for m in n])
    fd = cm.field_desc(3, capi.CENTER, [(BC[bc], BC[bc])] * 3, ext=1)
    p, f = api.CartesianField(mesh, fd, ctx), api.CartesianField(mesh, fd, ctx)
    a = f.download()
    sl = f.index_slices(f.assignableRange)
    a[sl] = np.random.default_rng(sum(n)).standard_normal(a[sl].shape)
    f.upload(a)
    getter = lambda e: f == e - 0.01 * (api.d2x(e) + api.d2y(e) + api.d2z(e))
    st = api.Solve(getter, p, api.StructSolverParams(tol=1e-9, maxIter=5, precision="mixed", preSweeps=sweeps[0], postSweeps=sweeps[1], zeroGuess=True))
    return st.niter, st.relerr, p.download()


@pytest.mark.parametrize("n,bc,sweeps", [
    ([56, 24, 16], "neum", (2, 2)),
    ([57, 25, 17], "dirc", (2, 2)),
    ([112, 48, 9], "dirc", (2, 2)),
    ([113, 49, 33], "neum", (2, 2)),
    ([12, 90, 31], "dirc", (2, 2)),
    ([11, 13, 97], "neum", (2, 2)),
    ([60, 28, 40], "dirc", (1, 1)),
    ([61, 57, 21], "neum", (1, 1)),
    ([64, 30, 24], "dirc", (1, 2)),
    ([64, 30, 24], "dirc", (3, 3)),
])
def test_fused_3d_steps_match_the_chunked_v_cycle(ctx, monkeypatch, n, bc, sweeps):
    want = _solve(ctx, monkeypatch, n, bc, sweeps, True)
    got = _solve(ctx, monkeypatch, n, bc, sweeps, False)
    assert got[0] == want[0] and got[1] == want[1]
    assert np.array_equal(got[2], want[2]), np.abs(got[2] - want[2]).max()


def test_batch_of_3d_and_2d_levels_equals_each_alone(ctx):
    P = lambda n, loc, bc: api.Problem(n, [1.0 / m for m in n], alpha=1.0, beta=0.01, loc=loc, bc=bc)
    probs = [P([57, 40, 33], capi.CENTER, capi.BC_NEUM), P([33, 33, 33], capi.CORNER, capi.BC_DIRC), P([200, 90], capi.CENTER, capi.BC_DIRC),
             P([24, 24, 24], capi.CENTER, capi.BC_DIRC), P([30, 30, 30], capi.CORNER, capi.BC_NEUM)]
    par = api.StructSolverParams(tol=1e-9, maxIter=40, precision="mixed", zeroGuess=True)
    rng = np.random.default_rng(2)
    B = api.Batch(probs, par, ctx)
    fs = []
    for i in range(len(probs)):
        fs.append(rng.standard_normal(B.size(i)))
        B.set(i, fs[i])
    st = B.solve()
    for i, p in enumerate(probs):
        one = api.Batch([p], par, ctx)
        one.set(0, fs[i])
        assert one.solve()[0].niter == st[i].niter
        assert np.array_equal(one.get(0), B.get(i)), i
