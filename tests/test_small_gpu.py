"""The one-CTA V-cycle of small levels (vectors in shared memory) against the chunked V-cycle, bit for bit: 2D
and 3D, cell- and node-centred, every boundary kind, extents around its thresholds, a warp's share and odd
ones, unequal sweep counts, levels below strips, below 3D tiles and below chunked levels."""
import numpy as np
import pytest

import common as cm
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu

BC = {"neum": capi.BC_NEUM, "dirc": capi.BC_DIRC, "per": capi.BC_PERIODIC}
SWITCHES = {"OPFLOW_MG_TILES": "0", "OPFLOW_MG_BOTTOM": "0", "OPFLOW_MG_ZMARCH": "0"}


def _solve(ctx, monkeypatch, n, bc, loc, sweeps, off):
    for k, v in SWITCHES.items():
        if k in off:
            monkeypatch.setenv(k, v)
        else:
            monkeypatch.delenv(k, raising=False)
    D = len(n)
    mesh = cm.mesh_uniform([m + 1 if loc == capi.CENTER else m for m in n])
    fd = cm.field_desc(D, loc, [(BC[bc], BC[bc])] * D, ext=1 if loc == capi.CENTER else 0)
    p, f = api.CartesianField(mesh, fd, ctx), api.CartesianField(mesh, fd, ctx)
    a = f.download()
    sl = f.index_slices(f.assignableRange)
    a[sl] = np.random.default_rng(sum(n)).standard_normal(a[sl].shape)
    f.upload(a)
    d2 = (api.d2x, api.d2y, api.d2z)[:D]

    def getter(e):
        t = 1.0 * e
        for d in d2:
            t = t - 0.01 * d(e)
        return f == t
    st = api.Solve(getter, p, api.StructSolverParams(tol=1e-9, maxIter=5, precision="mixed", preSweeps=sweeps[0], postSweeps=sweeps[1], zeroGuess=True))
    return st.niter, st.relerr, p.download()


@pytest.mark.parametrize("n,bc,loc,sweeps", [
    ([96, 96], "neum", "C", (2, 2)), ([97, 96], "dirc", "C", (2, 2)), ([13, 12], "dirc", "C", (2, 2)), ([40, 230], "dirc", "C", (2, 2)),
    ([9, 700], "neum", "C", (2, 2)), ([64, 64], "per", "C", (2, 2)), ([300, 200], "per", "C", (2, 2)), ([160, 161], "neum", "C", (3, 1)),
    ([75, 51], "dirc", "N", (2, 2)), ([129, 65], "dirc", "N", (1, 2)), ([33, 200], "dirc", "N", (4, 4)), ([50, 31], "neum", "C", (1, 1)),
    ([16, 16, 16], "neum", "C", (2, 2)), ([15, 17, 13], "dirc", "C", (2, 2)), ([40, 33, 31], "dirc", "C", (2, 2)), ([9, 8, 30], "neum", "C", (1, 2)),
    ([16, 12, 20], "per", "C", (2, 2)), ([17, 15, 13], "dirc", "N", (2, 2)), ([33, 30, 25], "dirc", "N", (2, 2)), ([70, 12, 9], "dirc", "C", (3, 3)),
])
def test_small_levels_match_the_chunked_v_cycle(ctx, monkeypatch, n, bc, loc, sweeps):
    loc = capi.CENTER if loc == "C" else capi.CORNER
    want = _solve(ctx, monkeypatch, n, bc, loc, sweeps, SWITCHES)
    for off in ({}, {"OPFLOW_MG_ZMARCH"}):
        got = _solve(ctx, monkeypatch, n, bc, loc, sweeps, off)
        assert got[0] == want[0] and got[1] == want[1], (off, got[:2], want[:2])
        assert np.array_equal(got[2], want[2]), (off, np.abs(got[2] - want[2]).max())


def test_batches_of_small_problems_equal_each_alone(ctx):
    P = lambda n, loc, bc: api.Problem(n, [1.0 / m for m in n], alpha=1.0, beta=0.01, loc=loc, bc=bc)
    probs = [P([57, 40], capi.CENTER, capi.BC_NEUM), P([33, 33], capi.CORNER, capi.BC_DIRC), P([12, 14, 10], capi.CENTER, capi.BC_DIRC),
             P([96, 96], capi.CENTER, capi.BC_DIRC), P([20, 21, 22], capi.CORNER, capi.BC_NEUM), P([200, 130], capi.CENTER, capi.BC_DIRC)]
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
