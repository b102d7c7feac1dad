"""A re-solve that keeps its matrix forms the right-hand side alone: inner cells straight from the known
field where the equation leaves nothing else there.  The solution after f changed has to be that of a
handler made afresh, bit for bit: f on either side, with and without a factor, added to other fields,
every boundary condition with values, 2D and 3D, centre and corner fields."""
import numpy as np
import pytest

import common as cm
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu

EQS = {
    "f_left": lambda f, g, L: (lambda e: f == e - 0.02 * L(e)),
    "f_right": lambda f, g, L: (lambda e: e - 0.02 * L(e) == f),
    "minus_f": lambda f, g, L: (lambda e: api.Eq(-f, 0.02 * L(e) - e)),
    "factor": lambda f, g, L: (lambda e: e - 0.02 * L(e) == 2.0 * f),
    "two_fields": lambda f, g, L: (lambda e: e - 0.02 * L(e) == f + g),
    "field_coefficient": lambda f, g, L: (lambda e: g * e - 0.02 * L(e) == f),
}


@pytest.mark.parametrize("eq", list(EQS))
@pytest.mark.parametrize("dims,loc,bc", [((40, 33), capi.CENTER, capi.BC_DIRC), ((40, 33), capi.CENTER, capi.BC_NEUM), ((33, 21), capi.CORNER, capi.BC_DIRC),
                                         ((14, 12, 16), capi.CENTER, capi.BC_DIRC), ((16, 16), capi.CENTER, capi.BC_PERIODIC), ((4, 4), capi.CENTER, capi.BC_DIRC)])
def test_a_kept_matrix_gives_the_fresh_solution(ctx, eq, dims, loc, bc):
    D = len(dims)
    mesh = cm.mesh_uniform([n + 1 if loc == capi.CENTER else n for n in dims])
    ext = 1 if loc == capi.CENTER else 0
    tgt = cm.field_desc(D, loc, [(bc, bc)] * D, [(0.5, -1.5)] * D, ext=ext)
    oth = cm.field_desc(D, loc, [(capi.BC_NEUM, capi.BC_NEUM)] * D if bc != capi.BC_PERIODIC else [(bc, bc)] * D, ext=ext)
    p, f, g = api.CartesianField(mesh, tgt, ctx), api.CartesianField(mesh, oth, ctx), api.CartesianField(mesh, oth, ctx)
    rng = np.random.default_rng(4)
    g.upload(1.0 + rng.random(g.shape))
    ops = [api.d2x, api.d2y, api.d2z][:D]
    lap = lambda e: sum((op(e) for op in ops[1:]), ops[0](e))
    getter = EQS[eq](f, g, lap)
    par = lambda static: api.StructSolverParams(tol=1e-9, maxIter=60, precision="mixed", staticMat=static, zeroGuess=True)
    f.upload(rng.standard_normal(f.shape))
    kept = api.makeEqnSolveHandler(getter, p, par(True))
    kept.solve()
    for _ in range(2):
        f.upload(rng.standard_normal(f.shape))
        a = kept.solve()
        x = p.download()
        b = api.Solve(getter, p, par(False))
        assert a.niter == b.niter and a.relerr == b.relerr
        assert np.array_equal(x, p.download())
