"""The whole padding update in one launch against the oracle's zones in turn, bit for bit, from arrays whose
ghost cells hold other values before: every boundary condition pair on 2D and 3D corner and centre fields,
ghost layers of one to four cells, ranges narrower than the ghost layer (which keep the zones in turn), and
many fields padded together after a batched assignment."""
import itertools

import numpy as np
import pytest

import common as cm
import oracle_lib as orc
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu

BCS = [capi.BC_DIRC, capi.BC_NEUM, capi.BC_PERIODIC, capi.BC_SYMM, capi.BC_ASYMM, capi.BC_UNDEFINED]


def _case(ctx, dims, loc, bcs, ext, seed):
    mesh = cm.mesh_uniform(list(dims))
    D = len(dims)
    vals = [(0.25 * (d + 1), -0.5 - d) for d in range(D)]
    fd = cm.field_desc(D, loc, bcs, vals, ext=ext)
    h = orc.HostField(mesh, fd)
    h.data[...] = np.random.default_rng(seed).standard_normal(h.data.shape)
    f = api.CartesianField(mesh, fd, ctx)
    f.upload(h.data, update_padding=False)
    return f, h


def _pairs(rng, D):
    out = []
    for _ in range(D):
        a, b = rng.choice(BCS, 2)
        if capi.BC_PERIODIC in (a, b):
            a = b = capi.BC_PERIODIC
        out.append((int(a), int(b)))
    return out


@pytest.mark.parametrize("loc", [capi.CORNER, capi.CENTER])
@pytest.mark.parametrize("dims", [(9, 7), (6, 12), (8, 7, 9), (4, 5), (3, 4, 6)])
def test_one_launch_matches_the_zones_in_turn(ctx, dims, loc):
    rng = np.random.default_rng(sum(dims) + loc)
    D = len(dims)
    cases = [[(b, b)] * D for b in BCS] + [_pairs(rng, D) for _ in range(12)]
    for k, bcs in enumerate(cases):
        for ext in (0, 1, 2, 4):
            f, h = _case(ctx, dims, loc, bcs, ext, 100 * k + ext)
            f.updatePadding()
            h.update_padding()
            got = f.download()
            assert np.array_equal(got, h.data), (bcs, ext, np.argwhere(got != h.data)[:5])


def test_fields_padded_together_after_a_batched_assignment(ctx):
    rng = np.random.default_rng(5)
    gs, hs, work = [], [], []
    for k, (dims, loc) in enumerate(itertools.product([(9, 7), (33, 40), (8, 7, 9)], [capi.CORNER, capi.CENTER])):
        f, h = _case(ctx, dims, loc, _pairs(rng, len(dims)), k % 3, k)
        gs.append(f)
        hs.append(h)
        work.append((f, 0.5 * f + 1.25))
    api.assign_batch(work, steps=3)
    nodes, _ = api.serialize(0.5 * cm.Leaf("u") + 1.25)
    for f, h in zip(gs, hs):
        for _ in range(3):
            orc.assign(h, nodes, [h])
        assert np.array_equal(f.download(), h.data)
