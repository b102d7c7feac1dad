"""The exact FTCS strips (a warp per tile of 30 columns) against the oracle, bit for bit: extents around a
tile's edges, power-of-two and other spacings and mixes of them, every order of the terms, subnormal and
huge values (the division's slow path for a power of two), the one significand for which the two-operation
division by 1/300 is off, and batches of uneven 2D and 3D grids."""
from fractions import Fraction

import numpy as np
import pytest

import common as cm
import oracle_lib as orc
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu


def _field(ctx, dims, values, seed):
    D = len(dims)
    mesh = cm.mesh_uniform(list(dims))
    fd = cm.field_desc(D, capi.CORNER, [(capi.BC_DIRC, capi.BC_DIRC)] * D)
    h = orc.HostField(mesh, fd)
    rng = np.random.default_rng(seed)
    a = values(rng, h.data[h.slices(h.assignable())].shape)
    h.data[h.slices(h.assignable())] = a
    h.update_padding()
    u = api.CartesianField(mesh, fd, ctx)
    u.upload(h.data, update_padding=False)
    return u, h


def _expr(u, dims, order):
    ops = [api.d2x, api.d2y, api.d2z]
    t = ops[order[0]](u)
    for d in order[1:]:
        t = t + ops[d](u)
    return u + 0.1 * (1.0 / (max(dims) - 1)) ** 2 * t


def _check(ctx, dims, order, values, steps=2, seed=3):
    u, h = _field(ctx, dims, values, seed)
    u.assign(_expr(u, dims, order), steps=steps)
    nodes, _ = api.serialize(_expr(cm.Leaf("u"), dims, order))
    for _ in range(steps):
        orc.assign(h, nodes, [h])
    got = u.download()
    assert np.array_equal(got, h.data, equal_nan=True), np.abs(got - h.data).max()


def _uniform(rng, shape):
    return rng.random(shape)


def _wild(rng, shape):
    """values over the whole exponent range, zeros and subnormals among them"""
    v = rng.standard_normal(shape) * 2.0 ** rng.integers(-1040, 900, shape)
    v[rng.random(shape) < 0.1] = 0.0
    return v


@pytest.mark.parametrize("dims", [(32, 32), (33, 5), (3, 40), (62, 35), (63, 33), (65, 129), (301, 50), (5, 3)])
@pytest.mark.parametrize("values", [_uniform, _wild])
def test_2d_strips_match_the_oracle(ctx, dims, values):
    for order in ((0, 1), (1, 0)):
        _check(ctx, dims, order, values)


@pytest.mark.parametrize("dims", [(33, 9, 17), (32, 6, 7), (65, 33, 9), (3, 3, 3), (61, 70, 40), (5, 65, 37), (301, 7, 6)])
@pytest.mark.parametrize("values", [_uniform, _wild])
def test_3d_strips_match_the_oracle(ctx, dims, values):
    for order in ((0, 1, 2), (2, 0, 1), (1, 2, 0)):
        _check(ctx, dims, order, values)


def test_the_significand_for_which_two_operations_are_not_enough(ctx):
    # x / h against fma(x, ch, x * cl) in exact arithmetic, near the quotients that fall next to a boundary
    h = 1.0 / 300
    ch = 1.0 / h
    cl = float((Fraction(1) - Fraction(ch) * Fraction(h)) / Fraction(h))
    H = int(h * 2.0 ** (52 - (np.frexp(h)[1] - 1)))
    bad = []
    for E in (53, 54):
        for j in range(-8, 9, 1):
            if j == 0 or H % 2 == 0:
                continue
            M = (-j * pow(H, -1, 1 << E)) % (1 << E)
            if M < (1 << 53):
                M += 1 << E
            if M >= (1 << 54) or M % 2 == 0:
                continue
            X = (M * H + j) >> E
            if (1 << 52) <= X < (1 << 53):
                two = float(Fraction(X) * Fraction(ch) + Fraction(float(X) * cl))
                if two != float(X) / h:
                    bad.append(X)
    assert len(bad) == 1, bad
    v = float(bad[0]) * 2.0 ** -60

    def values(rng, shape):
        a = np.zeros(shape)
        a[..., 1::3] = v  # neighbours are 0, so the differences along x are +-v
        a[..., 0] = -v
        return a
    _check(ctx, (301, 7), (0, 1), values, steps=1)
    _check(ctx, (301, 6, 5), (0, 1, 2), values, steps=1)


def test_batched_2d_and_3d_grids_match_their_own_assignments(ctx):
    sizes = [(33, 31), (301, 64), (17, 18, 19), (65, 65, 33), (3, 3), (129, 65)]
    fs, gs = [], []
    for k, dims in enumerate(sizes):
        fs.append(_field(ctx, dims, _uniform if k % 2 else _wild, 50 + k)[0])
        gs.append(_field(ctx, dims, _uniform if k % 2 else _wild, 50 + k)[0])
    order = [(0, 1), (1, 0), (0, 1, 2), (2, 1, 0), (0, 1), (0, 1)]
    api.assign_batch([(u, _expr(u, d, o)) for u, d, o in zip(fs, sizes, order)], steps=3)
    for u, d, o in zip(gs, sizes, order):
        u.assign(_expr(u, d, o), steps=3)
    for a, b in zip(fs, gs):
        assert np.array_equal(a.download(), b.download(), equal_nan=True)
