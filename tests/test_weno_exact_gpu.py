"""The fused WENO5-RK3 kernel's divisions and folded operations against the oracle, bit for bit: line
lengths around a thread's points, power-of-two and other spacings (1/300 leaves one significand out of the
two-operation division), both sides, and values that reach every branch: smooth, jumps, constants, zeros,
and magnitudes over most of the exponent range."""
import sys

import numpy as np
import pytest

import common as cm
import oracle_lib as orc
from opflow_gb300 import _capi as capi
from opflow_gb300 import api

pytestmark = pytest.mark.gpu

VALUES = {
    "random": lambda r, s: r.random(s),
    "smooth": lambda r, s: 1.0 + 1e-3 * np.sin(2 * np.pi * np.arange(s[-1]) / s[-1]) + 0 * r.random(s),
    "jumps": lambda r, s: np.where(r.random(s) < 0.3, 1.0, 0.0),
    "constant": lambda r, s: np.full(s, 0.7),
    "integers": lambda r, s: r.integers(-4, 5, s).astype(float),
    "tiny": lambda r, s: r.standard_normal(s) * 2.0 ** r.integers(-60, -20, s),
    "tails": lambda r, s: np.exp(-np.minimum(700.0, np.arange(s[-1]) ** 2 / 3.0)) + 0 * r.random(s),
    "wide": lambda r, s: r.standard_normal(s) * 2.0 ** r.integers(-280, 240, s),
}


@pytest.mark.parametrize("n", [7, 15, 16, 17, 40, 256, 300, 1025])
@pytest.mark.parametrize("upwind", [False, True])
def test_fused_weno_matches_the_oracle(ctx, n, upwind):
    ny, steps, dt = 5, 2, 0.3 / n
    mesh = cm.mesh_uniform([n + 1, ny + 1])
    fd = cm.field_desc(2, capi.CENTER, [(capi.BC_PERIODIC, capi.BC_PERIODIC)] * 2, ext=3)
    L = [cm.Leaf(x) for x in ("u", "u1", "u2")]
    nodes = [api.serialize(e, L)[0] for e in cm.weno_stage_exprs(L[0], L[1], L[2], dt, upwind=upwind)]
    for k, (name, values) in enumerate(VALUES.items()):
        h = [orc.HostField(mesh, fd) for _ in range(3)]
        sl = h[0].slices(h[0].assignable())
        h[0].data[sl] = values(np.random.default_rng(100 + k), h[0].data[sl].shape)
        h[0].update_padding()
        u = api.CartesianField(mesh, fd, ctx)
        u.upload(h[0].data, update_padding=False)
        api.weno_rk3(u, dt, steps, upwind=upwind)
        for _ in range(steps):
            for dst, nd in zip((h[1], h[2], h[0]), nodes):
                orc.assign(dst, nd, h)
        got, want = u.download()[sl], h[0].data[sl]
        assert np.array_equal(got, want, equal_nan=True), (name, np.abs(got - want).max())


@pytest.mark.parametrize("n", [17, 97, 300])
@pytest.mark.parametrize("upwind", [False, True])
@pytest.mark.parametrize("low,high", [(-1074, -1000), (-1074, -1040), (-1060, -900)])
def test_fused_weno_below_the_normal_range(ctx, monkeypatch, n, upwind, low, high):
    values = lambda r, s: r.standard_normal(s) * 2.0 ** r.integers(low, low + 30, s) * 2.0 ** r.integers(0, high - low - 29, s)
    monkeypatch.setattr(sys.modules[__name__], "VALUES", {"subnormal": values})
    test_fused_weno_matches_the_oracle(ctx, n, upwind)
