"""float32 <-> float64 by integer operations (csrc/f32bits.h) against the conversions, on the CPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "f32bits.h"
using namespace opg;
extern "C" void widen(const uint32_t* a, uint64_t* r, uint8_t* ok, long n) {
    for (long k = 0; k < n; ++k) {
        const Bits64 w = f32_to_f64_bits(a[k]);
        r[k] = (uint64_t) w.hi << 32 | w.lo;
        ok[k] = f32_plain(a[k]);
    }
}
extern "C" void narrow(const uint64_t* a, uint32_t* r, uint8_t* ok, long n) {
    for (long k = 0; k < n; ++k) {
        r[k] = f64_to_f32_bits((uint32_t) (a[k] >> 32), (uint32_t) a[k]);
        ok[k] = f64_plain((uint32_t) (a[k] >> 32), (uint32_t) a[k]);
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("bits")
    (d / "b.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "opflow_gb300", "csrc"), str(d / "b.cpp"), "-o", str(d / "b.so")])
    return ctypes.CDLL(str(d / "b.so"))


def _run(fn, a, out):
    r, ok = np.zeros(a.shape, out), np.zeros(a.shape, np.uint8)
    fn(*(ctypes.c_void_p(x.ctypes.data) for x in (a, r, ok)), ctypes.c_long(a.size))
    return r, ok.astype(bool)


def test_widening(lib):
    rng = np.random.default_rng(1)
    exps = (np.arange(256, dtype=np.uint32) << 23)[:, None]
    a = (exps | rng.integers(0, 1 << 23, (256, 2000), dtype=np.uint32)).ravel()
    a = np.concatenate([a, exps.ravel(), (exps | 0x7FFFFF).ravel()])
    a = np.concatenate([a, a | np.uint32(1 << 31)])
    r, ok = _run(lib.widen, a, np.uint64)
    with np.errstate(all="ignore"):
        want = a.view(np.float32).astype(np.float64).view(np.uint64)
    assert np.array_equal(r[ok], want[ok])
    e = (a >> 23) & 0xFF
    assert np.array_equal(ok, ((e > 0) & (e < 255)) | ((a << np.uint32(1)) == 0))


def test_narrowing(lib):
    rng = np.random.default_rng(2)
    exps = (np.arange(2048, dtype=np.uint64) << np.uint64(52))[:, None]
    m = rng.integers(0, 1 << 52, (2048, 300), dtype=np.uint64)
    half = np.uint64(1 << 28)
    keep = ~np.uint64((1 << 29) - 1)
    tails = [m, (m & keep) | half, ((m & keep) | half) - np.uint64(1), (m & keep) | (half + np.uint64(1)), m & keep, m | ~keep,
             m | np.uint64((1 << 52) - (1 << 29))]
    a = np.concatenate([(exps | (t & np.uint64((1 << 52) - 1))).ravel() for t in tails] + [exps.ravel()])
    a = np.concatenate([a, a | np.uint64(1 << 63)])
    r, ok = _run(lib.narrow, a, np.uint32)
    with np.errstate(all="ignore"):
        want = a.view(np.float64).astype(np.float32).view(np.uint32)
    assert np.array_equal(r[ok], want[ok])
    e = ((a >> np.uint64(52)) & np.uint64(0x7FF)).astype(int)
    assert np.array_equal(ok, ((e >= 897) & (e <= 1150)) | ((a << np.uint64(1)) == 0))
