"""The library's host side over a CUDA runtime without a device (tests/fake_cuda): calls that have to
survive, and what they allocate, upload and wait for.  Each runs in a process of its own."""
import glob
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEAD = """
import ctypes as C, sys
sys.path[:0] = %r
from opflow_gb300 import _capi as capi
capi.LIB_PATH = sys.argv[1]
from opflow_gb300 import api
import common as cm
count = lambda name: C.c_int.in_dll(capi.lib(), "fake_" + name)
ctx = api.Context(0)
def field(dims, loc=capi.CORNER, bc=capi.BC_DIRC, ext=0, ctx=ctx):
    return api.CartesianField(cm.mesh_uniform(list(dims)), cm.field_desc(len(dims), loc, [(bc, bc)] * len(dims), ext=ext), ctx)
""" % [ROOT, os.path.join(ROOT, "tests")]


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from opflow_gb300 import build
    build.build()
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    out = str(tmp_path_factory.mktemp("fake") / "lib.so")
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", inc, os.path.join(ROOT, "tests", "fake_cuda", "fake_cudart.cpp")] +
                          sorted(glob.glob(os.path.join(build.BUILD, "*.o"))) + ["-o", out])
    return out


def _run(lib, code):
    r = subprocess.run([sys.executable, "-c", HEAD + code, lib], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-2000:])


def test_a_batch_with_fields_that_have_nothing_to_assign(fake):
    # node-centred Dirichlet fields of two nodes along a direction: every node is a boundary node
    _run(fake, """
work = [(u, cm.ftcs_expr(u, 0.01, len(d))) for d in [(2, 8), (8, 2), (9, 9), (8, 2, 8), (2, 8, 8), (8, 8, 2), (9, 8, 7)] for u in [field(d)]]
api.assign_batch(work, steps=2)
""")


def test_march_length_of_an_empty_box(tmp_path):
    from opflow_gb300 import build
    src = tmp_path / "t.cu"
    src.write_text("""#include "stencil_exact.h"
int main() {
    for (int d = 0; d < 3; ++d)
        for (int nd = 2; nd <= 3; ++nd)
            for (int empty = 0; empty < 2; ++empty) {
                opg::Box b;
                for (int q = 0; q < nd; ++q) b.hi[q] = 9;
                if (empty) b.hi[d] = b.lo[d];
                const int m = opg::exact_march(b, nd, 152, empty ? 0. : 1.);
                if (m < 4 || m > 32) return 1;
            }
    return 0;
}
""")
    exe = str(tmp_path / "t")
    subprocess.check_call([build._nvcc(), "-O0", "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, str(src), "-o", exe] + build.ARCH)
    assert subprocess.run([exe]).returncode == 0


def test_a_failed_padding_leaves_the_field_to_be_padded(fake):
    # every allocation of a batched assignment fails once; the next call pads all the same
    _run(fake, """
u, v = field((9, 9)), field((9, 9))
failed = 0
for n in range(1, 20):
    u.upload(u.download(), update_padding=False)
    count("fail_alloc").value = n
    try:
        api.assign_batch([(u, 2.0 * v)])
    except capi.OpflowError as e:
        assert e.code == capi.E_NOMEM
        failed += 1
    done = count("fail_alloc").value > 0
    count("fail_alloc").value = 0
    if done:
        break
    at = count("launches").value
    api.assign_batch([(u, 2.0 * v)])
    assert count("launches").value - at == 2, (n, count("launches").value - at)  # the assignment and the boundary nodes
    at = count("launches").value
    api.assign_batch([(u, 2.0 * v)])
    assert count("launches").value - at == 1, n  # which hold their values now
assert failed >= 2
""")


def test_programs_given_up_early_are_those_that_do_not_fit(fake, tmp_path):
    # around the kernel's limit, of loads, constants, negations, quotients and values of one direction
    from opflow_gb300 import build
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text("""#include "tape.h"
#include <cstdio>
using namespace opg;
int main() {
    int early = 0, fit = 0;
    for (int n = 100; n <= 900; n += 7)
        for (int kind = 0; kind < 4; ++kind)
            for (int hoist = 0; hoist < 2; ++hoist) {
                Tape T;
                FieldView f{};
                f.sy = 100;
                f.sz = 10000;
                int v = T.cst(0.5);
                bool gave_up = false;
                for (int q = 0; q < n; ++q) {
                    const int off[3] = {q % 90, q / 90, 0};
                    int t = kind == 1 ? T.bin(T_MUL, T.pos(T_X, q & 1, q % 5), T.cst(1. + q)) : T.load(0, f, off);
                    if (kind == 2) t = T.neg(t);
                    if (kind == 3) t = T.bin(T_DIV, t, T.bin(T_ADD, T.pos(T_X, 0, 0), T.cst(q)));
                    v = T.bin(q % 3 ? T_ADD : T_SUB, v, t);
                    gave_up = gave_up || T.too_long();
                }
                T.out(T_OUT, 0, v);
                Box b;
                b.hi[0] = b.hi[1] = 50;
                const bool ok = T.finish(b, hoist);
                if (gave_up && ok) return printf("%d values of kind %d\\n", n, kind), 1;
                early += gave_up;
                fit += ok;
            }
    return early > 0 && fit > 0 ? 0 : 2;
}
""")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", build.CSRC, "-I", inc, str(src), fake, "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
