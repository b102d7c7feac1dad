"""The float64 quotients built from fused operations (f64div.h) against the device's IEEE division, bit for
bit (quotient(): a neighbour where the quotient is made to lie near the middle of two numbers): operands over the whole range with quotients that overflow, underflow and lie near the middle of two
numbers, zeros, subnormals, infinities and NaN."""
import subprocess

import pytest

from opflow_gb300 import build

SRC = r"""
#include <cstdio>
#include "f64div.h"
using namespace opg;
__device__ double bits(unsigned long long b) { return __longlong_as_double((long long) b); }
__device__ unsigned long long mix(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__global__ void check(long long n, unsigned long long* bad, double* first) {
    const double special[] = {0., 5e-324, 1e-310, 2.2250738585072014e-308, 1e-200, 1., 3., 1.7976931348623157e308, bits(0x7FF0000000000000ull), bits(0x7FF8000000000000ull)};
    for (long long t = blockIdx.x * (long long) blockDim.x + threadIdx.x; t < n; t += (long long) gridDim.x * blockDim.x) {
        const unsigned long long u = mix(2 * t + 1), v = mix(2 * t + 2), w = mix(u ^ v);
        double a = bits(u), b = bits(v);
        switch (w & 7) {
            case 0: break;                                                        // any bits at all
            case 1: a = special[(w >> 8) % 10]; if (w & 1024) a = -a; break;
            case 2: b = special[(w >> 8) % 10]; if (w & 1024) b = -b; break;
            case 3: a = special[(w >> 8) % 10]; b = special[(w >> 16) % 10]; if (w & 1024) b = -b; break;
            case 4: {                                                             // ordinary exponents
                a = bits((u & 0x800FFFFFFFFFFFFFull) | (1000 + (w >> 8) % 46) << 52);
                b = bits((v & 0x800FFFFFFFFFFFFFull) | (1000 + (w >> 16) % 46) << 52);
                break;
            }
            case 5: {                                                             // quotients near a middle
                b = bits((v & 0x800FFFFFFFFFFFFFull) | (1000 + (w >> 16) % 46) << 52);
                const double q = bits((u & 0xFFFFFFFFFFFFFull) | 1023ull << 52);
                a = __fma_rn(b, q, b * 1.1102230246251565e-16);                   // b (q + ulp(q) / 2)
                break;
            }
            case 6: b = bits((v & 0x800FFFFFFFFFFFFFull) | 1020ull << 52); a = b * (1. + (double) (int) ((w >> 8) % 9 - 4) * 2.220446049250313e-16); break;
            default: {                                                            // both in the range, the quotient at its ends or beyond
                a = bits((u & 0x800FFFFFFFFFFFFFull) | ((w & 8 ? 1760 : 210) + (w >> 8) % 40) << 52);
                b = bits((v & 0x800FFFFFFFFFFFFFull) | ((w & 8 ? 210 : 1760) + (w >> 16) % 560) << 52);
            }
        }
        const double want = __ddiv_rn(a, b);
        const double got[2] = {quotient(a, b), div_rn<true>(a, b, recip_fast(b))};
        for (int q = 0; q < 2; ++q) {
            // (elsewhere quotient() rounds one in 2^50 otherwise; 2^27 are tried)
            const long long off = __double_as_longlong(got[q]) - __double_as_longlong(want), slack = q == 0 && ((w & 7) == 5 || (w & 7) == 6);
            if ((off > slack || off < -slack) && !(got[q] != got[q] && want != want) && atomicAdd(&bad[q], 1ull) == 0) {
                first[3 * q] = a;
                first[3 * q + 1] = b;
                first[3 * q + 2] = got[q];
            }
        }
    }
}
int main() {
    struct { unsigned long long bad[2]; double first[6]; } h, *d;
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 2;
    check<<<608, 256>>>(1ll << 27, d->bad, d->first);
    if (cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    for (int q = 0; q < 2; ++q)
        if (h.bad[q]) printf("%d: %llu differ, first %a / %a: %a\n", q, h.bad[q], h.first[3 * q], h.first[3 * q + 1], h.first[3 * q + 2]);
    return h.bad[0] || h.bad[1];
}
"""


@pytest.mark.gpu
def test_quotients_are_the_ieee_ones(ctx, tmp_path):
    src, exe = tmp_path / "t.cu", str(tmp_path / "t")
    src.write_text(SRC)
    subprocess.check_call([build._nvcc()] + build.NVCC_FLAGS + ["-I", build.CSRC, str(src), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
