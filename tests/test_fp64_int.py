"""bmxg_fp64.cuh: the FP64 square root, quotient and comparisons on the integer
pipe equal the IEEE ones bit for bit -- over random operands, short significands,
quotients and squares beside the rounding boundaries, powers of two, subnormals,
zeros, infinities and NaN -- on the host with the FP32 approximations moved to the
ends of their error range, and on the device with its own."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "boltzmannmfx_gb300", "csrc")

COMMON = r"""
#include "bmxg_fp64.cuh"
#include <cstdio>
#include <cstdlib>
using namespace bmxg;
struct Mix { uint64_t s; BMXG_HD uint64_t operator()() { uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull; z = (z ^ (z >> 27)) * 0x94D049BB133111EBull; return z ^ (z >> 31); } };
BMXG_HD bool same(double a, double b) { return bits64(a) == bits64(b) || (a != a && b != b); }
BMXG_HD int one(Mix &g, int mode)
{
    const uint64_t frac = 0xfffffffffffffull;
    uint64_t a = g(), b = g();
    if (mode < 6) {
        a = (a & ~(0x7ffull << 52)) | ((uint64_t)(983 + g() % 80) << 52);
        b = (b & ~(0x7ffull << 52)) | ((uint64_t)(983 + g() % 80) << 52);
    }
    if (mode == 1) { a &= ~(0xffffffull << (g() % 28)); b &= ~(0xfffffull << (g() % 32)); }
    if (mode == 2) { b &= ~frac; b |= (g() & 7); a = (a & ~frac) | ((0ull - (g() & 15)) & frac); }
    if (mode == 3) a = (a & ~frac) | (b & frac);
    if (mode == 4) { // a quotient beside halfway between two doubles: a = b (q + 1/2 ulp), rounded
        const double q = from_bits64((g() & frac) | 0x3ff0000000000000ull);
        a = bits64(from_bits64(b) * q + from_bits64(b) * 0x1p-53);
    }
    if (mode == 6) { const uint64_t v[8] = {0, 1, 0x10000000000000ull, 0x7ff0000000000000ull, 0x7fefffffffffffffull,
                     0x7ff8000000000000ull, 0x3ff0000000000000ull, 0xfffffffffffffull};
        a = v[g() & 7] | (g() << 63); if (g() & 1) b = v[g() & 7] | (g() << 63); }
    const double A = from_bits64(a), B = from_bits64(b);
    double X = from_bits64(a & ~(1ull << 63));
    if (mode == 5) { // a square beside halfway: (odd 54-bit)^2 rounded, a neighbour of it
        const uint64_t h = (g() >> 11) | (1ull << 53) | 1ull;
        const double d = (double)h;
        X = from_bits64(bits64(d * d) + g() % 3 - 1);
    }
    Divisor D;
    int bad = 0;
    const double s = sqrt_rn(X, &D);
    bad |= !same(s, sqrt(X));
    bad |= !same(div_rn(A, B), A / B) << 1;
    bad |= !same(div_by(B, D), B / s) << 2;
    bad |= (lt_bits(A, B) != (A < B) || le_bits(A, B) != (A <= B)) << 3;
    bad |= (le_nonneg(X, fabs(B)) != (X <= fabs(B))) << 4;
    bad |= !same(plus_zero(A), A + 0.0) << 5;
    return bad;
}
"""

HOST = COMMON + r"""
int main() {
    for (int u = -2; u <= 2; ++u) {
        host_approx::ulps() = u;
        Mix g{(uint64_t)(u + 5)};
        for (int k = 0; k < 2000000; ++k)
            if (int bad = one(g, k & 7)) { std::printf("mode %d ulps %d: %d\n", k & 7, u, bad); return 1; }
    }
    return 0;
}
"""

DEVICE = COMMON + r"""
__global__ void run(int *bad) {
    Mix g{(uint64_t)(blockIdx.x * blockDim.x + threadIdx.x) * 1000003ull + 17ull};
    for (int k = 0; k < 512; ++k) if (int b = one(g, k & 7)) atomicOr(bad, b | (1 << (8 + (k & 7))));
}
int main() {
    int *d = nullptr, h = -1;
    if (cudaMalloc(&d, 4) || cudaMemset(d, 0, 4)) return 2;
    run<<<512, 128>>>(d);
    if (cudaMemcpy(&h, d, 4, cudaMemcpyDeviceToHost)) return 3;
    std::printf("bad %x\n", h);
    return h != 0;
}
"""


def _run(cmd, exe):
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_host(tmp_path):
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text(HOST)
    _run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(src), "-o", exe], exe)


@pytest.mark.gpu
def test_device(tmp_path, gpu_lib):
    from boltzmannmfx_gb300 import build
    src, exe = tmp_path / "t.cu", str(tmp_path / "t")
    src.write_text(DEVICE)
    _run([build.nvcc(), *build.flags(), str(src), "-o", exe], exe)
