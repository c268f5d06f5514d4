"""The branch-free reciprocal and square root of the assembly kernels
(asm_dmma.cuh) against CUDA's correctly rounded ones, bit for bit, over the range that the
kernels' fast path admits ([2^-900, 2^900), a reciprocal's low word not all ones, which
they check before they use it), and the refined form's FP32 reciprocal against
CUDA's, to an ulp. A small program includes the kernels' own header and counts
the differences on the device."""
import subprocess

import pytest

from rbf_b200 import build as B

pytestmark = pytest.mark.gpu

PROGRAM = r'''
#include <cstdio>
#include "asm_refined.cuh"
using namespace rbfb;
typedef unsigned long long u64;

__device__ u64 mix(u64 z) {  // splitmix64
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ bool in_range(double v) { return dm::mag_word(v) >= dm::kLow && dm::mag_word(v) < dm::kHigh; }
__device__ double step(double v, long long ulps) {
    return __longlong_as_double(__double_as_longlong(v) + ulps);
}
// the exponent of operand i: every one of the range in turn
__device__ double scaled(double m, u64 i) { return scalbn(m, (int)(i % 1800) - 900); }

// Operand i of a family: 0 random mantissas; 1 next to 1 and 2; 2 next to squares; 3
// next to what a rounding midpoint is the root of; 4 next to what one is the reciprocal of
__device__ double operand(int family, u64 i) {
    const double m = __longlong_as_double((long long)((mix(i) >> 12) | 0x3ff0000000000000ull));  // [1, 2)
    const long long off = (long long)(mix(~i) % 9) - 4;
    if (family == 0) return scaled(m, i / 7);
    if (family == 1) {
        const long long ulps = (long long)(i >> 12) % (1 << 20);
        return scaled(i & 1 ? step(1.0, ulps) : step(2.0, -1 - ulps), i / 2);
    }
    if (family == 2) {
        const double r = __longlong_as_double(__double_as_longlong(m) & ~0x3ffffffll);  // 26 bits: r * r is exact
        return scaled(step(r * r, off), i / 7);
    }
    const double half = ldexp(1.0, -53);  // half an ulp of m
    if (family == 3) return scaled(step(fma(m, m, 2.0 * m * half), off), 2 * (i / 7));
    return scaled(step(__drcp_rn(m) * (1.0 - half / m), off), i / 7);
}

__global__ void count64(int family, u64 n, u64* bad) {
    u64 b[3] = {0, 0, 0};
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const double a = operand(family, i);
        if (!in_range(a)) continue;
        ++b[2];
        const double s = mix(i ^ 0x55) & 1 ? -a : a;
        if (__double2loint(s) != -1)
            b[0] += __double_as_longlong(dm::rcp_fast(s)) != __double_as_longlong(__drcp_rn(s));
        b[1] += __double_as_longlong(dm::sqrt_fast(a)) != __double_as_longlong(__dsqrt_rn(a));
    }
    for (int j = 0; j < 3; ++j) atomicAdd(bad + j, b[j]);
}

__global__ void count32(u64* worst) {  // every mantissa at every fourth exponent of the range
    int w = 0;
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < (60ull << 23); i += (u64)gridDim.x * blockDim.x) {
        const unsigned word = (((unsigned)(i >> 23) * 4 + 7) << 23) | (unsigned)(i & 0x7fffff);
        if (word >= ir::kHigh32) continue;
        const float a = __uint_as_float(word);
        const int d = (int)__float_as_uint(ir::rcp_fast(a)) - (int)__float_as_uint(__frcp_rn(a));
        w = max(w, abs(d));
    }
    atomicMax(worst, (u64)w);
}

int main() {
    u64 *d, h[3], w = 0;
    cudaMalloc(&d, 4 * sizeof(u64));
    const u64 n[5] = {1ull << 31, 1ull << 29, 1ull << 29, 1ull << 29, 1ull << 29};
    for (int f = 0; f < 5; ++f) {
        cudaMemset(d, 0, 4 * sizeof(u64));
        count64<<<148 * 16, 256>>>(f, n[f], d);
        if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
        std::printf("family %d rcp %llu sqrt %llu of %llu\n", f, h[0], h[1], h[2]);
    }
    cudaMemset(d, 0, 4 * sizeof(u64));
    count32<<<148 * 16, 256>>>(d);
    if (cudaMemcpy(&w, d, sizeof(w), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    std::printf("fp32 %llu\n", w);
    return 0;
}
'''


def test_reciprocal_and_root_are_correctly_rounded(torch_cuda, tmp_path):
    src, exe = tmp_path / "count.cu", tmp_path / "count"
    src.write_text(PROGRAM)
    r = subprocess.run([B.nvcc()] + B.NVCC_FLAGS + [str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    lines = r.stdout.strip().splitlines()
    assert len(lines) == 6
    for line in lines[:5]:
        f = line.split()
        assert int(f[7]) > 1 << 28, line  # operands in range
        assert (f[3], f[5]) == ("0", "0"), line
    assert int(lines[5].split()[1]) <= 1, lines[5]
