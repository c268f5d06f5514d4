// spmv.cu -- applying an assembled operator: out = A u over the fixed-width
// CSR (ja, values) of the assembly, then the boundary fix out[b] = u[b] for the
// listed boundary rows. The reference sketches exactly this step after its
// assembly (A.spmv(x, y) and the parallel_for over boundary nodes,
// src/main.cpp:57-66), with neither piece implemented.
//
// A row's k products are summed in row order with fused multiply-adds from
// zero: acc = fma(values[s*k+j], u[ja[s*k+j]], acc), j = 0..k-1. The order is
// pinned so the result is reproducible (the CPU oracle does the same).
#include <cuda_runtime.h>

#include <algorithm>

#include "row_sum.cuh"
#include "runtime.h"
#include "stream_copy.cuh"

namespace rbfb {

// A warp takes kTileRows rows (32 of short rows): their entries, one piece of ja
// and values, are copied into shared memory with 16-byte asynchronous copies
// under an L2 evict-first policy, and each lane sums its own row from there,
// eight gathers of u in flight. A thread-per-row walk of global memory touches a
// line per lane and load: 1.6 GB through the L1s for 437 MB of operator, and the
// L1 bound it. 16 rows a warp leave room for 32 warps per SM. 1M rows, k = 35:
// 128 -> 79 us (5.5 TB/s of the operator's bytes); 32 rows a warp, 16 warps: 92.
// k a multiple of 4 would put the rows of all lanes on a few banks: they are
// copied one by one with padding (PAD).
constexpr int kSpmvWarps = 4, kTileRows = 16;
struct TileShape {
    int rows;    // rows a warp
    int kv, kj;  // entries from a row to the next in shared memory: weights, columns
    __host__ __device__ size_t warp_bytes() const {
        return (static_cast<size_t>(rows) * kv + 4) / 2 * 16 + (static_cast<size_t>(rows) * kj + 7) / 4 * 16;
    }
};
inline TileShape tile_shape(int k) {
    // 48 entries a row, padded: 8 rows 31.6 us (150k rows), 16 33.6
    TileShape t{k <= 17 ? 32 : k % 4 == 0 && k >= 44 ? 8 : kTileRows, k, k};
    if (k % 4 == 0) {
        t.kv = k + 2;
        t.kj = k / 4 % 2 ? k : k + 4;
    }
    return t;
}

template <bool PAD>
__global__ void __launch_bounds__(kSpmvWarps * 32, 8)
    spmv_tiled_kernel(int n, int k, TileShape t, const int* __restrict__ ja,
                      const double* __restrict__ values, const double* __restrict__ u,
                      double* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char spmv_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double* sv = reinterpret_cast<double*>(spmv_smem + wid * t.warp_bytes());
    int* sj = reinterpret_cast<int*>(sv + (t.rows * t.kv + 4) / 2 * 2);
    const unsigned long long pol = evict_first_policy();
    const int tiles = (n + t.rows - 1) / t.rows;
    // PAD: this lane's first 16-byte chunk of weights and of columns, and the step
    // of 32 chunks, as (row, chunk in the row)
    const int cv = k / 2, cj = k / 4;
    for (int tile = blockIdx.x * kSpmvWarps + wid; tile < tiles; tile += gridDim.x * kSpmvWarps) {
        const int s0 = tile * t.rows, rows = min(t.rows, n - s0);
        const long long q0 = static_cast<long long>(s0) * k, qa = PAD ? q0 : q0 & ~3LL;
        const int m = static_cast<int>(q0 - qa) + rows * k;
        const double* gv = values + qa;
        const int* gj = ja + qa;
        if constexpr (PAD) {
            for (int c = lane, r = lane / cv, i = lane - r * cv; c < m / 2; c += 32) {
                cp_async_stream<16>(sv + r * t.kv + 2 * i, gv + 2 * c, pol);
                for (i += 32; i >= cv; i -= cv) ++r;
            }
            for (int c = lane, r = lane / cj, i = lane - r * cj; c < m / 4; c += 32) {
                cp_async_stream<16>(sj + r * t.kj + 4 * i, gj + 4 * c, pol);
                for (i += 32; i >= cj; i -= cj) ++r;
            }
        } else {
            for (int c = lane; c < m / 2; c += 32) cp_async_stream<16>(sv + 2 * c, gv + 2 * c, pol);
            if ((m & 1) && lane == 0) cp_async_stream<8>(sv + m - 1, gv + m - 1, pol);
            for (int c = lane; c < m / 4; c += 32) cp_async_stream<16>(sj + 4 * c, gj + 4 * c, pol);
            for (int e = (m & ~3) + lane; e < m; e += 32) cp_async_stream<4>(sj + e, gj + e, pol);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncwarp();
        if (lane < rows) {
            const int lead = static_cast<int>(q0 - qa);
            const double* v = sv + lead + lane * t.kv;
            const int* j = sj + lead + lane * t.kj;
            double acc = 0.0;
            int i = 0;
#pragma unroll 1
            for (; i + 8 <= k; i += 8) {
                double x[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) x[c] = __ldg(u + j[i + c]);
#pragma unroll
                for (int c = 0; c < 8; ++c) acc = fma(v[i + c], x[c], acc);
            }
            for (; i < k; ++i) acc = fma(v[i], __ldg(u + j[i]), acc);
            out[s0 + lane] = acc;
        }
        __syncwarp();  // the slab is refilled
    }
}

// Unaligned arrays and very long rows: one thread per row (row_sum).
__global__ void spmv_fixed_kernel(int n, int k, const int* __restrict__ ja,
                                  const double* __restrict__ values, const double* __restrict__ u,
                                  double* __restrict__ out, bool vec) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const long long q = static_cast<long long>(s) * k;
        out[s] = row_sum(ja, values, q, q + k, vec, [u](int j) { return __ldg(u + j); });
    }
}

constexpr int kTiledMaxK = 128;  // above: the slabs leave too few warps

int launch_spmv(int n, int k, const int* ja, const double* values, const double* u, double* out,
                cudaStream_t st) {
    const bool vec = rows_vectorizable(ja, values);
    if (!vec || k > kTiledMaxK) {
        const int blocks = std::min((n + 255) / 256, 148 * 16);
        spmv_fixed_kernel<<<blocks, 256, 0, st>>>(n, k, ja, values, u, out, vec);
        return RBFB_OK;
    }
    const TileShape t = tile_shape(k);
    const size_t smem = kSpmvWarps * t.warp_bytes();
    auto* kern = k % 4 == 0 ? &spmv_tiled_kernel<true> : &spmv_tiled_kernel<false>;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(smem)) != cudaSuccess)
        return RBFB_ECUDA;
    const int per_block = kSpmvWarps * t.rows;
    const int blocks = std::min((n + per_block - 1) / per_block, 148 * 64);
    kern<<<blocks, kSpmvWarps * 32, smem, st>>>(n, k, t, ja, values, u, out);
    return RBFB_OK;
}

__global__ void boundary_fix_kernel(int nb, const int* __restrict__ bnd,
                                    const double* __restrict__ u, double* __restrict__ out) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x)
        out[bnd[b]] = u[bnd[b]];
}

}  // namespace rbfb

extern "C" int rbfb_spmv(int n, int k, const int* ja, const double* values, const double* u,
                         double* out, const int* bnd, int nbnd, void* stream) {
    if (n < 0 || k < 1 || nbnd < 0 || (n > 0 && (!ja || !values || !u || !out)) ||
        (nbnd > 0 && !bnd))
        return RBFB_EINVAL;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n > 0) {
        const int rc = rbfb::launch_spmv(n, k, ja, values, u, out, st);
        if (rc) return rc;
    }
    if (nbnd > 0) {
        const int blocks = std::min((nbnd + 255) / 256, 148 * 4);
        rbfb::boundary_fix_kernel<<<blocks, 256, 0, st>>>(nbnd, bnd, u, out);
    }
    return cudaGetLastError() == cudaSuccess ? RBFB_OK : RBFB_ECUDA;
}
