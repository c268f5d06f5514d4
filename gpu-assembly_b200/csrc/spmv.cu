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
// L1 bound it. 16 rows a warp leave room for 32 warps per SM. 1M rows, k = 35, the
// operator from HBM: 131 us by a thread a row, 94 so (4.5 TB/s of its bytes); again and again, what
// is in L2 of it, 128 and 83, with 32 rows and 16 warps 92.
// k a multiple of 4 would put the rows of all lanes on a few banks: their rows
// are padded by a 16-byte piece (PAD; 60,000 rows, k = 36: 9.9 us, 10.0 walked).
constexpr int kSpmvWarps = 4, kTileRows = 16;
struct TileShape {
    int rows;    // rows a warp
    int kv, kj;  // entries from a row to the next in shared memory: weights, columns
    int mv, mj;  // padded rows: 2^16 / (16-byte pieces a row), rounded up
    __host__ __device__ size_t warp_bytes() const {
        return (static_cast<size_t>(rows) * kv + 4) / 2 * 16 + (static_cast<size_t>(rows) * kj + 7) / 4 * 16;
    }
};
inline TileShape tile_shape(int k) {
    TileShape t{k <= 17 ? 32 : kTileRows, k, k, 0, 0};
    if (k % 4 == 0) {
        t.kv = k + 2;
        t.kj = k / 4 % 2 ? k : k + 4;
        t.mv = (65536 + k / 2 - 1) / (k / 2);
        t.mj = (65536 + k / 4 - 1) / (k / 4);
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
    const int warps = blockDim.x >> 5;
    for (int tile = blockIdx.x * warps + wid; tile < tiles; tile += gridDim.x * warps) {
        const int s0 = tile * t.rows, rows = min(t.rows, n - s0);
        const long long q0 = static_cast<long long>(s0) * k, qa = PAD ? q0 : q0 & ~3LL;
        const int m = static_cast<int>(q0 - qa) + rows * k;
        const double* gv = values + qa;
        const int* gj = ja + qa;
        if constexpr (PAD) {
            // the row of piece c, c / (pieces a row), by a product: exact for every
            // tile (at most 1,024 pieces)
            for (int c = lane; c < m / 2; c += 32)
                cp_async_stream<16>(sv + 2 * c + ((c * t.mv) >> 16) * (t.kv - k), gv + 2 * c, pol);
            for (int c = lane; c < m / 4; c += 32)
                cp_async_stream<16>(sj + 4 * c + ((c * t.mj) >> 16) * (t.kj - k), gj + 4 * c, pol);
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
            out[s0 + lane] = row_sum_shared<8>(v, j, k, [u](int c) { return __ldg(u + c); }, 0.0);
        }
        __syncwarp();  // the slab is refilled
    }
}

// Unaligned arrays, short and very long rows: one thread per row (row_sum).
__global__ void spmv_fixed_kernel(int n, int k, const int* __restrict__ ja,
                                  const double* __restrict__ values, const double* __restrict__ u,
                                  double* __restrict__ out, bool vec) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const long long q = static_cast<long long>(s) * k;
        out[s] = row_sum(ja, values, q, q + k, vec, [u](int j) { return __ldg(u + j); });
    }
}

// Rows that go by tiles. Shorter ones: a tile is a few hundred bytes, and its fixed cost
// stays (k = 4, 1M rows: 22 us a tile of 32 rows at a time, 11.2 us a thread a row; k =
// 8 24 and 22; k = 9 25 and 36); the padded rows of 12 entries only beyond L2 (400,000 rows
// 15.4 and 13.1, 800,000 26 and 31). Longer ones: the slabs leave too few warps.
constexpr int kTiledMinK = 9, kTiledMaxK = 128;
constexpr long long kL2Bytes = 126ll * 1000 * 1000;

bool by_tiles(int n, int k) {
    if (k == 12) return static_cast<long long>(n) * k * 12 > kL2Bytes / 4 * 3;
    return k >= kTiledMinK && k <= kTiledMaxK;
}

int launch_spmv(int n, int k, const int* ja, const double* values, const double* u, double* out,
                cudaStream_t st) {
    const bool vec = rows_vectorizable(ja, values);
    if (!vec || !by_tiles(n, k)) {
        const int blocks = std::min((n + 255) / 256, 148 * 16);
        spmv_fixed_kernel<<<blocks, 256, 0, st>>>(n, k, ja, values, u, out, vec);
        return RBFB_OK;
    }
    const TileShape t = tile_shape(k);
    // Blocks of one warp even out the last wave, which counts while the operator
    // comes from L2 (k = 35, 150,000 rows: 15.2 us, four warps 17.9), and for long rows, of
    // which an SM holds few blocks of four (k = 100, 60,000 rows: 22.0 us against 26.4; 600,000:
    // 176 against 210; k = 60, 60,000 rows: 14.1 and 14.2). Beyond L2 four are as good or better
    // for the others (k = 44, 700,000 rows: 80 us against 84).
    const int warps = k >= 60 || static_cast<long long>(n) * k * 12 <= kL2Bytes ? 1 : kSpmvWarps;
    const size_t smem = warps * t.warp_bytes();  // at most 45.5 KB
    auto* kern = k % 4 == 0 ? &spmv_tiled_kernel<true> : &spmv_tiled_kernel<false>;
    const int per_block = warps * t.rows;
    const int blocks = std::min((n + per_block - 1) / per_block, 148 * 256 / warps);
    kern<<<blocks, warps * 32, smem, st>>>(n, k, t, ja, values, u, out);
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
