// lbm.cu -- D2Q9 lattice Boltzmann kernels on sm_100a: equilibrium, moments,
// BGK collision, and semi-Lagrangian streaming through assembled RBF-FD
// interpolation operators, fused with the collision.
//
// Replaces feq_kernel, macros_kernel, bgk_kernel and bgk_kernel_split of
// src/lbm/d2q9_kernels.cu:13-150 (C++ twins of src/lbm/d2q9_kernels.cuf:
// 55-257). Same lattice (direction 0 at rest; 1-4 E, N, W, S; 5-8 NE, NW, SW,
// SE), same planar storage (direction a of node i at pdf[i + n*a]), same
// arithmetic: every product, sum and quotient of the reference's expressions
// in its order, each rounded once (no contraction into fused multiply-adds),
// for float and double. The results are bit-identical to the reference's
// kernels compiled without contraction and to the oracle's CPU restatement.
//
// Streaming is what the reference's assembly exists for (semi-Lagrangian
// streaming with interpolation operators, src/rbf_operators.h:292-298) but
// does not ship: population a of node s after streaming is the interpolation
// of the post-collision field f_a at the departure point x_s - c_a dt,
// sum_j W_a[s*k + j] * f_a[ja[s*k + j]], with W_a the weights of the
// interpolation right-hand side at that point (rbfb_assemble with
// RBFB_OP_INTERP and the 8 departure points). The sum runs in entry order,
// j = 0 first: the first product rounded, then one fused multiply-add an
// entry, as a CSR row product does. A warp stages 32 nodes' rows in shared
// memory and each lane sums its own node's row; the oracle restates that
// order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "rbf_b200.h"
#include "row_sum.cuh"
#include "stream_copy.cuh"

namespace rbfb {
namespace lbm {

// Arithmetic rounded once per operation, per type.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double quo(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double fmaT(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float quo(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float fmaT(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// D2Q9 constants in the working precision, formed as the reference forms
// them (src/lbm/d2q9_kernels.h:16-31): a quotient of two small integers, and
// 3 times a weight, each rounded in T.
template <typename T>
struct Lattice {
    static constexpr T w0 = T(4) / T(9);
    static constexpr T ws = T(1) / T(9);
    static constexpr T wd = T(1) / T(36);
    static constexpr T three_w0 = T(3) * w0;
    static constexpr T three_ws = T(3) * ws;
    static constexpr T three_wd = T(3) * wd;
    static constexpr T one_third = T(1) / T(3);
    static constexpr T one_half = T(1) / T(2);
    static constexpr T three_halves = T(3) / T(2);
};

// Density and velocity of populations f[0..8].
template <typename T>
__device__ __forceinline__ void moments(const T (&f)[9], T& rho, T& ux, T& uy) {
    rho = add(add(add(add(f[5], f[7]), add(f[6], f[8])), add(add(f[1], f[3]), add(f[2], f[4]))),
              f[0]);
    const T invrho = quo(T(1), rho);
    ux = mul(invrho, add(add(sub(f[5], f[7]), sub(f[8], f[6])), sub(f[1], f[3])));
    uy = mul(invrho, add(add(sub(f[5], f[7]), sub(f[6], f[8])), sub(f[2], f[4])));
}

// The direction-independent part of the equilibrium, 1/3 - u.u/2.
template <typename T>
__device__ __forceinline__ T indp_of(T uxsq, T uysq) {
    using L = Lattice<T>;
    return sub(L::one_third, mul(L::one_half, add(uxsq, uysq)));
}

// The equilibrium terms: e[a] = 3 w_a rho (indp + c_a.u + 3/2 (c_a.u)^2)
// without the factor 3 w_a rho, as pairs of opposite directions share them.
template <typename T>
struct EqTerms {
    T t13p, t13m, t24p, t24m, t57p, t57m, t68m, t68p;
};
template <typename T>
__device__ __forceinline__ EqTerms<T> eq_terms(T ux, T uy, T uxsq, T uysq, T indp) {
    using L = Lattice<T>;
    EqTerms<T> e;
    const T v13 = add(indp, mul(L::three_halves, uxsq));
    e.t13p = add(v13, ux);
    e.t13m = sub(v13, ux);
    const T v24 = add(indp, mul(L::three_halves, uysq));
    e.t24p = add(v24, uy);
    e.t24m = sub(v24, uy);
    const T xpy = add(ux, uy);
    const T v57 = add(indp, mul(mul(L::three_halves, xpy), xpy));
    e.t57p = add(v57, xpy);
    e.t57m = sub(v57, xpy);
    const T xmy = sub(ux, uy);
    const T v68 = add(indp, mul(mul(L::three_halves, xmy), xmy));
    e.t68m = sub(v68, xmy);
    e.t68p = add(v68, xmy);
    return e;
}

// BGK relaxation of f towards the equilibrium of its own moments: out[a] =
// (1 - omega) f[a] + omega 3 w_a rho (...), the reference's bgk_kernel body.
template <typename T>
__device__ __forceinline__ void collide(const T (&f)[9], T omega, T (&out)[9], T& rho, T& ux,
                                        T& uy, T& indp) {
    using L = Lattice<T>;
    const T omegabar = sub(T(1), omega);
    const T ow0 = mul(omega, L::three_w0);
    const T ows = mul(omega, L::three_ws);
    const T owd = mul(omega, L::three_wd);
    moments(f, rho, ux, uy);
    const T uxsq = mul(ux, ux);
    const T uysq = mul(uy, uy);
    indp = indp_of(uxsq, uysq);
    const EqTerms<T> e = eq_terms(ux, uy, uxsq, uysq, indp);
    out[0] = add(mul(omegabar, f[0]), mul(mul(ow0, rho), indp));
    out[1] = add(mul(omegabar, f[1]), mul(mul(ows, rho), e.t13p));
    out[3] = add(mul(omegabar, f[3]), mul(mul(ows, rho), e.t13m));
    out[2] = add(mul(omegabar, f[2]), mul(mul(ows, rho), e.t24p));
    out[4] = add(mul(omegabar, f[4]), mul(mul(ows, rho), e.t24m));
    out[5] = add(mul(omegabar, f[5]), mul(mul(owd, rho), e.t57p));
    out[7] = add(mul(omegabar, f[7]), mul(mul(owd, rho), e.t57m));
    out[6] = add(mul(omegabar, f[6]), mul(mul(owd, rho), e.t68m));
    out[8] = add(mul(omegabar, f[8]), mul(mul(owd, rho), e.t68p));
}

template <typename T>
__global__ void feq_kernel(int n, const T* __restrict__ rho, const T* __restrict__ ux,
                           const T* __restrict__ uy, T* __restrict__ pdf) {
    using L = Lattice<T>;
    const size_t N = static_cast<size_t>(n);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const T r = rho[i], u = ux[i], v = uy[i];
        const T uxsq = mul(u, u), uysq = mul(v, v);
        const T indp = indp_of(uxsq, uysq);
        const EqTerms<T> e = eq_terms(u, v, uxsq, uysq, indp);
        pdf[i] = mul(mul(L::three_w0, r), indp);
        pdf[i + N * 1] = mul(mul(L::three_ws, r), e.t13p);
        pdf[i + N * 3] = mul(mul(L::three_ws, r), e.t13m);
        pdf[i + N * 2] = mul(mul(L::three_ws, r), e.t24p);
        pdf[i + N * 4] = mul(mul(L::three_ws, r), e.t24m);
        pdf[i + N * 5] = mul(mul(L::three_wd, r), e.t57p);
        pdf[i + N * 7] = mul(mul(L::three_wd, r), e.t57m);
        pdf[i + N * 6] = mul(mul(L::three_wd, r), e.t68m);
        pdf[i + N * 8] = mul(mul(L::three_wd, r), e.t68p);
    }
}

template <typename T>
__global__ void macros_kernel(int n, const T* __restrict__ pdf, T* __restrict__ rho,
                              T* __restrict__ ux, T* __restrict__ uy) {
    const size_t N = static_cast<size_t>(n);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        T f[9];
#pragma unroll
        for (int a = 0; a < 9; ++a) f[a] = pdf[i + N * a];
        T r, u, v;
        moments(f, r, u, v);
        rho[i] = r;
        ux[i] = u;
        uy[i] = v;
    }
}

// bgk_kernel (indp == nullptr) and bgk_kernel_split: collision in place.
template <typename T>
__global__ void bgk_kernel(int n, T omega, T* __restrict__ pdf, T* __restrict__ rho,
                           T* __restrict__ ux, T* __restrict__ uy, T* __restrict__ indp) {
    const size_t N = static_cast<size_t>(n);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        T f[9], o[9], r, u, v, d;
#pragma unroll
        for (int a = 0; a < 9; ++a) f[a] = pdf[i + N * a];
        collide(f, omega, o, r, u, v, d);
        rho[i] = r;
        ux[i] = u;
        uy[i] = v;
        if (indp) indp[i] = d;
#pragma unroll
        for (int a = 0; a < 9; ++a) pdf[i + N * a] = o[a];
    }
}

constexpr int kMaxStencil = 64;  // largest stencil of a streaming step
constexpr int kTileWarps = 4;  // warps a CTA; each warp owns a 32-node tile at a time

// How a tile's rows are copied into its slabs: in 16-byte pieces of one run, in
// 16-byte pieces row by row (k a multiple of 4: rows one after another would put
// all lanes on a few banks), or entry by entry (arrays that are not 16-byte
// aligned; an even k is padded to the next odd).
enum Copy { kRun16, kRows16, kRun8, kPad8 };

// Entries from a row to the next in shared memory.
template <int COPY>
__host__ __device__ constexpr int weight_stride(int k) {
    return COPY == kRows16 ? k + 2 : COPY == kPad8 ? k + 1 : k;
}
template <int COPY>
__host__ __device__ inline int index_stride(int k) {
    return COPY == kRows16 ? (k / 4 % 2 ? k : k + 4) : COPY == kPad8 ? k + 1 : k;
}

// A lane's walk over the pieces of rows that are copied row by row: its first
// piece's row and place in the row, and the step of 32 pieces (formed once a warp: the
// divisions cost more than a short row's copy).
struct Pieces {
    int row, r, c, dr, dc;
};
template <int COPY, typename V>
__device__ __forceinline__ Pieces pieces(int k, int lane) {
    const int row = COPY == kRows16 ? k / (16 / static_cast<int>(sizeof(V))) : k;
    const int r = lane / row, dr = 32 / row;
    return {row, r, lane - r * row, dr, 32 - dr * row};
}

// Copies the tile's m entries into a slab, rows ks entries apart.
template <int COPY, typename V>
__device__ __forceinline__ void copy_slab(V* dst, const V* src, int m, const Pieces& p, int ks, int lane,
                                          unsigned long long pol) {
    constexpr int per = 16 / sizeof(V);
    if constexpr (COPY == kRun16) {
        const int chunks = m / per;
        for (int q = lane; q < chunks; q += 32)
            cp_async_stream<16>(dst + q * per, src + q * per, pol);
        for (int e = chunks * per + lane; e < m; e += 32)
            cp_async_stream<sizeof(V)>(dst + e, src + e, pol);
    } else if constexpr (COPY == kRun8) {
        for (int q = lane; q < m; q += 32) cp_async_stream<sizeof(V)>(dst + q, src + q, pol);
    } else {
        constexpr int step = COPY == kRows16 ? per : 1;
        int r = p.r, c = p.c;
        for (int q = lane; q < m / step; q += 32) {
            cp_async_stream<step * sizeof(V)>(dst + r * ks + c * step, src + q * step, pol);
            r += p.dr;
            c += p.dc;
            if (c >= p.row) {
                c -= p.row;
                ++r;
            }
        }
    }
}

// Semi-Lagrangian streaming of the post-collision field pdf_in through the
// interpolation operators W (8 arrays of n*k weights, direction a at
// W + (a-1)*n*k, rows like ja), then the BGK collision, into pdf_out. The
// moments of the streamed populations go to rho, ux, uy (any may be null).
// A warp takes a tile of 32 consecutive nodes: it copies the tile's index rows
// and the first direction's weight rows into shared memory; for each direction
// it starts the copy of the next one and has each lane sum its own node's row in
// entry order (the first product rounded, then one fused multiply-add an entry),
// gathering pdf_in through the indices. Then every lane collides its node and the
// warp writes 32 consecutive entries of each direction, as streaming stores.
//
// Bound by memory where enough warps are resident to cover the gathers, so:
// KT > 0 fixes k at compile time: the index rows land in the second weight slab
// and each lane keeps its own in registers for the tile, which saves the index
// slab and its reads, and the gathers of a row are in flight at once.
// 1M nodes (100k), FP64, us, in the general kernel and in that of the size: k = 15 264
// and 188 (42, 22), k = 18 361 and 218 (47, 27), k = 24 589 and 312 (64, 38); k = 21 259 us, 6.46
// TB/s, with the two fields in turn. A size has its kernel where 16-byte copies can be: n k even.
// Resident CTAs that the registers are cut for: those that the slabs allow, at
// most 6 for short rows and 4 (128 registers) from 16 entries on, where more
// gathers in flight are worth more than more warps. 1M nodes, k = 15 187 (6) and
// 195 us (4), k = 16 223 and 209, k = 21 254 and 248; left to itself the compiler
// takes 56 registers for k = 21 in FP32, 330 us against 229.
// KT = kShort: any k of a few entries. The batch of eight gathers, most of it
// predicated off, and its 100 registers cost such rows up to 1.75 times the time of a plain
// loop: FP64, 600,000 nodes, k = 1 33 against 57 us, k = 9 (odd n) 86 and 109. As many CTAs
// as 64 registers (FP32: 40) allow.
constexpr int kShort = -1;
constexpr int resident(int kt, int stride, bool fp32) {
    const int fit = 227 * 1024 / (kTileWarps * 32 * 2 * stride * 8 + 1024);
    const int most = kt > 0 && kt < 16 ? 6 : 4;
    return kt == kShort ? (fp32 ? 12 : 8) : kt == 0 ? most : fit < most ? fit : most;
}
template <typename T, int COPY, int KT>
__global__ void __launch_bounds__(kTileWarps * 32, resident(KT, weight_stride<COPY>(KT), sizeof(T) == 4))
    stream_collide_kernel(
    int n, int k, const int* __restrict__ ja, const double* __restrict__ W, T omega,
    const T* __restrict__ pdf_in, T* __restrict__ pdf_out, T* __restrict__ rho,
    T* __restrict__ ux, T* __restrict__ uy) {
    extern __shared__ __align__(16) unsigned char tile_smem[];
    if (KT > 0) k = KT;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int kv = weight_stride<COPY>(k), kj = index_stride<COPY>(k);
    const int slab = 32 * kv;
    double* wbuf = reinterpret_cast<double*>(tile_smem) + static_cast<size_t>(wid) * 2 * slab;
    int* jbuf = KT > 0 ? reinterpret_cast<int*>(wbuf + slab)
                       : reinterpret_cast<int*>(reinterpret_cast<double*>(tile_smem) +
                                                static_cast<size_t>(kTileWarps) * 2 * slab) +
                             static_cast<size_t>(wid) * 32 * kj;
    const size_t N = static_cast<size_t>(n);
    const size_t nnz = N * static_cast<size_t>(k);
    const unsigned long long pol = evict_first_policy();
    const Pieces pw = pieces<COPY, double>(k, lane), pj = pieces<COPY, int>(k, lane);
    const int tiles = (n + 31) >> 5;
    for (int tile = blockIdx.x * kTileWarps + wid; tile < tiles; tile += gridDim.x * kTileWarps) {
        const int s0 = tile << 5;
        const int cnt = min(32, n - s0);
        const int m = cnt * k;
        const size_t base = static_cast<size_t>(s0) * k;
        copy_slab<COPY>(jbuf, ja + base, m, pj, kj, lane, pol);
        copy_slab<COPY>(wbuf, W + base, m, pw, kv, lane, pol);
        cp_async_commit();
        int jrow[KT > 0 ? KT : 1];
        if constexpr (KT > 0) {  // the lane's index row, then the slab is free
            cp_async_wait<0>();
            __syncwarp();
            if (lane < cnt)
#pragma unroll
                for (int j = 0; j < KT; ++j) jrow[j] = jbuf[lane * kj + j];
            __syncwarp();
        }
        T f[9];
#pragma unroll
        for (int a = 1; a < 9; ++a) {
            if (a < 8) {
                copy_slab<COPY>(wbuf + (a & 1) * slab, W + static_cast<size_t>(a) * nnz + base, m, pw, kv,
                                lane, pol);
                cp_async_commit();
            }
            cp_async_wait_pending(a < 8 ? 1 : 0);
            __syncwarp();
            if (lane < cnt) {
                const double* wr = wbuf + ((a - 1) & 1) * slab + lane * kv;
                const T* pa = pdf_in + N * a;
                if constexpr (KT > 0) {
                    T v = mul(static_cast<T>(wr[0]), pa[jrow[0]]);
#pragma unroll
                    for (int j = 1; j < KT; ++j) v = fmaT(static_cast<T>(wr[j]), pa[jrow[j]], v);
                    f[a] = v;
                } else if constexpr (KT == kShort) {
                    const int* jr = jbuf + lane * kj;
                    T v = mul(static_cast<T>(wr[0]), pa[jr[0]]);
#pragma unroll 8
                    for (int j = 1; j < k; ++j) v = fmaT(static_cast<T>(wr[j]), pa[jr[j]], v);
                    f[a] = v;
                } else {
                    // a sum from -0 gives the first product itself
                    f[a] = row_sum_shared<8>(wr, jbuf + lane * kj, k, [pa](int c) { return pa[c]; }, T(-0.0));
                }
            }
            __syncwarp();  // every lane is done with this slab before it is refilled
        }
        const int s = s0 + lane;
        if (lane < cnt) {
            f[0] = pdf_in[s];  // the rest population does not move
            T o[9], r, u, v, d;
            collide(f, omega, o, r, u, v, d);
#pragma unroll
            for (int a = 0; a < 9; ++a) __stcs(pdf_out + s + N * a, o[a]);
            if (rho) __stcs(rho + s, r);
            if (ux) __stcs(ux + s, u);
            if (uy) __stcs(uy + s, v);
        }
    }
}

template <typename T, int COPY, int KT>
int launch_stream_collide(int n, int k, const int* ja, const double* W, T omega, const T* pin,
                          T* pout, T* rho, T* ux, T* uy, cudaStream_t st) {
    auto kern = stream_collide_kernel<T, COPY, KT>;
    auto bytes = [](int rows_of) {
        return static_cast<size_t>(kTileWarps) * 32 *
               (2 * weight_stride<COPY>(rows_of) * sizeof(double) +
                (KT > 0 ? 0 : index_stride<COPY>(rows_of) * sizeof(int)));
    };
    const size_t smem = bytes(k);
    // the limit is the process's, not this call's: always the largest that a call can
    // ask for, or another thread's launch would be refused
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(bytes(KT > 0 ? k : kMaxStencil))) != cudaSuccess)
        return RBFB_ECUDA;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kTileWarps * 32, smem) !=
            cudaSuccess ||
        per_sm < 1)
        return RBFB_ECUDA;
    const int tiles = (n + 31) / 32;
    const int blocks = std::max(1, std::min((tiles + kTileWarps - 1) / kTileWarps,
                                            std::max(sms, 1) * per_sm));
    kern<<<blocks, kTileWarps * 32, smem, st>>>(n, k, ja, W, omega, pin, pout, rho, ux, uy);
    return cudaGetLastError() == cudaSuccess ? RBFB_OK : RBFB_ECUDA;
}

// A kernel for each stencil size up to kMaxFixed, from kMinFixed (degree 1) on, for
// aligned arrays and an even n k (every direction's weights then start on a 16-byte boundary).
constexpr int kMinFixed = 5, kMaxFixed = 32;
template <typename T, int KT, class... A>
int launch_fixed(int n, int k, A... args) {
    if constexpr (KT > kMaxFixed) {
        return launch_stream_collide<T, kRun16, 0>(n, k, args...);
    } else {
        if (k != KT) return launch_fixed<T, KT + 1>(n, k, args...);
        return launch_stream_collide<T, KT % 4 ? kRun16 : kRows16, KT>(n, k, args...);
    }
}

template <typename T>
int stream_collide(int n, int k, const int* ja, const double* W, T omega, const T* pin, T* pout,
                   T* rho, T* ux, T* uy, cudaStream_t st) {
    // 16-byte copies need 16-byte aligned rows: ja, W and every direction's
    // array (n*k even)
    const bool vec = ((reinterpret_cast<uintptr_t>(ja) | reinterpret_cast<uintptr_t>(W)) & 15) == 0 &&
                     ((static_cast<long long>(n) * k) & 1) == 0;
    if (vec && k >= kMinFixed && k <= kMaxFixed)
        return launch_fixed<T, kMinFixed>(n, k, ja, W, omega, pin, pout, rho, ux, uy, st);
    // rows that are short and have no kernel of their size (fewer than kMinFixed entries, or
    // an odd n k): FP32 9 entries are better off with the batches (33 us against 36)
    if (k <= (sizeof(T) == 4 ? 8 : 10)) {
        if (k % 2 == 0 && (k > 2 || sizeof(T) == 8))
            return launch_stream_collide<T, kPad8, kShort>(n, k, ja, W, omega, pin, pout, rho, ux, uy, st);
        if (vec)
            return launch_stream_collide<T, kRun16, kShort>(n, k, ja, W, omega, pin, pout, rho, ux, uy, st);
        return launch_stream_collide<T, kRun8, kShort>(n, k, ja, W, omega, pin, pout, rho, ux, uy, st);
    }
    if (vec && k % 4 == 0)
        return launch_stream_collide<T, kRows16, 0>(n, k, ja, W, omega, pin, pout, rho, ux, uy, st);
    if (vec) return launch_stream_collide<T, kRun16, 0>(n, k, ja, W, omega, pin, pout, rho, ux, uy, st);
    if (k & 1)
        return launch_stream_collide<T, kRun8, 0>(n, k, ja, W, omega, pin, pout, rho, ux, uy, st);
    return launch_stream_collide<T, kPad8, 0>(n, k, ja, W, omega, pin, pout, rho, ux, uy, st);
}

int blocks_for(int n) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(1, std::min((n + 255) / 256, std::max(sms, 1) * 16));
}

}  // namespace lbm
}  // namespace rbfb

using namespace rbfb::lbm;

extern "C" {

int rbfb_lbm_feq(int n, int precision, const void* rho, const void* ux, const void* uy, void* pdf,
                 void* stream) {
    if (n < 0 || !rho || !ux || !uy || !pdf) return RBFB_EINVAL;
    if (n == 0) return RBFB_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (precision == RBFB_FP64)
        feq_kernel<double><<<blocks_for(n), 256, 0, st>>>(
            n, static_cast<const double*>(rho), static_cast<const double*>(ux),
            static_cast<const double*>(uy), static_cast<double*>(pdf));
    else if (precision == RBFB_LBM_FP32)
        feq_kernel<float><<<blocks_for(n), 256, 0, st>>>(
            n, static_cast<const float*>(rho), static_cast<const float*>(ux),
            static_cast<const float*>(uy), static_cast<float*>(pdf));
    else
        return RBFB_EINVAL;
    return cudaGetLastError() == cudaSuccess ? RBFB_OK : RBFB_ECUDA;
}

int rbfb_lbm_macros(int n, int precision, const void* pdf, void* rho, void* ux, void* uy,
                    void* stream) {
    if (n < 0 || !rho || !ux || !uy || !pdf) return RBFB_EINVAL;
    if (n == 0) return RBFB_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (precision == RBFB_FP64)
        macros_kernel<double><<<blocks_for(n), 256, 0, st>>>(
            n, static_cast<const double*>(pdf), static_cast<double*>(rho),
            static_cast<double*>(ux), static_cast<double*>(uy));
    else if (precision == RBFB_LBM_FP32)
        macros_kernel<float><<<blocks_for(n), 256, 0, st>>>(
            n, static_cast<const float*>(pdf), static_cast<float*>(rho), static_cast<float*>(ux),
            static_cast<float*>(uy));
    else
        return RBFB_EINVAL;
    return cudaGetLastError() == cudaSuccess ? RBFB_OK : RBFB_ECUDA;
}

int rbfb_lbm_bgk(int n, int precision, double omega, void* pdf, void* rho, void* ux, void* uy,
                 void* indp, void* stream) {
    if (n < 0 || !rho || !ux || !uy || !pdf) return RBFB_EINVAL;
    if (n == 0) return RBFB_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (precision == RBFB_FP64)
        bgk_kernel<double><<<blocks_for(n), 256, 0, st>>>(
            n, omega, static_cast<double*>(pdf), static_cast<double*>(rho),
            static_cast<double*>(ux), static_cast<double*>(uy), static_cast<double*>(indp));
    else if (precision == RBFB_LBM_FP32)
        bgk_kernel<float><<<blocks_for(n), 256, 0, st>>>(
            n, static_cast<float>(omega), static_cast<float*>(pdf), static_cast<float*>(rho),
            static_cast<float*>(ux), static_cast<float*>(uy), static_cast<float*>(indp));
    else
        return RBFB_EINVAL;
    return cudaGetLastError() == cudaSuccess ? RBFB_OK : RBFB_ECUDA;
}

int rbfb_lbm_stream_collide(int n, int precision, int k, const int* ja, const double* W,
                            double omega, const void* pdf_in, void* pdf_out, void* rho, void* ux,
                            void* uy, void* stream) {
    if (n < 0 || k < 1 || k > kMaxStencil || !ja || !W || !pdf_in || !pdf_out || pdf_in == pdf_out)
        return RBFB_EINVAL;
    if (n == 0) return RBFB_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (precision == RBFB_FP64)
        return stream_collide<double>(n, k, ja, W, omega, static_cast<const double*>(pdf_in),
                                      static_cast<double*>(pdf_out), static_cast<double*>(rho),
                                      static_cast<double*>(ux), static_cast<double*>(uy), st);
    if (precision == RBFB_LBM_FP32)
        return stream_collide<float>(n, k, ja, W, static_cast<float>(omega),
                                     static_cast<const float*>(pdf_in),
                                     static_cast<float*>(pdf_out), static_cast<float*>(rho),
                                     static_cast<float*>(ux), static_cast<float*>(uy), st);
    return RBFB_EINVAL;
}

}  // extern "C"
