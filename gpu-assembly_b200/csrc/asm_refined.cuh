// asm_refined.cuh -- batched RBF-FD assembly on sm_100a, the refined form: the
// saddle-point system factored in FP32 in shared memory, the solution refined
// with FP64 residuals until the predicted error is below the tolerance, and the
// stencils whose refinement stalls listed for the FP64 kernel.
//
// Replaces assemble_interp_weights<Config> (src/rbf_operators.h:292-376) for the
// precision pattern of FP32 factors and an FP64 result.
//
// One warp owns a stencil of n = npoly(P) + k_s unknowns, any n <= NMAX. Its
// working set:
//   S  the system in FP32, row-major with the right-hand sides as columns n ..
//      n+NRHS-1, factored in place (rows are never swapped: piv[c] is the row
//      that became the pivot row at step c; 1 / pivot in the pivot's place);
//   M  the system in FP64 for the residual: it is symmetric, so the 8 x 8
//      tiles on and below the diagonal alone (10.5 KB at n = 45, 18 KB whole);
//   b  the FP64 right-hand sides.
//
// Elimination: panels of 8 columns as in asm_dmma.cuh, in FP32 with packed
// fused multiply-adds (fma.rn.f32x2) for the trailing columns.
//
// Solution: lane (g, q) = (lane / 4, lane % 4) holds right-hand side q of the
// unknowns 8 t + g in registers, the FP32 correction y[t] as well as the FP64
// solution x[t]. A block of 8 steps of either substitution is 8 shuffles, whose
// results every lane keeps and applies to its rows of the other blocks from two
// 16-byte loads of multipliers: 0.3k instructions a triangle at n = 45, against
// 0.8k step by step with a lane a row.
//
// Residual b - M x on the FP64 tensor cores (mma.sync m8n8k4, FP64 sums in
// ascending column order): the tiles are stored with their column halves
// swapped in rows 2, 3, 6, 7, which makes a tile's fragment and its transpose's
// both free of bank conflicts. 0.25k instructions at n = 45, against 1.6k a
// row to a lane.
//
// Bound by latency: shared memory holds ten stencils an SM (23 KB each at n =
// 45), 2.5 warps a scheduler, which issue 40 % of the cycles; 11.3k warp
// instructions and 2.8 sweeps a stencil. Of a stencil's 63k cycles the gather
// takes 0.7, the fill 11, the elimination 19 and the solution 32 (2.7 a forward,
// 3.1 a backward substitution, 3.2 a residual). 262,144 stencils of k = 35,
// degree 3: 12.27 ms before (a row to a lane throughout, the residual and the
// sweep's bookkeeping on scalars: 21.9k instructions), 6.40 ms now.
#pragma once

#include <cstdint>

#include "asm_dmma.cuh"

namespace rbfb {
namespace ir {

using dm::Item;

template <int NMAX_, int NRHS, int KMAX_>
struct Layout {
    static constexpr int NMAX = NMAX_, KMAX = KMAX_;
    static constexpr int NT = (NMAX + 7) / 8;  // blocks of 8 unknowns
    static_assert(NMAX <= 96, "pivot keys carry the list position in 7 bits");
    static_assert(NRHS <= 4, "four lanes hold an unknown's right-hand sides");
    // Row stride in 16-byte vectors: odd, so the 32 rows a warp reads down
    // one column fall in different bank groups.
    static constexpr int LV0 = (NMAX + NRHS + 3) / 4;
    static constexpr int LDS = 4 * ((LV0 % 2) ? LV0 : LV0 + 1);
    static_assert(8 * NT <= LDS, "a row holds every panel's columns");
    static constexpr int al16(int b) { return (b + 15) & ~15; }
    // neighbour coordinates; from the end of the fill on the lists of unused
    // rows and the next stencil's ja row (as asm_dmma.cuh)
    static constexpr int off_xy = 0;
    static constexpr int off_list = 0;
    static constexpr int off_nja = 2 * al16(NMAX);
    static constexpr int xy_bytes =
        al16(16 * KMAX > off_nja + 4 * KMAX ? 16 * KMAX : off_nja + 4 * KMAX);
    static constexpr int off_s = xy_bytes;
    static constexpr int off_m = off_s + NMAX * LDS * 4;
    static constexpr int off_b = off_m + NT * (NT + 1) / 2 * 512;
    static constexpr int off_piv = off_b + 8 * NT * 32;
    static constexpr int bytes = off_piv + al16(8 * NT);
};

__device__ __forceinline__ float4 lds4(const float* s) { return *reinterpret_cast<const float4*>(s); }
__device__ __forceinline__ void unpack(float4 v, float* d) {
    d[0] = v.x;
    d[1] = v.y;
    d[2] = v.z;
    d[3] = v.w;
}

// c0, c1 -= m * (b0, b1): one packed FP32 fused multiply-add of sm_100a
// (fma.rn.f32x2; each component rounded once, as fmaf).
__device__ __forceinline__ void fnma2(float m, float b0, float b1, float& c0, float& c1) {
    unsigned long long mm, bb, cc, d;
    const float nm = -m;
    asm("mov.b64 %0, {%1, %1};" : "=l"(mm) : "f"(nm));
    asm("mov.b64 %0, {%1, %2};" : "=l"(bb) : "f"(b0), "f"(b1));
    asm("mov.b64 %0, {%1, %2};" : "=l"(cc) : "f"(c0), "f"(c1));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(mm), "l"(bb), "l"(cc));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(c0), "=f"(c1) : "l"(d));
}

// Pivots of the FP32 factors: magnitudes in [2^-120, 2^120). A stencil with
// another one is left to the FP64 kernel.
constexpr uint32_t kLow32 = 7u << 23, kHigh32 = 247u << 23;

// 1 / a to an ulp, for |a| in that range: an approximation and one Newton step.
__device__ __forceinline__ float rcp_fast(float a) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
    return fmaf(y, fmaf(-a, y, 1.0f), y);
}

// Element (a, b) of an 8 x 8 tile of M.
__device__ __forceinline__ int cell(int a, int b) { return 8 * a + (b ^ ((a & 2) << 1)); }

// M(r, c) = M(c, r) = v, r >= c.
__device__ __forceinline__ void put(double* M, int r, int c, double v) {
    const int I = r >> 3, J = c >> 3;
    double* T = M + (I * (I + 1) / 2 + J) * 64;
    T[cell(r & 7, c & 7)] = v;
    if (I == J) T[cell(c & 7, r & 7)] = v;
}

template <int LDS, int NP, int Q>
__device__ __forceinline__ void fill_pair(float* Sn, double* M, int i, int j, double2 a, double2 b,
                                          uint32_t& wmin, uint32_t& wmax) {
    const double r2 = dist2(dsub(b.x, a.x), dsub(b.y, a.y));
    const double v = dm::phs_fast<Q>(r2);
    wmin = min(wmin, (uint32_t)__double2hiint(r2));
    wmax = max(wmax, (uint32_t)__double2hiint(r2));
    const float f = (float)v;
    Sn[i * LDS + j] = f;
    Sn[j * LDS + i] = f;
    put(M, NP + max(i, j), NP + min(i, j), v);
}

// The system in S, M and b (fill_matrix / fill_rhs, src/rbf_operators.h:
// 116-185), the pairs walked as in asm_dmma.cuh; zeros past n up to whole
// blocks, which the substitutions and the residual read. Returns whether a
// value left the range of the branch-free forms.
template <class L, int NRHS, int P, int Q>
__device__ __forceinline__ bool fill_system(const AsmParams& p, float* S, double* M, double* b,
                                            const double2* xy, int ks, int e, int lane) {
    constexpr int NP = npoly(P), LDS = L::LDS;
    const int n = NP + ks, nt = (n + 7) >> 3;
    uint32_t wmin = dm::kLow, wmax = 0;
    float* Sn = S + NP * LDS + NP;
    const int half = (ks - 1) >> 1;
    const int ib = ks & ~31;
    for (int i0 = 0; i0 < ib; i0 += 32) {
        const int i = i0 + lane;
        const double2 a = xy[i];
        int j = i + 1;
        j = j >= ks ? j - ks : j;
        const int dend = half + ((ks & 1) == 0 && i < ks / 2 ? 1 : 0);
        for (int d = 1; d <= dend; ++d) {
            fill_pair<LDS, NP, Q>(Sn, M, i, j, a, xy[j], wmin, wmax);
            ++j;
            j = j >= ks ? j - ks : j;
        }
    }
    {
        const int rows = ks - ib, count = ib ? rows * half : ks * (ks - 1) / 2;
        int i = ib + lane, d = 1;
        if (rows > 0) {
            while (i >= ks) {
                i -= rows;
                ++d;
            }
            for (int t = lane; t < count; t += 32) {
                int j = i + d;
                j = j >= ks ? j - ks : j;
                fill_pair<LDS, NP, Q>(Sn, M, i, j, xy[i], xy[j], wmin, wmax);
                i += 32;
                while (i >= ks) {
                    i -= rows;
                    ++d;
                }
            }
        }
    }
    for (int i = lane; i < ks; i += 32) {
        const int r = NP + i;
        const double2 c = xy[i];
        double mon[NP];
        monomials<P>(c.x, c.y, mon);
#pragma unroll
        for (int m = 0; m < NP; ++m) {
            S[r * LDS + m] = (float)mon[m];
            S[m * LDS + r] = (float)mon[m];
            put(M, r, m, mon[m]);
        }
        S[r * LDS + r] = 0.f;
        put(M, r, r, 0.0);
        double rv[NRHS];
        if (p.plain_ops) {
            dm::rhs_plain<Q, NRHS>(p, c.x, c.y, rv, wmin, wmax);
        } else {
            rhs_node<P, Q, NRHS>(p, c.x, c.y, e, rv);
#pragma unroll
            for (int q = 0; q < NRHS; ++q) wmax = max(wmax, dm::mag_word(rv[q]));
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            b[4 * r + q] = q < NRHS ? rv[q < NRHS ? q : 0] : 0.0;
            if (q < NRHS) S[r * LDS + n + q] = (float)rv[q < NRHS ? q : 0];
        }
    }
    for (int f = lane; f < NP * NP; f += 32) {
        const int r = f / NP, c = f % NP;
        S[r * LDS + c] = 0.f;
        if (r >= c) put(M, r, c, 0.0);
    }
    for (int f = lane; f < 4 * NP; f += 32) {
        const int r = f >> 2, q = f & 3;
        const double v = q < NRHS && q < p.nrhs ? rhs_poly<P>(p, q, r, e) : 0.0;
        b[f] = v;
        if (q < NRHS) S[r * LDS + n + q] = (float)v;
    }
    if (n & 7) {  // up to whole blocks
        double* T = M + (nt - 1) * nt / 2 * 64;
        const int first = n & 7;  // of the last block's rows
        for (int f = lane; f < 64 * nt; f += 32) {
            const int a = (f >> 3) & 7, c = f & 7;
            if (a >= first || (f >= 64 * (nt - 1) && c >= first)) T[(f & ~63) + cell(a, c)] = 0.0;
        }
        for (int f = 4 * n + lane; f < 32 * nt; f += 32) b[f] = 0.0;
        for (int c = n + NRHS; c < 8 * nt; ++c)
            for (int r = lane; r < n; r += 32) S[r * LDS + c] = 0.f;
    }
    return wmin < dm::kLow || wmax >= dm::kHigh;
}

// The steps of one panel: columns c0 .. c0+7, the first tend of them, on the m
// rows of list, R list positions a lane (asm_dmma.cuh panel, in FP32: the key is
// the value's own magnitude word, and a row's panel columns are two vectors).
// Returns whether a pivot left the range of kLow32, kHigh32.
template <int R, int LDS>
__device__ __forceinline__ bool panel(float* S, const uint8_t* list, uint8_t* next, uint8_t* piv, int m,
                                      int held, int c0, int tend, int lane) {
    constexpr unsigned ALL = 0xffffffffu;
    float* Sc = S + c0;
    float a[R][8];
    int off[R], keep[R];  // keep: leading vectors still to be written back
    uint32_t kmask[R], kcon[R];
#pragma unroll
    for (int sl = 0; sl < R; ++sl) {
        const int pos = lane + 32 * sl;
        const bool v = pos < m;
        off[sl] = list[v ? pos : 0] * LDS;
        kmask[sl] = v ? 0x7fffff80u : 0u;
        kcon[sl] = v ? 127u - (uint32_t)pos : 0u;
        keep[sl] = v ? 2 : 0;
        unpack(lds4(Sc + off[sl]), a[sl]);
        unpack(lds4(Sc + off[sl] + 4), a[sl] + 4);
    }
    // steps past tend run on a dummy that loses to every pivot in range
    if (R == 1 && lane == 31 && tend < 8) kcon[0] = kLow32 | 96u;
    uint32_t key;
    int bsl;
    float bv;
    auto keys = [&](int t) {
        key = (__float_as_uint(a[0][t]) & kmask[0]) | kcon[0];
        bsl = 0;
        bv = a[0][t];
#pragma unroll
        for (int sl = 1; sl < R; ++sl) {
            const uint32_t kk = (__float_as_uint(a[sl][t]) & kmask[sl]) | kcon[sl];
            const bool better = kk > key;
            bv = better ? a[sl][t] : bv;
            bsl = better ? sl : bsl;
            key = better ? kk : key;
        }
    };
    keys(0);
    uint32_t best = __reduce_max_sync(ALL, key), low = kHigh32, high = 0;
    auto step = [&](int t) {
        low = min(low, best);
        high = max(high, best);
        const float rv = rcp_fast(bv);  // 1 / pivot, if this lane owns the pivot
        const int owner = (int)(~best & 31u);
        int po = off[0];
        float bn = a[0][t + 1 < 8 ? t + 1 : t];
#pragma unroll
        for (int sl = 1; sl < R; ++sl) {
            po = bsl == sl ? off[sl] : po;
            if (t + 1 < 8) bn = bsl == sl ? a[sl][t + 1] : bn;
        }
        const float inv = __shfl_sync(ALL, rv, owner);
        const float un = t + 1 < 8 ? __shfl_sync(ALL, bn, owner) : 0.f;
        const float* U = Sc + __shfl_sync(ALL, po, owner);
        const bool own = lane == owner && (R > 1 || kmask[0]);
#pragma unroll
        for (int sl = 0; sl < R; ++sl) {
            const bool used = own && (R == 1 || bsl == sl);
            if (used) {
#pragma unroll
                for (int j = t & ~3; j < 8; j += 4)  // 1 / pivot in the pivot's place
                    *reinterpret_cast<float4*>(Sc + off[sl] + j) =
                        make_float4(j == t ? rv : a[sl][j], j + 1 == t ? rv : a[sl][j + 1],
                                    j + 2 == t ? rv : a[sl][j + 2], j + 3 == t ? rv : a[sl][j + 3]);
                piv[c0 + t] = (uint8_t)(off[sl] / LDS);
            }
            kmask[sl] = used ? 0u : kmask[sl];
            kcon[sl] = used ? 0u : kcon[sl];
            keep[sl] = used ? t >> 2 : keep[sl];
        }
#pragma unroll
        for (int sl = 0; sl < R; ++sl) {
            a[sl][t] = a[sl][t] * inv;
            if (t + 1 < 8) a[sl][t + 1] = fmaf(-a[sl][t], un, a[sl][t + 1]);
        }
        if (t + 1 < 8) {
            keys(t + 1);
            best = __reduce_max_sync(ALL, key);
        }
        __syncwarp();
        if (t + 2 < 8) {
            float u[8];
            if (t + 2 < 4) unpack(lds4(U), u);
            unpack(lds4(U + 4), u + 4);
#pragma unroll
            for (int sl = 0; sl < R; ++sl) {
                if (t & 1) a[sl][t + 2] = fmaf(-a[sl][t], u[t + 2], a[sl][t + 2]);
#pragma unroll
                for (int j = t + 2 + (t & 1); j < 8; j += 2)
                    fnma2(a[sl][t], u[j], u[j + 1], a[sl][j], a[sl][j + 1]);
            }
        }
    };
    step(0);
    step(1);
    step(2);
    step(3);
    if (R > 1 || tend > 4) {
        step(4);
        step(5);
        step(6);
        step(7);
    }
    if (lane < held) next[lane] = (uint8_t)lane;
    int left = held;
#pragma unroll
    for (int sl = 0; sl < R; ++sl) {
        float* dst = Sc + off[sl];
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (j < keep[sl])
                *reinterpret_cast<float4*>(dst + 4 * j) =
                    make_float4(a[sl][4 * j], a[sl][4 * j + 1], a[sl][4 * j + 2], a[sl][4 * j + 3]);
        const unsigned alive = __ballot_sync(ALL, kmask[sl] != 0u);
        if (kmask[sl]) next[left + __popc(alive & ((1u << lane) - 1u))] = (uint8_t)(off[sl] / LDS);
        left += __popc(alive);
    }
    return low < kLow32 || high >= kHigh32 || left != held + m - tend;
}

// The panel's pivot rows over the columns right of it: row t takes the updates
// of the steps before its own, in order, two columns a lane.
template <int LDS>
__device__ __forceinline__ void pivot_rows(float* S, const float* const (&row)[8], int c0, int tend,
                                           int W, int lane) {
    for (int col = 8 + 2 * lane; c0 + col < W; col += 64) {
        float u[8][2], l[8][8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const float2 w = *reinterpret_cast<const float2*>(row[t] + col);
            u[t][0] = w.x;
            u[t][1] = w.y;
        }
#pragma unroll
        for (int t = 1; t < 8; ++t) {
            unpack(lds4(row[t]), l[t]);
            if (t > 4) unpack(lds4(row[t] + 4), l[t] + 4);
        }
#pragma unroll
        for (int tp = 0; tp < 7; ++tp)
#pragma unroll
            for (int t = tp + 1; t < 8; ++t) fnma2(l[t][tp], u[tp][0], u[tp][1], u[t][0], u[t][1]);
#pragma unroll
        for (int t = 1; t < 8; ++t)
            if (t < tend)
                *reinterpret_cast<float2*>(const_cast<float*>(row[t]) + col) = make_float2(u[t][0], u[t][1]);
    }
}

// The unused rows over the columns right of the panel: a lane holds its row's
// 8 multipliers and walks the columns in vectors of four, the pivot rows' values
// broadcast. With few rows left, groups of 16 or 8 lanes share the columns.
template <int LDS>
__device__ __forceinline__ void update_rows(float* S, const float* const (&row)[8], const uint8_t* list,
                                            int m, int c0, int W, int lane) {
    const int rl = m > 16 ? 32 : m > 8 ? 16 : 8;
    const int v0 = lane / rl, vs = 32 / rl;
    const int nv = (W - c0 - 8 + 3) >> 2;
    for (int pos = lane & (rl - 1); pos < m; pos += 32) {
        float* C = S + list[pos] * LDS + c0;
        float l[8];
        unpack(lds4(C), l);
        unpack(lds4(C + 4), l + 4);
#pragma unroll 2
        for (int v = v0; v < nv; v += vs) {
            const int col = 8 + 4 * v;
            float c[4];
            unpack(lds4(C + col), c);
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const float4 u = lds4(row[t] + col);
                fnma2(l[t], u.x, u.y, c[0], c[1]);
                fnma2(l[t], u.z, u.w, c[2], c[3]);
            }
            *reinterpret_cast<float4*>(C + col) = make_float4(c[0], c[1], c[2], c[3]);
        }
    }
}

// Blocked elimination of the n x n system in S (lists, held rows: asm_dmma.cuh).
// Returns whether a pivot left the range.
template <class L, int NRHS>
__device__ __forceinline__ bool eliminate(float* S, uint8_t* lists, uint8_t* piv, int n, int np, int lane) {
    constexpr int LDS = L::LDS, LSTRIDE = (L::NMAX + 15) / 16 * 16, RMAX = (L::NMAX + 31) / 32;
    const int W = n + NRHS;
    bool bad = false;
    int m = n;
    uint8_t *cur = lists, *nxt = lists + LSTRIDE;
#pragma unroll 1
    for (int c0 = 0; c0 < n; c0 += 8) {
        const int tend = min(8, n - c0);
        const int held = c0 == 0 && np >= 8 ? np : 0;
        const uint8_t* from = cur + held;
        const int mp = m - held;
        if (RMAX > 2 && mp > 64)
            bad |= panel<(RMAX > 2 ? 3 : 1), LDS>(S, from, nxt, piv, mp, held, c0, tend, lane);
        else if (RMAX > 1 && mp > 32)
            bad |= panel<(RMAX > 1 ? 2 : 1), LDS>(S, from, nxt, piv, mp, held, c0, tend, lane);
        else
            bad |= panel<1, LDS>(S, from, nxt, piv, mp, held, c0, tend, lane);
        __syncwarp();
        m -= tend;
        uint8_t* tmp = cur;
        cur = nxt;
        nxt = tmp;
        if (c0 + 8 < W) {
            const unsigned long long pr = *reinterpret_cast<const unsigned long long*>(piv + c0);
            const float* row[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) row[t] = S + dm::packed_row(pr, t < tend ? t : 0) * LDS + c0;
            pivot_rows<LDS>(S, row, c0, tend, W, lane);
            __syncwarp();
            update_rows<LDS>(S, row, cur + held, m - held, c0, W, lane);
            __syncwarp();
        }
    }
    return bad;
}

// The block row of the factors that lane (g, .) needs: 8 columns of its row.
__device__ __forceinline__ void block8(const float* s, float* u) {
    unpack(lds4(s), u);
    unpack(lds4(s + 4), u + 4);
}

// y = L^-1 y in place (unit lower factors), blocks of 8 steps in order. The
// blocks from nt on take part rather than a branch each, which would keep the
// chains of one block from overlapping: their entries of y hold no unknown
// afterwards, nor do those past n in the last block.
template <int NT>
__device__ __forceinline__ void forward(const float* S, const int (&prow)[NT], float (&y)[NT], int nt,
                                        int lane) {
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int b = 0; b < NT; ++b) {
        if (b < nt) {
            float l[8], z[8];
            block8(S + prow[b] + 8 * b, l);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                z[r] = __shfl_sync(0xffffffffu, y[b], 4 * r + q);
                y[b] = fmaf(r < g ? -l[r] : 0.f, z[r], y[b]);
            }
#pragma unroll
            for (int t = b + 1; t < NT; ++t) {
                float u[8];
                block8(S + prow[t] + 8 * b, u);
#pragma unroll
                for (int r = 0; r < 8; ++r) y[t] = fmaf(-u[r], z[r], y[t]);
            }
        }
    }
}

// y = U^-1 y in place, blocks of 8 steps from the last; steps past n give zero.
template <int NT>
__device__ __forceinline__ void backward(const float* S, const int (&prow)[NT], float (&y)[NT], int n,
                                         int nt, int lane) {
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int b = NT - 1; b >= 0; --b) {
        if (b < nt) {
            const float* row = S + prow[b] + 8 * b;
            float u[8], x[8];
            block8(row, u);
            const float dv = 8 * b + g < n ? row[g] : 0.f;  // 1 / pivot
#pragma unroll
            for (int r = 7; r >= 0; --r) {
                x[r] = __shfl_sync(0xffffffffu, y[b] * dv, 4 * r + q);
                y[b] = fmaf(r > g ? -u[r] : 0.f, x[r], y[b]);
            }
            y[b] = y[b] * dv;
#pragma unroll
            for (int t = 0; t < b; ++t) {
                float w[8];
                block8(S + prow[t] + 8 * b, w);
#pragma unroll
                for (int r = 7; r >= 0; --r) y[t] = fmaf(-w[r], x[r], y[t]);
            }
        }
    }
}

// b - M x, rounded to FP32 into S's right-hand-side columns (row order).
template <class L, int NRHS>
__device__ __forceinline__ void residual(float* S, const double* M, const double* b,
                                         const double (&x)[L::NT], int n, int nt, int lane) {
    constexpr int NT = L::NT;
    const int g = lane >> 2, q = lane & 3;
    const int down = cell(g, q), across = cell(q, g);  // fragments of a tile, of its transpose
    double c[NT][2];
#pragma unroll
    for (int I = 0; I < NT; ++I) {
        c[I][0] = 0.0;
        c[I][1] = 0.0;
        if (q < 2) {
            const double2 v = dm::lds2(b + 4 * (8 * I + g) + 2 * q);
            c[I][0] = v.x;
            c[I][1] = v.y;
        }
    }
#pragma unroll
    for (int J = 0; J < NT; ++J) {
        if (J < nt) {
            double x0 = __shfl_sync(0xffffffffu, x[J], 4 * q + (g & 3));
            double x1 = __shfl_sync(0xffffffffu, x[J], 16 + 4 * q + (g & 3));
            x0 = g < NRHS ? -x0 : 0.0;
            x1 = g < NRHS ? -x1 : 0.0;
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                const double* T = M + (I >= J ? I * (I + 1) / 2 + J : J * (J + 1) / 2 + I) * 64;
                dm::mma884(I >= J ? T[down] : T[across], x0, c[I][0], c[I][1]);
                dm::mma884(I >= J ? T[down ^ 4] : T[across + 32], x1, c[I][0], c[I][1]);
            }
        }
    }
#pragma unroll
    for (int I = 0; I < NT; ++I) {
        const int r = 8 * I + g;
        if (r < n) {
            float* dst = S + r * L::LDS + n + 2 * q;
            if (2 * q < NRHS) dst[0] = (float)c[I][0];
            if (2 * q + 1 < NRHS) dst[1] = (float)c[I][1];
        }
    }
}

// One stencil by one warp. fetched: its raw neighbour coordinates are on their
// way into xy; nx, if its s >= 0, is fetched for the next call. count: not a
// repetition (its statistics and its place in the list of the stalled are kept).
template <class L, int NRHS, int P, int Q>
__device__ __forceinline__ void assemble(const AsmParams& p, const Item& it, const Item& nx, bool fetched,
                                         bool count, char* base, int lane) {
    constexpr int NP = npoly(P), NT = L::NT;
    constexpr unsigned ALL = 0xffffffffu;
    double2* xy = reinterpret_cast<double2*>(base + L::off_xy);
    float* S = reinterpret_cast<float*>(base + L::off_s);
    double* M = reinterpret_cast<double*>(base + L::off_m);
    double* b = reinterpret_cast<double*>(base + L::off_b);
    uint8_t* lists = reinterpret_cast<uint8_t*>(base + L::off_list);
    uint8_t* piv = reinterpret_cast<uint8_t*>(base + L::off_piv);
    int* nja = reinterpret_cast<int*>(base + L::off_nja);
    const int g = lane >> 2, q = lane & 3;
    if (!fetched) dm::fetch_nodes<L, false>(p, it, base, lane);
    cp_async_wait_all();
    __syncwarp();
    const int ks = it.ks, n = NP + ks, nt = (n + 7) >> 3;
    const int e = dm::gather_scale<L::KMAX, true, false>(p, dm::offset_of(p, it), ks, it.x0, it.y0, xy, lane);
    __syncwarp();
    bool bad = fill_system<L, NRHS, P, Q>(p, S, M, b, xy, ks, e, lane);
    bad = bad || e < -dm::kMaxExp || e > dm::kMaxExp;
    __syncwarp();
    dm::init_order(lists, piv, n, lane);
    if (nx.s >= 0)
        for (int j = lane; j < nx.ks; j += 32) cp_async4(nja + j, p.ja + dm::offset_of(p, nx) + j);
    __syncwarp();
    bad = eliminate<L, NRHS>(S, lists, piv, n, NP, lane) || bad;
    bool failed = __any_sync(ALL, bad);
    if (nx.s >= 0) dm::fetch_nodes<L, true>(p, nx, base, lane);

    int prow[NT];
    float y[NT];
    double x[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) prow[t] = piv[8 * t + g < n ? 8 * t + g : 0] * L::LDS;
#pragma unroll
    for (int t = 0; t < NT; ++t) x[t] = 0.0;
    // one loop for the first solution and the sweeps: the substitutions are in
    // the code once (0.7k instructions, which the instruction cache feels)
    int sweeps = 0;
    float prev = 3.4e38f;
    for (;;) {
#pragma unroll
        for (int t = 0; t < NT; ++t)
            y[t] = 8 * t + g < n && q < NRHS ? S[prow[t] + n + q] : 0.f;
        __syncwarp();
        if (sweeps > 0) forward<NT>(S, prow, y, nt, lane);
        backward<NT>(S, prow, y, n, nt, lane);
        // x += d; convergence on max|d| / max|x| per right-hand side (as
        // magnitude words, so that a NaN wins)
        uint32_t dmax = 0, xmax = 0;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const float d = 8 * t + g < n ? y[t] : 0.f;  // only unknowns count
            x[t] = x[t] + (double)d;
            dmax = max(dmax, __float_as_uint(fabsf(d)));
            xmax = max(xmax, __float_as_uint(fabsf((float)x[t])));
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            dmax = max(dmax, __shfl_xor_sync(ALL, dmax, o));
            xmax = max(xmax, __shfl_xor_sync(ALL, xmax, o));
        }
        const float ratio = xmax ? __uint_as_float(dmax) / __uint_as_float(xmax) : __uint_as_float(dmax);
        const float worst = __uint_as_float(__reduce_max_sync(ALL, __float_as_uint(ratio)));
        // The correction of sweep k measures the error before it (tau_k);
        // the error left after it is about tau_k * rho / (1 - rho) with
        // rho = tau_k / tau_(k-1) the observed contraction (about
        // cond(M) * 2^-24). Converged when that prediction is below tol
        // (or the correction itself is at the FP64 floor). A contraction
        // above 0.1 means cond(M) > ~1e6: the prediction is unreliable
        // there and the FP64 rounding floor of the system itself nears the
        // tolerance, so such a stencil (and a NaN) goes to the FP64 kernel.
        if (sweeps > 0) {
            const float rho = sweeps >= 2 ? worst / fmaxf(prev, 1e-38f) : 1.0f;
            const float left = rho < 0.1f ? worst * rho / (1.0f - rho) : worst;
            if (!(worst == worst)) failed = true;
            else if (left <= (float)p.ir_tol || worst <= 1e-15f) break;
            else if (sweeps >= 2 && rho > 0.1f) failed = true;
            prev = worst;
        }
        failed = failed || sweeps >= p.max_sweeps;
        if (failed) break;
        ++sweeps;
        residual<L, NRHS>(S, M, b, x, n, nt, lane);
        __syncwarp();
    }
    if (lane == 0 && count) {
        if (p.sweeps_sum) atomicAdd(p.sweeps_sum, (unsigned long long)sweeps);
        if (p.sweeps_max) atomicMax(p.sweeps_max, sweeps);
        if (failed) {
            const int fo = p.list_off_dev ? *p.list_off_dev : 0;
            p.fb_list[fo + atomicAdd(p.fb_count, 1)] = it.s;
        } else if (p.info) {
            p.info[it.s - p.row_base] = 0;
        }
    }
    if (!failed && q < NRHS && q < p.nrhs) {
        // rescaled node weights, src/rbf_operators.h:368-375
        double* dst = out_column(p, q) + dm::offset_of(p, it);
        const int sh = -op_order(p.col_op[q]) * e;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int j = 8 * t + g - NP;
            if (j >= 0 && j < ks) dst[j] = dm::mul_pow2<false>(x[t], sh);
        }
    }
    __syncwarp();
}

// GPB stencils in flight a CTA, a persistent grid in a static stride; the CTA's
// stencils advance together for the instruction cache (asm_dmma.cuh).
template <int NMAX, int NRHS, int P, int Q, int GPB, int MINB>
__global__ void __launch_bounds__(32 * GPB, MINB) ir_kernel(const __grid_constant__ AsmParams p) {
    using L = Layout<NMAX, NRHS, NMAX - npoly(P)>;
    extern __shared__ __align__(16) char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    char* smem = smem_raw + warp * L::bytes;
    const int n = p.nitems_dev ? *p.nitems_dev : p.nitems;
    const int* list = (p.list && p.list_off_dev) ? p.list + *p.list_off_dev : p.list;
    const int stride = gridDim.x * GPB;
    // past the end a warp repeats the last stencil (it writes the same weights)
    auto item = [&](int i0) {
        const int i = min(i0 + warp, n - 1);
        return dm::item_of(p, list ? list[i] : p.item_base + i);
    };
    bool fetched = false;
    Item it{};
    int i0 = blockIdx.x * GPB;
    if (i0 < n) it = item(i0);
    for (; i0 < n; i0 += stride) {
        Item nx{-1, 0, 0, 0.0, 0.0};
        if (i0 + stride < n) nx = item(i0 + stride);
        if (GPB > 1) __syncthreads();
        assemble<L, NRHS, P, Q>(p, it, nx, fetched, i0 + warp < n, smem, lane);
        it = nx;
        fetched = true;
    }
}

}  // namespace ir
}  // namespace rbfb
