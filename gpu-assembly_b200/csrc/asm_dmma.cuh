// asm_dmma.cuh -- batched FP64 RBF-FD assembly on sm_100a: the saddle-point
// system in shared memory, a blocked right-looking Gaussian elimination with
// row-implicit partial pivoting whose trailing updates, and the block updates
// of the back substitution, run on the FP64 tensor cores (mma.sync m8n8k4).
//
// Replaces assemble_interp_weights<Config> (src/rbf_operators.h:292-376),
// whose solve is cuSolverDx gesv_partial_pivot with one stencil per CTA.
//
// Why the tensor cores give the same bits: on this part an FP64 m8n8k4
// multiply-accumulate is the chain of four fused multiply-adds in ascending k
// onto the accumulator, each rounded once. Two of them (k = 0..3, then
// 4..7) apply the eight updates of a panel, -l times u, in step order,
// which is what the scalar elimination does. The FP64 rate is that of the
// CUDA cores (64 multiply-adds a cycle per SM), but one instruction carries
// 256 of them, so the update of an 8 x 8 tile takes 2 multiply-adds, one
// 16-byte load and one store a lane instead of 16 and their operand loads:
// the kernel is bound by instruction issue and by the latency of its pivot
// chain, not by the FP64 pipe.
//
// A stencil belongs to NW warps. With NW = 1 a CTA holds several
// stencils, one a warp; with NW > 1 the CTA is one stencil: warp 0 runs the
// serial parts (the panels, the back substitution), the others share the fill
// and apply the trailing updates of panel p while warp 0, which updates the
// next panel's columns itself, already factors panel p + 1: one barrier a
// panel. The system is not padded: n = npoly(P) + k_s unknowns, any n <=
// NMAX, row-major in S (row = equation, column = unknown, then the NRHS
// right-hand sides), polynomial block first. Rows are never swapped: piv[c]
// is the row that became the pivot row at step c, and list[] holds the rows
// not yet used, ascending.
//
// Panel of columns c0 .. c0+7, lane l holding list positions l, l+32, ...:
//   1. the rows' 8 columns are loaded into registers;
//   2. 8 steps. Step c: the pivot is the unused row of largest key (the
//      magnitude word of a(r, c) without its 7 lowest bits, 127 - list
//      position in them: ties go to the lowest row -- the oracle's rule),
//      found by one redux.sync that was issued as soon as column c was
//      final; 1 / pivot and the pivot row's next column travel by shuffle
//      (they are on the serial chain), its other columns through S, where
//      the owner writes its final panel row with 1 / pivot in the pivot's
//      place; every unused row takes l = a(r,c) * (1 / pivot) and
//      a(r,j) = fma(-l, u(j), a(r,j)) for the panel columns j > c;
//   3. unused rows write their multipliers back; the list is compacted.
// Then, per 8-column tile right of the panel: the panel's pivot rows take the
// updates of the steps before theirs, and the unused rows (8 a tile) all 8.
//
// Back substitution from the last block of 8 steps: lane (g, q) holds the
// right-hand side q of the block's step g, the 8 steps run in registers
// (multiply by 1 / pivot, shuffle, fused multiply-add), and the rows of every
// earlier block take the block's 8 updates, last step first, as two m8n8k4.
// Steps below npoly(P), the polynomial multipliers, are not needed for the
// weights and not taken.
#pragma once

#include <cstdint>

#include "asm_common.cuh"

namespace rbfb {
namespace dm {

// Shared-memory (or global scratch) layout of one stencil.
template <int NMAX_, int NRHS, int KMAX_>
struct Layout {
    static constexpr int NMAX = NMAX_, KMAX = KMAX_;
    static constexpr int W = NMAX + NRHS;
    static_assert(NMAX <= 96, "pivot keys carry the list position in 7 bits");
    // Row stride in 16-byte vectors: odd, so the 32 rows a warp reads down
    // one column fall in different bank groups.
    static constexpr int LV0 = (W + 1) / 2;
    static constexpr int LDS = 2 * ((LV0 % 2) ? LV0 : LV0 + 1);
    static_assert((NMAX + 7) / 8 * 8 <= LDS, "a row holds every panel's columns");
    // whole 8-column tiles fit a row: the last tile needs no column check
    static constexpr bool kWhole = (W + 7) / 8 * 8 <= LDS;
    static constexpr int al16(int b) { return (b + 15) & ~15; }
    // the shifted, scaled neighbour coordinates (x, y); from the end of the
    // fill to the next stencil's prefetch the slot holds the two lists of
    // unused rows and the next stencil's ja row
    static constexpr int off_xy = 0;
    static constexpr int off_list = 0;
    static constexpr int off_nja = 2 * al16(NMAX);
    static constexpr int xy_bytes =
        al16(16 * KMAX > off_nja + 4 * KMAX ? 16 * KMAX : off_nja + 4 * KMAX);
    static constexpr int off_s = xy_bytes;
    static constexpr int off_piv = off_s + NMAX * LDS * 8;
    // shared between the stencil's warps: [2] a warp left the fast range, [3]
    // the scale exponent
    static constexpr int off_nia = off_piv + al16((NMAX + 7) / 8 * 8);
    static constexpr int bytes = off_nia + 16;
};

// All warps of a stencil.
template <int NW>
__device__ __forceinline__ void stencil_sync() {
    if constexpr (NW == 1)
        __syncwarp();
    else
        asm volatile("bar.sync 1, %0;\n" ::"n"(NW * 32) : "memory");
}

__device__ __forceinline__ void mma884(double a, double b, double& c0, double& c1) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

__device__ __forceinline__ double2 lds2(const double* s) { return *reinterpret_cast<const double2*>(s); }
__device__ __forceinline__ void sts2(double* s, double a, double b) {
    *reinterpret_cast<double2*>(s) = make_double2(a, b);
}

// The fast path's range: operands of the branch-free reciprocal and square
// root, and pivots, have a magnitude word (high 32 bits without the sign) in
// [kLow, kHigh), |x| in [2^-900, 2^900); the scale exponent is at most kMaxExp
// in magnitude. A stencil that leaves it (coincident nodes, a zero pivot, an
// infinity or NaN, a value that the branch-free forms do not cover) is redone
// by the careful path, whose results are the plain algorithm's.
constexpr uint32_t kLow = 123u << 20, kHigh = 1923u << 20;
constexpr int kMaxExp = 500;

// 1 / a, correctly rounded, for the fast range and a low word other than ~0. From an
// approximation y of at least 20 bits, with e = 1 - a y (|e| < 2^-20, to 2^-53 of
// itself): 1 / a = y / (1 - e) = y (1 + e + e^2 + e^3 + ...). y + y (e + e^2) leaves e^3
// < 2^-60 and its own rounding: within 1/2 + 2^-7 ulp of 1 / a. The residual 1 - a y
// of such a y is exact in one fused multiply-add, and Markstein's final step y + y (1 - a y)
// then rounds correctly for every a whose mantissa is not all ones (P. Markstein, IA-64
// and Elementary Functions, 2000, ch. 8).
__device__ __forceinline__ double rcp_fast(double a) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-a, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    return fma(y, fma(-a, y, 1.0), y);
}

// sqrt(a), correctly rounded, for the fast range (same source, ch. 9). From y ~ 1 /
// sqrt(a) of at least 20 bits: g = a y, h = y / 2, and r = 1/2 - g h, so that a y^2 = 1 - 2 r
// and sqrt(a) = g (1 - 2 r)^(-1/2) = g (1 + r + 3/2 r^2 + 5/2 r^3 + ...), likewise 1 / (2
// sqrt(a)) from h. Two terms leave 5/2 r^3 < 2^-58 and the rounding; the residual a - g^2
// is exact in one fused multiply-add, and g + h (a - g^2) rounds correctly.
__device__ __forceinline__ double sqrt_fast(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    double g = dmul(a, y), h = dmul(0.5, y);
    const double r = fma(-g, h, 0.5);
    const double t = fma(dmul(1.5, r), r, r);
    g = fma(g, t, g);
    h = fma(h, t, h);
    return fma(h, fma(-g, g, a), g);
}

// phi(r) = r^Q from r^2 in the reference's product order (phs64).
template <int Q>
__device__ __forceinline__ double phs_fast(double r2) {
    const double s = sqrt_fast(r2);
    if constexpr (Q == 1) {
        return s;
    } else if constexpr (Q == 3) {
        return dmul(r2, s);
    } else if constexpr (Q == 5) {
        return dmul(dmul(r2, r2), s);
    } else if constexpr (Q == 7) {
        const double r4 = dmul(r2, r2);
        return dmul(dmul(r4, r2), s);
    } else {
        double p = s;
#pragma unroll
        for (int i = 0; i < (Q - 1) / 2; ++i) p = dmul(p, r2);
        return p;
    }
}

__device__ __forceinline__ uint32_t mag_word(double v) { return (uint32_t)__double2hiint(v) & 0x7fffffffu; }

// x * 2^e, rounded once (as scalbn).
template <bool CAREFUL>
__device__ __forceinline__ double mul_pow2(double x, int e) {
    if constexpr (CAREFUL) return scalbn(x, e);
    return dmul(x, __hiloint2double((1023 + e) << 20, 0));
}

// Gather + FP64 shift to the centre (x0, y0) (+ minimum image), and the
// power-of-two radius scale (src/rbf_operators.h:354-358), by one warp. With
// PF xy holds the raw prefetched coordinates on entry. Returns the exponent.
template <int KMAX, bool PF, bool CAREFUL>
__device__ __forceinline__ int gather_scale(const AsmParams& p, long long off, int ks, double x0,
                                            double y0, double2* xy, int lane) {
    constexpr int KPL = (KMAX + 31) / 32;
    double gx[KPL], gy[KPL];
    bool far = false;
#pragma unroll
    for (int t = 0; t < KPL; ++t) {
        const int j = lane + t * 32;
        gx[t] = 0.0;
        gy[t] = 0.0;
        if (j < ks) {
            double2 v;
            if constexpr (PF) {
                v = xy[j];
            } else {
                const int nb = __ldg(p.ja + off + j);
                v = make_double2(__ldg(p.x + nb), __ldg(p.y + nb));
            }
            gx[t] = dsub(v.x, x0);
            gy[t] = dsub(v.y, y0);
            far = far || !(fabs(gx[t]) < 0.25 * p.Lx) || !(fabs(gy[t]) < 0.25 * p.Ly);
        }
    }
    // the minimum image d - L rint(d / L): below a quarter period the quotient
    // rounds to zero and the result is d itself, without the division
    if (p.Lx > 0.0 || p.Ly > 0.0) {
        if (__any_sync(0xffffffffu, far)) {
#pragma unroll
            for (int t = 0; t < KPL; ++t) {
                gx[t] = min_image(gx[t], p.Lx);
                gy[t] = min_image(gy[t], p.Ly);
            }
        }
    }
    int e;
    if constexpr (CAREFUL) {
        int emax = -100000;
#pragma unroll
        for (int t = 0; t < KPL; ++t) {
            if (gx[t] != 0.0) emax = max(emax, ilogb(fabs(gx[t])) + 1);
            if (gy[t] != 0.0) emax = max(emax, ilogb(fabs(gy[t])) + 1);
        }
        e = __reduce_max_sync(0xffffffffu, emax);
        e = (p.scale && e > -100000) ? e : 0;
    } else {
        uint32_t w = 0;
#pragma unroll
        for (int t = 0; t < KPL; ++t) w = max(w, max(mag_word(gx[t]), mag_word(gy[t])));
        w = __reduce_max_sync(0xffffffffu, w);
        e = (p.scale && w) ? (int)(w >> 20) - 1022 : 0;
    }
#pragma unroll
    for (int t = 0; t < KPL; ++t) {
        const int j = lane + t * 32;
        if (j < ks)
            xy[j] = make_double2(mul_pow2<CAREFUL>(gx[t], -e), mul_pow2<CAREFUL>(gy[t], -e));
    }
    return e;
}

// phi of the pair (i, j) into S's phi block Sn (both halves); its squared
// distance's magnitude into [wmin, wmax].
template <int LDS, int Q, bool CAREFUL>
__device__ __forceinline__ void fill_pair(double* Sn, int i, int j, double2 a, double2 b, uint32_t& wmin,
                                          uint32_t& wmax) {
    const double r2 = dist2(dsub(b.x, a.x), dsub(b.y, a.y));
    double v;
    if constexpr (CAREFUL) {
        v = phs64<Q>(r2);
    } else {
        v = phs_fast<Q>(r2);
        wmin = min(wmin, (uint32_t)__double2hiint(r2));
        wmax = max(wmax, (uint32_t)__double2hiint(r2));
    }
    Sn[i * LDS + j] = v;
    Sn[j * LDS + i] = v;
}

// The right-hand sides of a node row for the operators Laplace, d/dx, d/dy
// alone (rhs_node's products, in its order).
template <int Q, int NRHS>
__device__ __forceinline__ void rhs_plain(const AsmParams& p, double xi, double yi, double* out,
                                          uint32_t& wmin, uint32_t& wmax) {
    const double r2 = dist2(xi, yi);
    const double rq2 = r2 == 0.0 ? 0.0 : phs_fast<Q - 2>(r2);
    wmin = min(wmin, r2 == 0.0 ? kLow : (uint32_t)__double2hiint(r2));
    wmax = max(wmax, (uint32_t)__double2hiint(r2));
    const double q = static_cast<double>(Q);
    const double qr = dmul(q, rq2);
#pragma unroll
    for (int c = 0; c < NRHS; ++c) {
        double v = 0.0;
        if (c < p.nrhs) {
            if (p.col_op[c] == kOpLaplace)
                v = dmul(q * q, rq2);
            else
                v = -dmul(qr, p.col_op[c] == kOpDx ? xi : yi);
        }
        out[c] = v;
    }
}

// The augmented system in S: phi block (each unordered pair once), monomial
// rows and columns, zero polynomial block, right-hand sides as columns n ..
// n+NRHS-1 (fill_matrix / fill_rhs, src/rbf_operators.h:116-185), and zeros in
// the columns past them that the back substitution's last block reads.
// The pairs are (i, i + d mod k), d = 1 .. k/2 (phi is symmetric to the bit: it
// takes squared differences). Whole groups of 32 rows: a lane keeps its row's
// coordinates and walks d. The other rows: flat over the threads, d outermost.
// Returns whether a value left the fast range (never with CAREFUL).
template <int LDS, int NRHS, int P, int Q, int NW, bool CAREFUL>
__device__ __forceinline__ bool fill_system(const AsmParams& p, double* S, const double2* xy, int ks,
                                            int e, int warp, int lane) {
    constexpr int NP = npoly(P), NT = 32 * NW;
    const int tid = 32 * warp + lane;
    const int n = NP + ks;
    uint32_t wmin = kLow, wmax = 0;
    double* Sn = S + NP * LDS + NP;
    const int half = (ks - 1) >> 1;  // whole shifts d; even ks: d = ks / 2 meets each pair twice
    const int ib = ks & ~31;
    for (int i0 = 0; i0 < ib; i0 += 32) {
        const int i = i0 + lane;
        const double2 a = xy[i];
        int j = i + 1 + warp;
        j = j >= ks ? j - ks : j;
        const int dend = half + ((ks & 1) == 0 && i < ks / 2 ? 1 : 0);
        for (int d = 1 + warp; d <= dend; d += NW) {
            fill_pair<LDS, Q, CAREFUL>(Sn, i, j, a, xy[j], wmin, wmax);
            j += NW;
            j = j >= ks ? j - ks : j;
        }
    }
    {
        const int rows = ks - ib, count = ib ? rows * half : ks * (ks - 1) / 2;
        int i = ib + tid, d = 1;
        if (rows > 0) {
            while (i >= ks) {
                i -= rows;
                ++d;
            }
            for (int t = tid; t < count; t += NT) {
                int j = i + d;
                j = j >= ks ? j - ks : j;
                fill_pair<LDS, Q, CAREFUL>(Sn, i, j, xy[i], xy[j], wmin, wmax);
                i += NT;
                while (i >= ks) {
                    i -= rows;
                    ++d;
                }
            }
        }
    }
    const int wend = (n + 7) & ~7;
    for (int i = tid; i < ks; i += NT) {
        const int r = NP + i;
        double* Sr = S + r * LDS;
        const double2 c = xy[i];
        double mon[NP + 1];
        monomials<P>(c.x, c.y, mon);
#pragma unroll
        for (int m = 0; m + 1 < NP; m += 2) sts2(Sr + m, mon[m], mon[m + 1]);
        if (NP & 1) Sr[NP - 1] = mon[NP - 1];
#pragma unroll
        for (int m = 0; m < NP; ++m) S[m * LDS + r] = mon[m];
        Sr[r] = 0.0;
        double rv[NRHS];
        if (!CAREFUL && p.plain_ops) {
            rhs_plain<Q, NRHS>(p, c.x, c.y, rv, wmin, wmax);
        } else {
            rhs_node<P, Q, NRHS>(p, c.x, c.y, e, rv);
#pragma unroll
            for (int q = 0; q < NRHS; ++q) wmax = max(wmax, mag_word(rv[q]));
        }
#pragma unroll
        for (int q = 0; q < NRHS; ++q) Sr[n + q] = rv[q];
    }
    for (int f = tid; f < NP * NP; f += NT) S[(f / NP) * LDS + f % NP] = 0.0;
    for (int f = tid; f < NP * NRHS; f += NT) {
        const int r = f / NRHS, q = f % NRHS;
        S[r * LDS + n + q] = q < p.nrhs ? rhs_poly<P>(p, q, r, e) : 0.0;
    }
    for (int c = n + NRHS; c < wend; ++c)
        for (int r = tid; r < n; r += NT) S[r * LDS + c] = 0.0;
    return !CAREFUL && (wmin < kLow || wmax >= kHigh);
}

// One lane's R list positions of a panel: the rows' 8 panel columns, their
// byte offsets in S and the operands of their pivot keys.
template <int R>
struct PanelRows {
    double a[R][8];
    int off[R];  // byte offset in S of the row's panel columns
    uint32_t kmask[R], kcon[R];
    int keep[R];  // leading column pairs that store_panel still has to write
};

template <int R, int LDS>
__device__ __forceinline__ void load_panel(PanelRows<R>& w, const char* Sc, const uint8_t* list,
                                           int m, int lane) {
#pragma unroll
    for (int sl = 0; sl < R; ++sl) {
        const int pos = lane + 32 * sl;
        const bool v = pos < m;
        w.off[sl] = list[v ? pos : 0] * (LDS * 8);
        w.kmask[sl] = v ? 0x7fffff80u : 0u;
        w.kcon[sl] = v ? 127u - (uint32_t)pos : 0u;
        w.keep[sl] = v ? 4 : 0;
        const double* src = reinterpret_cast<const double*>(Sc + w.off[sl]);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const double2 x = lds2(src + j);
            w.a[sl][j] = x.x;
            w.a[sl][j + 1] = x.y;
        }
    }
}

// The multipliers back to S (a pivot row's own were written with it from the
// pair of its step on), the list of the rows still unused compacted into next
// from position base. Returns the position after them.
template <int R, int LDS>
__device__ __forceinline__ int store_panel(const PanelRows<R>& w, char* Sc, uint8_t* next, int base,
                                           int lane) {
#pragma unroll
    for (int sl = 0; sl < R; ++sl) {
        double* dst = reinterpret_cast<double*>(Sc + w.off[sl]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < w.keep[sl]) sts2(dst + 2 * j, w.a[sl][2 * j], w.a[sl][2 * j + 1]);
        const bool alive = w.kmask[sl] != 0u;
        const unsigned b = __ballot_sync(0xffffffffu, alive);
        if (alive)
            next[base + __popc(b & ((1u << lane) - 1u))] = (uint8_t)(w.off[sl] / (LDS * 8));
        base += __popc(b);
    }
    return base;
}

// The steps of one panel (columns c0 .. c0 + 7, the first tend of them) on the
// m rows of list, by one warp with R list positions a lane; next receives the
// rows 0 .. held-1, which sit this panel out, and the rows still unused. One basic block (two for the last panel), no slow paths:
// the scheduler fills the latencies of the pivot chain. Steps past tend run on
// a dummy candidate that loses to every pivot of the fast range and stores
// nothing. Returns whether a pivot left the fast range.
template <int R, int LDS>
__device__ __forceinline__ bool panel(double* S, const uint8_t* list, uint8_t* next, uint8_t* piv,
                                      int m, int held, int c0, int tend, int lane) {
    constexpr unsigned ALL = 0xffffffffu;
    char* Sc = reinterpret_cast<char*>(S + c0);
    PanelRows<R> w;
    load_panel<R, LDS>(w, Sc, list, m, lane);
    if (R == 1 && lane == 31 && tend < 8) w.kcon[0] = kLow | 96u;
    // this lane's best candidate of column t: its key, its slot, its value
    uint32_t key;
    int bsl;
    double bv;
    auto keys = [&](int t) {
        key = ((uint32_t)__double2hiint(w.a[0][t]) & w.kmask[0]) | w.kcon[0];
        bsl = 0;
        bv = w.a[0][t];
#pragma unroll
        for (int sl = 1; sl < R; ++sl) {
            const uint32_t kk = ((uint32_t)__double2hiint(w.a[sl][t]) & w.kmask[sl]) | w.kcon[sl];
            const bool better = kk > key;
            bv = better ? w.a[sl][t] : bv;
            bsl = better ? sl : bsl;
            key = better ? kk : key;
        }
    };
    keys(0);
    uint32_t best = __reduce_max_sync(ALL, key), low = kHigh, high = 0;
    bool odd = false;
    auto step = [&](int t) {
        low = min(low, best);
        high = max(high, best);
        odd = odd || __double2loint(bv) == -1;
        const double rv = rcp_fast(bv);  // 1 / pivot, if this lane owns the pivot
        const int owner = (int)(~best & 31u);
        int off = w.off[0];
        double bn = w.a[0][t + 1 < 8 ? t + 1 : t];
#pragma unroll
        for (int sl = 1; sl < R; ++sl) {
            off = bsl == sl ? w.off[sl] : off;
            if (t + 1 < 8) bn = bsl == sl ? w.a[sl][t + 1] : bn;
        }
        const double inv = __shfl_sync(ALL, rv, owner);
        const double un = t + 1 < 8 ? __shfl_sync(ALL, bn, owner) : 0.0;
        const double* U = reinterpret_cast<const double*>(Sc + __shfl_sync(ALL, off, owner));
        const bool own = lane == owner && (R > 1 || w.kmask[0]);
#pragma unroll
        for (int sl = 0; sl < R; ++sl) {
            const bool used = own && (R == 1 || bsl == sl);
            if (used) {
                double* dst = reinterpret_cast<double*>(Sc + w.off[sl]);
#pragma unroll
                for (int j = t & ~1; j < 8; j += 2)  // 1 / pivot in the pivot's place
                    sts2(dst + j, j == t ? rv : w.a[sl][j], j + 1 == t ? rv : w.a[sl][j + 1]);
                piv[c0 + t] = (uint8_t)(w.off[sl] / (LDS * 8));
            }
            w.kmask[sl] = used ? 0u : w.kmask[sl];
            w.kcon[sl] = used ? 0u : w.kcon[sl];
            w.keep[sl] = used ? t >> 1 : w.keep[sl];
        }
        // multipliers (a row already used is never stored again)
#pragma unroll
        for (int sl = 0; sl < R; ++sl) {
            w.a[sl][t] = dmul(w.a[sl][t], inv);
            if (t + 1 < 8) w.a[sl][t + 1] = fma(-w.a[sl][t], un, w.a[sl][t + 1]);
        }
        if (t + 1 < 8) {
            keys(t + 1);
            best = __reduce_max_sync(ALL, key);
        }
        __syncwarp();
        if (t + 2 < 8) {
            double u[8];
#pragma unroll
            for (int j = ((t + 2) / 2) * 2; j < 8; j += 2) {
                const double2 x = lds2(U + j);
                u[j] = x.x;
                u[j + 1] = x.y;
            }
#pragma unroll
            for (int j = t + 2; j < 8; ++j)
#pragma unroll
                for (int sl = 0; sl < R; ++sl) w.a[sl][j] = fma(-w.a[sl][t], u[j], w.a[sl][j]);
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
    const int left = store_panel<R, LDS>(w, Sc, next, held, lane);
    return odd || low < kLow || high >= kHigh || left != held + m - tend;
}

// The same steps for any pivot: correctly rounded quotients of every kind,
// the status of a zero pivot in info.
template <int R, int LDS>
__device__ __forceinline__ void panel_careful(double* S, const uint8_t* list, uint8_t* next,
                                              uint8_t* piv, int m, int c0, int tend, int lane,
                                              int& info) {
    constexpr unsigned ALL = 0xffffffffu;
    char* Sc = reinterpret_cast<char*>(S + c0);
    PanelRows<R> w;
    load_panel<R, LDS>(w, Sc, list, m, lane);
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        if (t >= tend) break;
        uint32_t key = 0;
        double bv = 1.0;
#pragma unroll
        for (int sl = 0; sl < R; ++sl) {
            const uint32_t kk = ((uint32_t)__double2hiint(w.a[sl][t]) & w.kmask[sl]) | w.kcon[sl];
            bv = kk > key ? w.a[sl][t] : bv;
            key = max(kk, key);
        }
        const uint32_t best = __reduce_max_sync(ALL, key);
        if (best < 128u && info == 0) info = c0 + t + 1;  // zero pivot column
        const int pos = 127 - (int)(best & 127u);
        const double rv = __drcp_rn(bv);
        const double inv = __shfl_sync(ALL, rv, pos & 31);
#pragma unroll
        for (int sl = 0; sl < R; ++sl) {
            if (lane + 32 * sl == pos) {
                double* dst = reinterpret_cast<double*>(Sc + w.off[sl]);
#pragma unroll
                for (int j = 0; j < 8; ++j) dst[j] = j == t ? rv : w.a[sl][j];
                piv[c0 + t] = (uint8_t)(w.off[sl] / (LDS * 8));
                w.kmask[sl] = 0u;
                w.kcon[sl] = 0u;
                w.keep[sl] = 0;
            }
        }
        __syncwarp();
        const double* U = reinterpret_cast<const double*>(Sc) + list[pos] * LDS;
#pragma unroll
        for (int sl = 0; sl < R; ++sl) {
            w.a[sl][t] = dmul(w.a[sl][t], inv);
#pragma unroll
            for (int j = t + 1; j < 8; ++j) w.a[sl][j] = fma(-w.a[sl][t], U[j], w.a[sl][j]);
        }
    }
    store_panel<R, LDS>(w, Sc, next, 0, lane);
}

// Row of S of step c0 + t, t = 0..7, from the packed pivot order.
__device__ __forceinline__ int packed_row(unsigned long long pr, int t) {
    return (int)((pr >> (8 * t)) & 0xffu);
}

// The panel's pivot rows over the 8-column tiles ct, ct + step, ... < nct
// right of it: row t takes the updates of the steps t' < t, in order. A lane
// takes one 16-byte vector of columns, 8 tiles a pass.
template <int LDS>
__device__ __forceinline__ void pivot_rows(double* S, unsigned long long pr, int c0, int tend, int ct,
                                           int step, int nct, int W, int lane) {
    double* row[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) row[t] = S + packed_row(pr, t < tend ? t : 0) * LDS + c0;
    for (int ct0 = ct; ct0 < nct; ct0 += 8 * step) {
        const int my = ct0 + (lane >> 2) * step;
        const int col = 8 + 8 * my + 2 * (lane & 3);  // from c0
        if (my < nct && c0 + col < W) {
            double u[8][2];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const double2 w = lds2(row[t] + col);
                u[t][0] = w.x;
                u[t][1] = w.y;
            }
            double l[8][8];
#pragma unroll
            for (int t = 1; t < 8; ++t)
#pragma unroll
                for (int tp = 0; tp < t; tp += 2) {
                    const double2 w = lds2(row[t] + tp);
                    l[t][tp] = w.x;
                    l[t][tp + 1] = w.y;
                }
#pragma unroll
            for (int tp = 0; tp < 7; ++tp)
#pragma unroll
                for (int t = tp + 1; t < 8; ++t) {
                    u[t][0] = fma(-l[t][tp], u[tp][0], u[t][0]);
                    u[t][1] = fma(-l[t][tp], u[tp][1], u[t][1]);
                }
#pragma unroll
            for (int t = 1; t < 8; ++t)
                if (t < tend) sts2(row[t] + col, u[t][0], u[t][1]);
        }
    }
}

// The unused rows at list positions pos0 .. pos0 + 8 RT - 1 (those below m)
// over the tiles ct, ct + step, ... < nct: C -= L U, the panel's 8 steps in
// order, as two m8n8k4 a tile. The fragments' row g is list position
// bitreverse(g) of its tile: the two rows of a quarter warp (16-byte accesses
// of C) are four positions apart, the four of a half warp (8-byte accesses
// of L) two: no bank conflict while the list is dense.
template <int RT, int LDS, bool WHOLE>
__device__ __forceinline__ void update_tiles(double* S, const uint8_t* list, unsigned long long pr,
                                             int pos0, int m, int c0, int ct, int step, int nct,
                                             int W, int lane) {
    const int g = lane >> 2, q = lane & 3;
    const double* b0 = S + packed_row(pr, q) * LDS + c0 + g;
    const double* b1 = S + packed_row(pr, q + 4) * LDS + c0 + g;
    double l0[RT], l1[RT];
    double* cp[RT];
    bool ok[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) {
        const int pos = pos0 + 8 * r + ((g & 1) << 2) + (g & 2) + (g >> 2);
        ok[r] = pos < m;
        double* row = S + list[ok[r] ? pos : 0] * LDS + c0;
        l0[r] = -row[q];
        l1[r] = -row[q + 4];
        cp[r] = row + 2 * q;
    }
#pragma unroll 1
    for (; ct < nct; ct += step) {
        const int col = 8 + 8 * ct;  // from c0
        const bool bin = WHOLE || c0 + col + g < W;
        const bool cin = WHOLE || c0 + col + 2 * q < W;
        const double u0 = bin ? b0[col] : 0.0, u1 = bin ? b1[col] : 0.0;
        double c[RT][2];
#pragma unroll
        for (int r = 0; r < RT; ++r) {
            const double2 w = cin ? lds2(cp[r] + col) : make_double2(0.0, 0.0);
            c[r][0] = w.x;
            c[r][1] = w.y;
        }
#pragma unroll
        for (int r = 0; r < RT; ++r) mma884(l0[r], u0, c[r][0], c[r][1]);
#pragma unroll
        for (int r = 0; r < RT; ++r) mma884(l1[r], u1, c[r][0], c[r][1]);
#pragma unroll
        for (int r = 0; r < RT; ++r)
            if ((r + 1 < RT || ok[r]) && cin) sts2(cp[r] + col, c[r][0], c[r][1]);
    }
}

template <int NMAX, int LDS, bool WHOLE>
__device__ __forceinline__ void trailing(double* S, const uint8_t* list, const uint8_t* piv, int m,
                                         int c0, int tend, int ct, int step, int nct, int W,
                                         int lane) {
    const unsigned long long pr = *reinterpret_cast<const unsigned long long*>(piv + c0);
    pivot_rows<LDS>(S, pr, c0, tend, ct, step, nct, W, lane);
    __syncwarp();
    // row tiles in groups of up to 4 (their multipliers stay in registers)
    for (int pos0 = 0; pos0 < m; pos0 += 32) {
        switch (min((m - pos0 + 7) / 8, 4)) {
            case 1: update_tiles<1, LDS, WHOLE>(S, list, pr, pos0, m, c0, ct, step, nct, W, lane); break;
            case 2: update_tiles<2, LDS, WHOLE>(S, list, pr, pos0, m, c0, ct, step, nct, W, lane); break;
            case 3: update_tiles<3, LDS, WHOLE>(S, list, pr, pos0, m, c0, ct, step, nct, W, lane); break;
            default: update_tiles<4, LDS, WHOLE>(S, list, pr, pos0, m, c0, ct, step, nct, W, lane); break;
        }
    }
}

// The list of unused rows: all of them. Every step of the pivot order starts as
// a valid row: a panel whose pivots leave the fast range may end before it has
// set them all, and its entries are read before the stencil is redone.
__device__ __forceinline__ void init_order(uint8_t* list, uint8_t* piv, int n, int lane) {
    for (int r = lane; r < n; r += 32) {
        list[r] = (uint8_t)r;
        piv[r] = (uint8_t)r;
    }
}

// Blocked right-looking elimination of the n x n system in S with its NRHS
// right-hand-side columns. lists: two lists of NMAX (rounded up to 16)
// entries, the first holding 0 .. n-1. A panel whose columns all lie in the
// zero polynomial block (c0 = 0 when np >= 8; np <= 15) leaves the polynomial
// rows out: they are zero there, so no candidate and no multiplier is lost. The result (warp
// 0): 0, or with CAREFUL c + 1 for the first zero pivot, without it nonzero
// when a pivot left the fast range. Ends with a barrier of the stencil's warps.
template <int NMAX, int LDS, bool WHOLE, int NRHS, int NW, bool CAREFUL>
__device__ __forceinline__ int eliminate(double* S, uint8_t* lists, uint8_t* piv, int n, int np,
                                         int warp, int lane) {
    constexpr int LSTRIDE = (NMAX + 15) / 16 * 16, RMAX = (NMAX + 31) / 32;
    const int W = n + NRHS;
    int info = 0, m = n;
    uint8_t *cur = lists, *nxt = lists + LSTRIDE;
#pragma unroll 1
    for (int c0 = 0; c0 < n; c0 += 8) {
        const int tend = min(8, n - c0);
        const int held = !CAREFUL && c0 == 0 && np >= 8 ? np : 0;
        if (NW == 1 || warp == 0) {
            const uint8_t* from = cur + held;
            const int mp = m - held;
            if constexpr (CAREFUL)
                panel_careful<RMAX, LDS>(S, cur, nxt, piv, m, c0, tend, lane, info);
            else if (RMAX > 2 && mp > 64)
                info |= panel<(RMAX > 2 ? 3 : 1), LDS>(S, from, nxt, piv, mp, held, c0, tend, lane);
            else if (RMAX > 1 && mp > 32)
                info |= panel<(RMAX > 1 ? 2 : 1), LDS>(S, from, nxt, piv, mp, held, c0, tend, lane);
            else
                info |= panel<1, LDS>(S, from, nxt, piv, mp, held, c0, tend, lane);
        }
        stencil_sync<NW>();
        m -= tend;
        uint8_t* tmp = cur;
        cur = nxt;
        nxt = tmp;
        const int nct = (W - c0 - 8 + 7) / 8;  // 8-column tiles right of the panel
        if (nct > 0) {
            const uint8_t* rows = cur + held;
            if constexpr (NW == 1) {
                trailing<NMAX, LDS, WHOLE>(S, rows, piv, m - held, c0, tend, 0, 1, nct, W, lane);
            } else if (warp == 0) {
                trailing<NMAX, LDS, WHOLE>(S, rows, piv, m - held, c0, tend, 0, 1, 1, W, lane);
            } else {
                trailing<NMAX, LDS, WHOLE>(S, rows, piv, m - held, c0, tend, warp, NW - 1, nct, W,
                                           lane);
            }
        }
        __syncwarp();
    }
    if (NW > 1) stencil_sync<NW>();
    return info;
}

// Back substitution (one warp) down to step cstop, the weights written as
// they come: out(q)[j] of unknown cstop + j, rescaled (src/rbf_operators.h:
// 368-375); NaN for a singular stencil. The blocks are whole: x of the steps
// past the last unknown is zero (their coefficients, the right-hand sides and
// the zeros after them, are finite; with CAREFUL they are taken as zero), and
// the steps of the last block below cstop are taken but not written.
template <int LDS, int NRHS, bool CAREFUL>
__device__ __forceinline__ void back_substitute(const AsmParams& p, double* S, const uint8_t* piv,
                                                int n, int cstop, long long off, int e, int info,
                                                int lane) {
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int SL = (NRHS + 3) / 4;  // right-hand sides a lane
    const int g = lane >> 2, q = lane & 3;
    double* dst[SL];
    int sh[SL];
#pragma unroll
    for (int s = 0; s < SL; ++s) {
        const int col = q + 4 * s;
        dst[s] = nullptr;
        sh[s] = 0;
        if (col < p.nrhs) {
            dst[s] = out_column(p, col) + off;
            sh[s] = -op_order(p.col_op[col]) * e;
        }
    }
    const int b0 = cstop >> 3;
#pragma unroll 1
    for (int b = (n - 1) >> 3; b >= b0; --b) {
        const int c = 8 * b + g;  // this lane's step
        const bool in = c < n;
        const double* row = S + piv[in ? c : 0] * LDS + 8 * b;
        double u[8], x[SL], y[SL];
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const double2 w = lds2(row + j);
            u[j] = !CAREFUL || 8 * b + j < n ? w.x : 0.0;
            u[j + 1] = !CAREFUL || 8 * b + j + 1 < n ? w.y : 0.0;
        }
        const double dv = in ? row[g] : 0.0;  // 1 / pivot
#pragma unroll
        for (int s = 0; s < SL; ++s) {
            const int col = q + 4 * s;
            y[s] = (in && col < NRHS) ? row[n - 8 * b + col] : 0.0;
            x[s] = 0.0;
        }
#pragma unroll
        for (int r = 7; r >= 0; --r) {
#pragma unroll
            for (int s = 0; s < SL; ++s) {
                const double v = dmul(y[s], dv);  // x in the lanes of step r
                x[s] = g == r ? v : x[s];
                y[s] = fma(-u[r], __shfl_sync(ALL, v, 4 * r + q), y[s]);
            }
        }
        const int j = c - cstop;
#pragma unroll
        for (int s = 0; s < SL; ++s)
            if (dst[s] && in && j >= 0)
                dst[s][j] = CAREFUL && info ? __longlong_as_double(0x7ff8000000000000ll)
                                            : mul_pow2<CAREFUL>(x[s], sh[s]);
        if (b == b0) break;
        // the rows of the earlier blocks take the block's steps, last first:
        // fragment k is step 7 - k (k < 4), 3 - (k - 4) (k >= 4)
        double x0 = __shfl_sync(ALL, x[0], 4 * (7 - q) + (g & 3));
        double x1 = __shfl_sync(ALL, x[0], 4 * (3 - q) + (g & 3));
        if constexpr (SL > 1) {
            const double k0 = __shfl_sync(ALL, x[SL - 1], 4 * (7 - q) + (g & 3));
            const double k1 = __shfl_sync(ALL, x[SL - 1], 4 * (3 - q) + (g & 3));
            x0 = g < 4 ? x0 : k0;
            x1 = g < 4 ? x1 : k1;
        }
        x0 = g < NRHS ? x0 : 0.0;
        x1 = g < NRHS ? x1 : 0.0;
        const bool in0 = !CAREFUL || 8 * b + 7 - q < n, in1 = !CAREFUL || 8 * b + 3 - q < n;
        const int yo = n + 2 * q - 8 * b;
#pragma unroll 1
        for (int t = b - 1; t >= b0; --t) {
            double* tr = S + piv[8 * t + g] * LDS + 8 * b;
            const double u0 = in0 ? -tr[7 - q] : 0.0;
            const double u1 = in1 ? -tr[3 - q] : 0.0;
            double y0 = 2 * q < NRHS ? tr[yo] : 0.0;
            double y1 = 2 * q + 1 < NRHS ? tr[yo + 1] : 0.0;
            mma884(u0, x0, y0, y1);
            mma884(u1, x1, y0, y1);
            if (2 * q < NRHS) tr[yo] = y0;
            if (2 * q + 1 < NRHS) tr[yo + 1] = y1;
        }
        __syncwarp();
    }
}

// The degree and PHS exponent of a stencil: fixed at compile time, or (P < 0)
// the stencil's own.
template <int P_, int Q_>
struct Shape {
    static constexpr int P = P_, Q = Q_;
    int p, q;
    __device__ __forceinline__ int np() const { return P >= 0 ? npoly(P) : npoly(p); }
};

template <int LDS, int NRHS, int P, int NW, bool CAREFUL>
__device__ __forceinline__ bool fill_q(const AsmParams& p, int Q, double* S, const double2* xy, int ks,
                                       int e, int warp, int lane) {
    switch (Q) {
        case 3: return fill_system<LDS, NRHS, P, 3, NW, CAREFUL>(p, S, xy, ks, e, warp, lane);
        case 5: return fill_system<LDS, NRHS, P, 5, NW, CAREFUL>(p, S, xy, ks, e, warp, lane);
        case 7: return fill_system<LDS, NRHS, P, 7, NW, CAREFUL>(p, S, xy, ks, e, warp, lane);
        default: return fill_system<LDS, NRHS, P, 9, NW, CAREFUL>(p, S, xy, ks, e, warp, lane);
    }
}

template <int LDS, int NRHS, int NW, bool CAREFUL, class Sh>
__device__ __forceinline__ bool fill_shape(const AsmParams& p, Sh sh, double* S, const double2* xy,
                                           int ks, int e, int warp, int lane) {
    if constexpr (Sh::P >= 0) {
        return fill_system<LDS, NRHS, Sh::P, Sh::Q, NW, CAREFUL>(p, S, xy, ks, e, warp, lane);
    } else {
        switch (sh.p) {
            case 1: return fill_q<LDS, NRHS, 1, NW, CAREFUL>(p, sh.q, S, xy, ks, e, warp, lane);
            case 2: return fill_q<LDS, NRHS, 2, NW, CAREFUL>(p, sh.q, S, xy, ks, e, warp, lane);
            case 3: return fill_q<LDS, NRHS, 3, NW, CAREFUL>(p, sh.q, S, xy, ks, e, warp, lane);
            default: return fill_q<LDS, NRHS, 4, NW, CAREFUL>(p, sh.q, S, xy, ks, e, warp, lane);
        }
    }
}

// Stencil s: its row in ja and the value arrays (in CSR form its first entry), its
// size, its centre.
struct Item {
    int s, row, ks;
    double x0, y0;
};
__device__ __forceinline__ Item item_of(const AsmParams& p, int s) {
    Item it{s, s - p.row_base, p.k, __ldg(p.x + s), __ldg(p.y + s)};
    if (p.ia) {
        it.row = __ldg(p.ia + s);
        it.ks = __ldg(p.ia + s + 1) - it.row;
    }
    return it;
}
// Its first entry there, in 64 bits: a fixed-width batch may hold more than 2^31. Formed
// where it is used: carried along it takes registers (600,000 stencils, k = 64: 37.0 ms,
// this way 36.2, in 32 bits 35.7).
__device__ __forceinline__ long long offset_of(const AsmParams& p, const Item& it) {
    return static_cast<long long>(static_cast<unsigned long long>(static_cast<unsigned>(it.row)) *
                                  static_cast<unsigned>(p.stride));
}

// The careful path of one stencil, from its global data: everything the fast
// path leaves out (coincident nodes, zero pivots, extreme magnitudes). Cold.
template <class L, int NRHS, int NW, class Sh>
__device__ __noinline__ void assemble_careful(const AsmParams& p, Sh sh, int s, int row, int ks,
                                              char* base, int warp, int lane) {
    constexpr int LDS = L::LDS;
    double2* xy = reinterpret_cast<double2*>(base + L::off_xy);
    double* S = reinterpret_cast<double*>(base + L::off_s);
    uint8_t* lists = reinterpret_cast<uint8_t*>(base + L::off_list);
    uint8_t* piv = reinterpret_cast<uint8_t*>(base + L::off_piv);
    int* nia = reinterpret_cast<int*>(base + L::off_nia);
    const long long off = offset_of(p, Item{s, row, ks, 0.0, 0.0});
    const int np = sh.np(), n = np + ks;
    stencil_sync<NW>();
    int e = 0;
    if (NW == 1 || warp == 0) {
        e = gather_scale<L::KMAX, false, true>(p, off, ks, p.x[s], p.y[s], xy, lane);
        if (NW > 1 && lane == 0) nia[3] = e;
    }
    stencil_sync<NW>();
    if (NW > 1) e = nia[3];
    fill_shape<LDS, NRHS, NW, true>(p, sh, S, xy, ks, e, warp, lane);
    stencil_sync<NW>();
    if (NW == 1 || warp == 0) init_order(lists, piv, n, lane);
    __syncwarp();
    const int info = eliminate<L::NMAX, LDS, L::kWhole, NRHS, NW, true>(S, lists, piv, n, np, warp, lane);
    if (NW == 1 || warp == 0) {
        back_substitute<LDS, NRHS, true>(p, S, piv, n, np, off, e, info, lane);
        if (lane == 0 && p.info) p.info[s - p.row_base] = info;
    }
    stencil_sync<NW>();
}

// The neighbour coordinates of stencil nx and its centre, asynchronously, by
// one warp: the ja row is in nja (STAGED) or read here.
template <class L, bool STAGED>
__device__ __forceinline__ void fetch_nodes(const AsmParams& p, const Item& nx, char* base, int lane) {
    constexpr int KPL = (L::KMAX + 31) / 32;
    double2* xy = reinterpret_cast<double2*>(base + L::off_xy);
    const int* nja = reinterpret_cast<const int*>(base + L::off_nja);
    int nb[KPL];
    if (STAGED) {
        cp_async_wait_all();
        __syncwarp();
    }
#pragma unroll
    for (int t = 0; t < KPL; ++t) {
        const int j = lane + 32 * t;
        nb[t] = j >= nx.ks ? 0 : STAGED ? nja[j] : __ldg(p.ja + offset_of(p, nx) + j);
    }
    __syncwarp();  // the ja row shares xy's slot
#pragma unroll
    for (int t = 0; t < KPL; ++t) {
        const int j = lane + 32 * t;
        if (j < nx.ks) {
            cp_async8(&xy[j].x, p.x + nb[t]);
            cp_async8(&xy[j].y, p.y + nb[t]);
        }
    }
}

// One stencil by its NW warps: gather, fill, eliminate, back-substitute,
// scatter, in the working set at base (shared memory, or with !SHARED global:
// no fetching ahead). fetched: its raw neighbour coordinates are on their way
// into xy (fetch_nodes). nx, if its s >= 0, is fetched for the
// next call by the stencil's last warp: the ja row while s is eliminated, the
// coordinates once the lists of unused rows, whose slot they share, are no
// longer read.
template <class L, int NRHS, int NW, bool SHARED, class Sh>
__device__ __forceinline__ void assemble(const AsmParams& p, Sh sh, const Item& it, const Item& nx,
                                         bool fetched, char* base, int warp, int lane) {
    constexpr int LDS = L::LDS;
    double2* xy = reinterpret_cast<double2*>(base + L::off_xy);
    double* S = reinterpret_cast<double*>(base + L::off_s);
    uint8_t* lists = reinterpret_cast<uint8_t*>(base + L::off_list);
    uint8_t* piv = reinterpret_cast<uint8_t*>(base + L::off_piv);
    int* nja = reinterpret_cast<int*>(base + L::off_nja);
    int* nia = reinterpret_cast<int*>(base + L::off_nia);
    const bool lead = NW == 1 || warp == 0, fetcher = NW == 1 || warp == NW - 1;
    if constexpr (SHARED) {
        if (!fetched && fetcher) fetch_nodes<L, false>(p, it, base, lane);
        cp_async_wait_all();
    }
    stencil_sync<NW>();
    const int ks = it.ks, np = sh.np(), n = np + ks;
    int e = 0;
    if (lead) {
        e = gather_scale<L::KMAX, SHARED, false>(p, offset_of(p, it), ks, it.x0, it.y0, xy, lane);
        if (NW > 1 && lane == 0) {
            nia[2] = 0;
            nia[3] = e;
        }
    }
    stencil_sync<NW>();
    if (NW > 1) e = nia[3];
    bool bad = fill_shape<LDS, NRHS, NW, false>(p, sh, S, xy, ks, e, warp, lane);
    bad = bad || e < -kMaxExp || e > kMaxExp;
    stencil_sync<NW>();
    if (lead) init_order(lists, piv, n, lane);
    if (SHARED && fetcher && nx.s >= 0)
        for (int j = lane; j < nx.ks; j += 32) cp_async4(nja + j, p.ja + offset_of(p, nx) + j);
    if (NW > 1 && bad) nia[2] = 1;
    __syncwarp();
    const int out = eliminate<L::NMAX, LDS, L::kWhole, NRHS, NW, false>(S, lists, piv, n, np, warp, lane);
    if constexpr (NW == 1) {
        bad = __any_sync(0xffffffffu, bad || out != 0);
    } else {
        if (lead && out) nia[2] = 1;
        stencil_sync<NW>();
        bad = nia[2] != 0;
    }
    if (bad) {
        if constexpr (SHARED) cp_async_wait_all();
        assemble_careful<L, NRHS, NW>(p, sh, it.s, it.row, ks, base, warp, lane);
        if (SHARED && fetcher && nx.s >= 0) fetch_nodes<L, false>(p, nx, base, lane);
        return;
    }
    if (SHARED && fetcher && nx.s >= 0) fetch_nodes<L, true>(p, nx, base, lane);
    if (lead) {
        back_substitute<LDS, NRHS, false>(p, S, piv, n, np, offset_of(p, it), e, 0, lane);
        if (lane == 0 && p.info) p.info[it.s - p.row_base] = 0;
    }
}

// Fixed-shape kernel: GPB stencils in flight a CTA (one when NW > 1), a
// persistent grid in a static stride over the stencils. The CTA's stencils
// advance together (a barrier each): its warps then run the same code at about
// the same time, which the instruction cache needs (a stencil runs through
// about 35 KB of straight-line code once).
template <int NMAX, int NRHS, int P, int Q, int NW, int GPB, int MINB>
__global__ void __launch_bounds__(32 * NW * GPB, MINB)
    dm_kernel(const __grid_constant__ AsmParams p) {
    static_assert(NW == 1 || GPB == 1, "a stencil of several warps has its CTA alone");
    using L = Layout<NMAX, NRHS, NMAX - npoly(P)>;
    extern __shared__ __align__(16) char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = NW == 1 ? warp : 0, wis = NW == 1 ? 0 : warp;
    char* smem = smem_raw + grp * L::bytes;
    const int n = p.nitems_dev ? *p.nitems_dev : p.nitems;
    const int* list = (p.list && p.list_off_dev) ? p.list + *p.list_off_dev : p.list;
    const int stride = gridDim.x * GPB;
    // past the end a warp repeats the last stencil (it writes the same weights)
    auto item = [&](int i0) {
        const int i = min(i0 + grp, n - 1);
        return item_of(p, list ? list[i] : p.item_base + i);
    };
    bool fetched = false;
    Item it{};
    int i0 = blockIdx.x * GPB;
    if (i0 < n) it = item(i0);
    for (; i0 < n; i0 += stride) {
        Item nx{-1, 0, 0, 0.0, 0.0};
        if (i0 + stride < n) nx = item(i0 + stride);
        if (GPB > 1) __syncthreads();
        assemble<L, NRHS, NW, true>(p, Shape<P, Q>{}, it, nx, fetched, smem, wis, lane);
        it = nx;
        fetched = true;
    }
}

// ---- one persistent launch for an uneven batch ------------------------------
//
// Ragged stencils in CSR form, each with its own size k_s = ia[s+1] - ia[s],
// degree P_s (degree[s], or P0 for all) and PHS exponent Q_s = phs, or
// 2 P_s - 1 when phs = 0: the reference's one-grid-over-all-stencils launch
// (src/rbf_operators.h:197-200,340) for stencils of any mix of shapes. A CTA
// claims its GPB next stencils from one device work counter, one round ahead.
// A system of up to NS unknowns is solved in the warp's shared-memory slot; a
// larger one (up to NG) in the warp's region of a global scratch buffer, which
// stays in L2. Supported: P_s in 1..4 and Q_s in {3, 5, 7, 9}; a stencil
// outside that (or above NG unknowns, or with no neighbour) sets *err and is
// skipped.
template <int NS, int NG, int NRHS>
struct CsrCfg {
    using SmemL = Layout<NS, NRHS, NS>;
    using GlobL = Layout<NG, NRHS, NG>;
    static constexpr size_t gbytes = (static_cast<size_t>(GlobL::bytes) + 255) & ~size_t(255);
};

template <int NS, int NG, int NRHS, int GPB, int MINB>
__global__ void __launch_bounds__(32 * GPB, MINB)
    dm_csr_kernel(const __grid_constant__ AsmParams p, const int8_t* degree, int P0, int phs,
                  char* gscratch, int* err) {
    using C = CsrCfg<NS, NG, NRHS>;
    extern __shared__ __align__(16) char smem_raw[];
    __shared__ int claim;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    char* slot = smem_raw + warp * C::SmemL::bytes;
    char* gslot = gscratch + (static_cast<size_t>(blockIdx.x) * GPB + warp) * C::gbytes;
    const int n = p.nitems;
    using Sh = Shape<-1, 0>;
    // a warp's stencil of a round, its shape, and where it runs (0: nowhere, 1:
    // shared memory, 2: global scratch)
    struct Work {
        Item it;
        Shape<-1, 0> sh;
        int where;
    };
    auto look = [&](int i0) {
        Work w{{-1, 0, 0, 0.0, 0.0}, {0, 0}, 0};
        const int i = i0 + warp;
        if (i >= n) return w;
        w.it = item_of(p, p.list ? __ldg(p.list + i) : p.item_base + i);
        w.sh.p = degree ? degree[w.it.s] : P0;
        w.sh.q = phs ? phs : 2 * w.sh.p - 1;
        const int P = w.sh.p, q = w.sh.q, m = w.it.ks + npoly(P);
        if (P >= 1 && P <= 4 && (q == 3 || q == 5 || q == 7 || q == 9) && w.it.ks >= 1 && m <= NG)
            w.where = m <= NS ? 1 : 2;
        else if (lane == 0)
            atomicExch(err, 1);
        return w;
    };
    auto next_round = [&]() {
        __syncthreads();
        if (threadIdx.x == 0) claim = atomicAdd(p.work, GPB);
        __syncthreads();
        return claim;
    };
    int i0 = next_round();
    Work cur = look(i0);
    bool fetched = false;
    while (i0 < n) {
        i0 = next_round();
        const Work next = look(i0);
        Item nx = next.it;
        if (next.where != 1 || cur.where != 1) nx.s = -1;
        if (cur.where == 1)
            assemble<typename C::SmemL, NRHS, 1, true>(p, cur.sh, cur.it, nx, fetched, slot, 0, lane);
        else if (cur.where == 2)
            assemble<typename C::GlobL, NRHS, 1, false>(p, cur.sh, cur.it, nx, false, gslot, 0, lane);
        fetched = nx.s >= 0;
        cur = next;
    }
}

}  // namespace dm
}  // namespace rbfb
