// knn.cu -- k-nearest-neighbour stencils on a uniform cell grid (sm_100a).
//
// Replaces the reference's tree searches: NodeSet::stencils(k) over a
// nanoflann k-d tree in the open plane (src/rbf_nodeset.h:155-181) and
// KdTree::knn_stencils(k) over SciPy's ckdtree in a periodic box
// (src/rbf_spatial.cpp:193-260). A tree walk is pointer chasing; on the GPU
// the nodes are binned instead:
//
//   1. bounding box (open plane, device reduction) or the box [0,L)^2;
//   2. cell of every node on a cx x cy grid, counting sort by cell:
//      start[] and the nodes' coordinates and indices in cell order;
//   3. the stencils of the nodes themselves: one warp per cell
//      (cell_query_kernel). The nodes of the (2R+1)^2 cells around it are
//      copied to shared memory once for all of the cell's nodes. For each of
//      them, those closer than a radius that lies inside the block are kept;
//      when at least k are, the k nearest are among them. They are ranked by a
//      counting sort on the squared distance (uniform over the circle, so the
//      buckets hold about half an entry) and exact comparisons inside a
//      bucket. Queries it cannot complete (leftover_kernel) and arbitrary
//      query points (query_kernel) take the general search: one warp per query,
//      a block that grows until k are found, ranking by comparison.
//
// Distances use the reference's arithmetic exactly: dx*dx + dy*dy of the
// plain differences, each operation rounded (nanoflann L2_Simple_Adaptor,
// nanoflann.hpp:690-699), and in a periodic box of ckdtree's wrapped
// differences (wrap_distance, ckdtree/src/distance.h:262-272) with both
// the nodes and the queries folded into [0, L) first (rbf_spatial.h:39-48,
// ckdtree wrap_position). Neighbours are ordered by (squared distance,
// index), which equals the reference's order wherever no two candidates tie.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <type_traits>

#include "asm_math.cuh"
#include "runtime.h"

namespace rbfb {
namespace knn {

constexpr int kPerCell = 2;   // target nodes per cell for arbitrary query points
constexpr int kCap = 256;     // candidate buffer per warp (entries)
constexpr int kWarps = 4;     // warps per CTA in the query kernel
constexpr int kMaxK = 128;
// Capacities of a warp's lists for k neighbours: a block's candidates, and the
// kept ones (k + 1 + 1.9 sqrt(k + 1) on average).
__host__ __device__ constexpr int cand_cap_of(int k) { return (static_cast<int>(6.5 * (k + 1)) + 31) / 32 * 32; }
__host__ __device__ constexpr int keep_cap_of(int k) { return (static_cast<int>(2.2 * (k + 1)) + 31) / 32 * 32; }
constexpr int kMaxCand = cand_cap_of(kMaxK), kMaxKeep = keep_cap_of(kMaxK);

struct Grid {
    double x0, y0;     // origin of the cell grid
    double hx, hy;     // cell sides
    int cx, cy;        // cells per axis
    double Lx, Ly;     // periods (> 0) or 0
    double per;        // mean nodes per cell
};

// What one search clears before it starts, followed by the cell counts.
struct Head {
    unsigned long long bbox[4];  // ordered images: max of -x, x, -y, y
    unsigned int ticket;         // blocks of the bounding-box kernel that are done
    int status;                  // 1: a query could not be completed
    int left;                    // queries that the search by cells left over
    int pad[5];
};
static_assert(sizeof(Head) == 64, "the counts after it stay aligned");

// detail::fold of the reference (src/rbf_spatial.h:39-48), rounded per op.
__device__ __forceinline__ double fold(double x, double L) {
    if (!(L > 0.0)) return x;
    x = dsub(x, dmul(L, floor(ddiv(x, L))));
    while (x >= L) x = dsub(x, L);
    while (x < 0.0) x = dadd(x, L);
    return x;
}

// ckdtree wrap_distance.
__device__ __forceinline__ double wrap_d(double d, double L) {
    if (!(L > 0.0)) return d;
    const double hb = 0.5 * L;
    if (d < -hb) return dadd(L, d);
    if (d > hb) return dsub(d, L);
    return d;
}

__device__ __forceinline__ double sqdist(double qx, double qy, double px, double py, double Lx,
                                         double Ly) {
    const double dx = wrap_d(dsub(qx, px), Lx);
    const double dy = wrap_d(dsub(qy, py), Ly);
    return dadd(dmul(dx, dx), dmul(dy, dy));
}

__device__ __forceinline__ int cell_coord(double v, double o, double h, int c) {
    int i = static_cast<int>(floor((v - o) / h));
    return i < 0 ? 0 : (i >= c ? c - 1 : i);
}

// ---- 1. bounding box ---------------------------------------------------------
// Order-preserving image of a double in the unsigned integers, above 0.
__device__ __forceinline__ unsigned long long key_of(double v) {
    const long long b = __double_as_longlong(v);
    return b >= 0 ? (unsigned long long)b | 0x8000000000000000ull : ~(unsigned long long)b;
}
__device__ __forceinline__ double unkey(unsigned long long k) {
    return (k & 0x8000000000000000ull) ? __longlong_as_double((long long)(k & 0x7fffffffffffffffull))
                                       : __longlong_as_double((long long)~k);
}

// The open-plane grid of a bounding box: at most `cells` cells, about square; a
// box without width (or height) is cut along its other side only.
__device__ inline Grid open_grid(double xmin, double xmax, double ymin, double ymax, int cells,
                                 double per) {
    double wx = xmax - xmin, wy = ymax - ymin;
    Grid g;
    if (!(wx > 0) || !(wy > 0)) {
        g.cx = wx > 0 ? cells : 1;
        g.cy = wy > 0 ? cells : 1;
    } else {
        const double a = wx / wy > 1e-18 && wx / wy < 1e18 ? sqrt(wx / wy) : 1.0;
        g.cx = min(cells, max(1, (int)fmin(sqrt((double)cells) * a, 2e9)));
        g.cy = max(1, cells / g.cx);
    }
    if (!(wx > 0)) wx = 1.0;
    if (!(wy > 0)) wy = 1.0;
    g.x0 = xmin;
    g.y0 = ymin;
    g.hx = wx / g.cx * (1.0 + 1e-12);
    g.hy = wy / g.cy * (1.0 + 1e-12);
    g.Lx = 0.0;
    g.Ly = 0.0;
    g.per = per;
    return g;
}

// One set of atomics a block (a warp each took 29 us at 1M nodes, against 6);
// the block that finishes last forms the grid.
__global__ void __launch_bounds__(256) bbox_kernel(const double* x, const double* y, int n, Head* head,
                                                   int cells, double per, Grid* gp) {
    double m[4] = {-1e308, -1e308, -1e308, -1e308};  // max of -x, x, -y, y
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double px = x[i], py = y[i];
        m[0] = fmax(m[0], -px);
        m[1] = fmax(m[1], px);
        m[2] = fmax(m[2], -py);
        m[3] = fmax(m[3], py);
    }
    __shared__ double sh[8][4];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        for (int o = 16; o > 0; o >>= 1) m[j] = fmax(m[j], __shfl_xor_sync(0xffffffffu, m[j], o));
        if (lane == 0) sh[w][j] = m[j];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double v = sh[0][threadIdx.x];
        for (int i = 1; i < 8; ++i) v = fmax(v, sh[i][threadIdx.x]);
        atomicMax(head->bbox + threadIdx.x, key_of(v));
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&head->ticket, 1u) == gridDim.x - 1) {
        __threadfence();
        double v[4];
        for (int j = 0; j < 4; ++j) v[j] = unkey(__ldcg(head->bbox + j));
        *gp = open_grid(-v[0], v[1], -v[2], v[3], cells, per);
    }
}

// ---- 2. binning ----------------------------------------------------------------
// Cell of every node and its rank among the nodes counted there so far. The
// grid comes from device memory, or (gp == nullptr) with the launch.
__global__ void cell_count_kernel(const double* x, const double* y, int n, const Grid* gp, Grid gv,
                                  int* cell_of, int* rank, int* count) {
    const Grid g = gp ? *gp : gv;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double px = fold(x[i], g.Lx), py = fold(y[i], g.Ly);
        const int c = cell_coord(py, g.y0, g.hy, g.cy) * g.cx + cell_coord(px, g.x0, g.hx, g.cx);
        cell_of[i] = c;
        rank[i] = atomicAdd(count + c, 1);
    }
}

// Exclusive scan in two launches: per block, then each block adds the totals of
// the blocks before it.
constexpr int kScanBlock = 1024;
__device__ __forceinline__ int block_sum_1024(int v, int* warp_sums) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = warp_sums[threadIdx.x & 31];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}
__global__ void __launch_bounds__(kScanBlock) scan_block_kernel(const int* in, int* out, int n,
                                                                int* block_sums) {
    __shared__ int warp_sums[32];
    const int i = blockIdx.x * kScanBlock + threadIdx.x;
    int v = i < n ? in[i] : 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int s = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += t;
    }
    if (lane == 31) warp_sums[w] = s;
    __syncthreads();
    if (w == 0) {
        int ws = warp_sums[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, ws, o);
            if (lane >= o) ws += t;
        }
        warp_sums[lane] = ws;
    }
    __syncthreads();
    const int excl = s - v + (w > 0 ? warp_sums[w - 1] : 0);
    if (i < n) out[i] = excl;
    if (threadIdx.x == kScanBlock - 1) block_sums[blockIdx.x] = excl + v;
}
__global__ void __launch_bounds__(kScanBlock) scan_add_kernel(int* out, int n, const int* sums) {
    __shared__ int warp_sums[32];
    int part = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += kScanBlock) part += sums[b];
    const int before = block_sum_1024(part, warp_sums);
    const int i = blockIdx.x * kScanBlock + threadIdx.x;
    if (i < n) out[i] += before;
}

__global__ void scatter_kernel(const double* x, const double* y, int n, const Grid* gp, Grid gv,
                               const int* cell_of, const int* rank, const int* start, int* sidx,
                               double2* sxy) {
    const double Lx = gp ? gp->Lx : gv.Lx, Ly = gp ? gp->Ly : gv.Ly;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int pos = start[cell_of[i]] + rank[i];
        sidx[pos] = i;
        sxy[pos] = make_double2(fold(x[i], Lx), fold(y[i], Ly));
    }
}

// All of the binning in one block, for small node sets, whose search would
// otherwise be mostly launches: 4,761 nodes in the open plane, k = 21, binning
// and query 41 us in seven launches, 28 in two (with the smaller cells of per_cell).
// One block is bound by its chain of barriers and memory latencies, ~12 us, which
// grows with n: at 8,192 nodes 33 us against 41 (periodic 35 against 38), and
// more nodes a thread would not fit its registers.
// Each thread keeps its nodes in registers; the cell counts and their scan live
// in shared memory.
constexpr int kSmallNodes = 8192, kSmallPer = kSmallNodes / 1024;
constexpr int kSmallCells = kSmallNodes / kPerCell, kSmallCellsPer = kSmallCells / 1024;
__global__ void __launch_bounds__(1024) small_bins_kernel(const double* x, const double* y, int n, int cells,
                                                          double per, Grid gv, Grid* gp, Head* head,
                                                          int* start, int* sidx,
                                                          double2* sxy) {
    __shared__ int count[kSmallCells];
    __shared__ double sh[32][4];
    __shared__ int warp_sums[32];
    __shared__ Grid g;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    double px[kSmallPer], py[kSmallPer];
#pragma unroll
    for (int j = 0; j < kSmallPer; ++j) {
        const int i = tid + 1024 * j;
        px[j] = i < n ? x[i] : 0.0;
        py[j] = i < n ? y[i] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kSmallCellsPer; ++j) count[tid + 1024 * j] = 0;
    if (gp) {
        double m[4] = {-1e308, -1e308, -1e308, -1e308};
#pragma unroll
        for (int j = 0; j < kSmallPer; ++j)
            if (tid + 1024 * j < n) {
                m[0] = fmax(m[0], -px[j]);
                m[1] = fmax(m[1], px[j]);
                m[2] = fmax(m[2], -py[j]);
                m[3] = fmax(m[3], py[j]);
            }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            for (int o = 16; o > 0; o >>= 1) m[j] = fmax(m[j], __shfl_xor_sync(0xffffffffu, m[j], o));
            if (lane == 0) sh[w][j] = m[j];
        }
        __syncthreads();
        if (w == 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                m[j] = sh[lane][j];
                for (int o = 16; o > 0; o >>= 1)
                    m[j] = fmax(m[j], __shfl_xor_sync(0xffffffffu, m[j], o));
            }
            if (lane == 0) g = open_grid(-m[0], m[1], -m[2], m[3], cells, per);
        }
    } else if (tid == 0) {
        g = gv;
    }
    __syncthreads();
    if (tid == 0) {
        head->status = 0;
        head->left = 0;
        if (gp) *gp = g;
    }
    int cell[kSmallPer], rk[kSmallPer];
#pragma unroll
    for (int j = 0; j < kSmallPer; ++j) {
        if (tid + 1024 * j < n) {
            px[j] = fold(px[j], g.Lx);
            py[j] = fold(py[j], g.Ly);
            cell[j] = cell_coord(py[j], g.y0, g.hy, g.cy) * g.cx + cell_coord(px[j], g.x0, g.hx, g.cx);
            rk[j] = atomicAdd(count + cell[j], 1);
        }
    }
    __syncthreads();
    // exclusive scan, kSmallCellsPer consecutive cells a thread
    int v[kSmallCellsPer], own = 0;
#pragma unroll
    for (int j = 0; j < kSmallCellsPer; ++j) {
        v[j] = count[tid * kSmallCellsPer + j];
        own += v[j];
    }
    int incl = own;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[w] = incl;
    __syncthreads();
    int before = lane < w ? warp_sums[lane] : 0;
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    int at = before + incl - own;
#pragma unroll
    for (int j = 0; j < kSmallCellsPer; ++j) {
        const int c = tid * kSmallCellsPer + j;
        count[c] = at;
        if (c <= cells) start[c] = at;
        at += v[j];
    }
    if (tid == 1023 && cells == kSmallCells) start[cells] = at;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSmallPer; ++j) {
        const int i = tid + 1024 * j;
        if (i < n) {
            const int pos = count[cell[j]] + rk[j];
            sidx[pos] = i;
            sxy[pos] = make_double2(px[j], py[j]);
        }
    }
}

// ---- 3. queries --------------------------------------------------------------------
struct QueryArgs {
    const Grid* g;     // device grid, or nullptr: gv
    Grid gv;
    const int* start;  // cells + 1 entries
    const int* sidx;
    const double2* sxy;
    int nq;
    const double* qx;  // query coordinates (query_kernel)
    const double* qy;
    int k;
    int* ja;
    int* status;  // set to 1 when a query could not be completed
    // cell_query_kernel: capacities of a warp's shared-memory lists; the nodes
    // (in cell order) that it leaves to leftover_kernel and their number
    int cand_cap, keep_cap;
    int split;  // warps a cell
    int most;   // queries a warp takes of its cell, the rest is left over
    int* list;
    int* left;
};

__device__ __forceinline__ bool key_less(unsigned long long da, int ia, unsigned long long db,
                                         int ib) {
    return da < db || (da == db && ia < ib);
}

// The general search: the k nearest nodes of (qx, qy), query number q, by one
// warp with kCap entries of scratch (d, id). It starts with the block of R rings
// of cells around the query's cell, and there with the radius (squared) est2, which
// only has to be a good guess: when fewer than k nodes lie inside, a wider one
// follows, up to the block's own bound, then a larger block.
__device__ __forceinline__ void search_one(const QueryArgs& a, const Grid& g, double qx, double qy,
                                           int q, int R, double est2, unsigned long long* d, int* id,
                                           int lane) {
    const int k = a.k;
    const int ccx = cell_coord(qx, g.x0, g.hx, g.cx);
    const int ccy = cell_coord(qy, g.y0, g.hy, g.cy);
    bool done = false;
    double reach = est2;
    for (int attempt = 0; attempt < 64 && !done; ++attempt) {
        // periodic axes: never more than one period (no cell twice); open
        // axes: up to the whole grid (the clamp below keeps it in range)
        const int Rx = g.Lx > 0 ? min(R, (g.cx - 1) / 2 + 1) : min(R, g.cx);
        const int Ry = g.Ly > 0 ? min(R, (g.cy - 1) / 2 + 1) : min(R, g.cy);
        const bool fullx = g.Lx > 0 ? (2 * Rx + 1 >= g.cx) : false;
        const bool fully = g.Ly > 0 ? (2 * Ry + 1 >= g.cy) : false;
        // x/y cell ranges (periodic: wrapped, never more than the grid)
        int xlo = ccx - Rx, xhi = ccx + Rx, ylo = ccy - Ry, yhi = ccy + Ry;
        if (g.Lx > 0) {
            if (fullx) { xlo = 0; xhi = g.cx - 1; }
        } else {
            xlo = max(xlo, 0);
            xhi = min(xhi, g.cx - 1);
        }
        if (g.Ly > 0) {
            if (fully) { ylo = 0; yhi = g.cy - 1; }
        } else {
            ylo = max(ylo, 0);
            yhi = min(yhi, g.cy - 1);
        }
        // distance from the query to the edge of the searched block
        double bx = 1e300, by = 1e300;
        if (g.Lx > 0) {
            if (!fullx) bx = fmin(qx - (ccx - Rx) * g.hx, (ccx + Rx + 1) * g.hx - qx);
        } else {
            if (ccx - Rx > 0) bx = fmin(bx, qx - (g.x0 + (ccx - Rx) * g.hx));
            if (ccx + Rx < g.cx - 1) bx = fmin(bx, g.x0 + (ccx + Rx + 1) * g.hx - qx);
        }
        if (g.Ly > 0) {
            if (!fully) by = fmin(qy - (ccy - Ry) * g.hy, (ccy + Ry + 1) * g.hy - qy);
        } else {
            if (ccy - Ry > 0) by = fmin(by, qy - (g.y0 + (ccy - Ry) * g.hy));
            if (ccy + Ry < g.cy - 1) by = fmin(by, g.y0 + (ccy + Ry + 1) * g.hy - qy);
        }
        double bound = fmin(bx, by);
        bound = bound * (1.0 - 1e-9) - 1e-15 * fmax(fabs(qx), fabs(qy));
        // Only candidates inside a circle of radius at most `bound`
        // (inscribed in the searched block) are kept: when at least k of
        // them are found, the k nearest nodes are among them, since every
        // node outside is farther than all of these; otherwise the radius
        // widens to the bound, then the block grows. (A block that covers
        // the whole domain keeps everything.)
        const double bound2 = bound >= 1e299 ? INFINITY : (bound > 0.0 ? bound * bound : 0.0);
        double keep2 = fmin(bound2, reach);
        // gather candidates chunk by chunk; the current best k stay at the front.
        // The block is a list of runs of consecutive cells (one per row, two
        // where a periodic row wraps). A batch of up to 32 runs is laid out
        // flat: lane t loads run t's bounds (all loads in flight at once),
        // a warp scan gives each run its offset, and the flat candidate
        // list is walked 32 at a time, each lane finding its run by a
        // shuffle binary search. The candidate set and its order are those
        // of a row-by-row walk.
        int have = 0;  // entries in the buffer (best-so-far first)
        int total = 0;
        const int nrows = yhi - ylo + 1;
        const int nruns = 2 * nrows;
        for (int rb = 0; rb < nruns; rb += 32) {
            int rbeg = 0, rlen = 0;  // this lane's run: first candidate, length
            {
                const int run = rb + lane;
                if (run < nruns) {
                    const int rr = run >> 1, part = run & 1;
                    int cyy = ylo + rr;
                    if (g.Ly > 0) cyy = ((cyy % g.cy) + g.cy) % g.cy;
                    int c0 = 0, c1 = -1;  // empty unless set below
                    if (g.Lx > 0 && !fullx) {
                        const int a0 = xlo, a1 = xhi;
                        if (a0 < 0) {
                            if (part == 0) { c0 = a0 + g.cx; c1 = g.cx - 1; } else { c0 = 0; c1 = a1; }
                        } else if (a1 >= g.cx) {
                            if (part == 0) { c0 = a0; c1 = g.cx - 1; } else { c0 = 0; c1 = a1 - g.cx; }
                        } else if (part == 0) {
                            c0 = a0; c1 = a1;
                        }
                    } else if (part == 0) {
                        c0 = xlo; c1 = xhi;
                    }
                    if (c1 >= c0) {
                        rbeg = a.start[cyy * g.cx + c0];
                        rlen = a.start[cyy * g.cx + c1 + 1] - rbeg;
                    }
                }
            }
            int incl = rlen;  // inclusive scan of the run lengths
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const int excl = incl - rlen;
            const int btotal = __shfl_sync(0xffffffffu, incl, 31);
            for (int base = 0; base < btotal; base += 32) {
                const int f = base + lane;
                // the run holding flat index f: the number of runs ending at or
                // before it (incl is non-decreasing over the lanes)
                int r = 0;
#pragma unroll
                for (int sh = 16; sh > 0; sh >>= 1) {
                    const int v = __shfl_sync(0xffffffffu, incl, r + sh - 1);
                    if (v <= f) r += sh;
                }
                const int jb = __shfl_sync(0xffffffffu, rbeg, r);
                const int jx = __shfl_sync(0xffffffffu, excl, r);
                const int j = jb + (f - jx);
                bool ok = f < btotal;
                unsigned long long dk = 0;
                int ik = 0;
                if (ok) {
                    const double2 c = a.sxy[j];
                    const double d2 = sqdist(qx, qy, c.x, c.y, g.Lx, g.Ly);
                    ok = d2 < keep2;
                    dk = (unsigned long long)__double_as_longlong(d2);
                    ik = a.sidx[j];
                }
                const unsigned bal = __ballot_sync(0xffffffffu, ok);
                const int cnt = __popc(bal);
                if (have + cnt > kCap) {
                    // merge: keep the k best of the buffer
                    __syncwarp();
                    int keepd[kCap / 32];
#pragma unroll
                    for (int u = 0; u < kCap / 32; ++u) {
                        const int c = lane + 32 * u;
                        int rank = kCap;
                        if (c < have) {
                            rank = 0;
                            for (int v = 0; v < have; ++v)
                                rank += key_less(d[v], id[v], d[c], id[c]);
                        }
                        keepd[u] = rank;
                    }
                    unsigned long long td[kCap / 32];
                    int ti[kCap / 32];
#pragma unroll
                    for (int u = 0; u < kCap / 32; ++u) {
                        const int c = lane + 32 * u;
                        td[u] = c < have ? d[c] : 0;
                        ti[u] = c < have ? id[c] : 0;
                    }
                    __syncwarp();
#pragma unroll
                    for (int u = 0; u < kCap / 32; ++u)
                        if (keepd[u] < k) {
                            d[keepd[u]] = td[u];
                            id[keepd[u]] = ti[u];
                        }
                    __syncwarp();
                    // nothing farther than the k-th found so far is needed
                    if (have >= k) keep2 = __longlong_as_double((long long)(d[k - 1] + 1));
                    have = min(have, k);
                }
                const int pos = have + __popc(bal & ((1u << lane) - 1u));
                if (ok) {
                    d[pos] = dk;
                    id[pos] = ik;
                }
                have += cnt;
                total += cnt;
                __syncwarp();
            }
        }
        if (total < k) {
            if (reach < bound2) {  // same block, a wider radius, then the full bound
                reach = reach == est2 && est2 > 0.0 ? 4.0 * est2 : INFINITY;
                continue;
            }
            R += max(1, R / 2);
            continue;
        }
        // rank the buffer, write the k best: one pass over the buffer, each
        // (broadcast) entry compared with all of the lane's own entries
        int myrank[kCap / 32];
        unsigned long long mine_d[kCap / 32];
        int mine_i[kCap / 32];
        const int nslot = (have + 31) / 32;  // warp-uniform
#pragma unroll
        for (int u = 0; u < kCap / 32; ++u) {
            const int c = lane + 32 * u;
            myrank[u] = 0;
            mine_d[u] = (u < nslot && c < have) ? d[c] : 0ull;
            mine_i[u] = (u < nslot && c < have) ? id[c] : 0;
        }
        // the slot count is warp-uniform: one loop body per count, so only
        // the live slots are compared
        auto rank_with = [&](auto ns) {
            constexpr int NS = decltype(ns)::value;
            for (int v = 0; v < have; ++v) {
                const unsigned long long dv = d[v];
                const int iv = id[v];
#pragma unroll
                for (int u = 0; u < NS; ++u) myrank[u] += key_less(dv, iv, mine_d[u], mine_i[u]);
            }
        };
        switch (nslot) {
            case 1: rank_with(std::integral_constant<int, 1>{}); break;
            case 2: rank_with(std::integral_constant<int, 2>{}); break;
            case 3: rank_with(std::integral_constant<int, 3>{}); break;
            case 4: rank_with(std::integral_constant<int, 4>{}); break;
            case 5: rank_with(std::integral_constant<int, 5>{}); break;
            case 6: rank_with(std::integral_constant<int, 6>{}); break;
            case 7: rank_with(std::integral_constant<int, 7>{}); break;
            default: rank_with(std::integral_constant<int, kCap / 32>{}); break;
        }
#pragma unroll
        for (int u = 0; u < kCap / 32; ++u)
            if (lane + 32 * u >= have) myrank[u] = kCap;
        // k-th distance: the entry of rank k-1, broadcast by two max-reductions
        unsigned long long dkth = 0;
#pragma unroll
        for (int u = 0; u < kCap / 32; ++u)
            if (myrank[u] == k - 1) dkth = d[lane + 32 * u];
        const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(dkth >> 32));
        const unsigned lo =
            __reduce_max_sync(0xffffffffu, ((unsigned)(dkth >> 32) == hi) ? (unsigned)dkth : 0u);
        const unsigned long long dk_all = ((unsigned long long)hi << 32) | lo;
        const double dk2 = __longlong_as_double((long long)dk_all);
        if (dk2 < bound * bound || (bound >= 1e299)) {
#pragma unroll
            for (int u = 0; u < kCap / 32; ++u)
                if (myrank[u] < k) a.ja[(size_t)q * k + myrank[u]] = id[lane + 32 * u];
            done = true;
        } else {
            R += max(1, R / 2);
        }
        __syncwarp();
    }
    if (!done && lane == 0) atomicExch(a.status, 1);
}

// Where the general search starts at a density of `per` nodes a cell: the rings of
// cells around the query's, and the radius (squared) at which k + 1 nodes are
// expected, with a 30 % margin.
__device__ __forceinline__ int rings_at(int k, double per) {
    return max(1, (int)ceil(0.5 * (sqrt((k + 1.0) / per * 1.27) - 1.0)) + 1);
}
__device__ __forceinline__ double radius2_at(int k, const Grid& g, double per) {
    return 1.69 * (k + 1) * g.hx * g.hy / (3.141592653589793 * per);
}

// Arbitrary query points, one warp each. Bounded to 8 CTAs (32 warps) per SM:
// 64 registers and a few spilled bytes instead of 96 registers and about 20
// warps; the search is issue-bound, and the extra warps fill the issue slots
// (2.75 -> 2.60 ms for 1M queries, k = 35).
__global__ void __launch_bounds__(kWarps * 32, 8) query_kernel(QueryArgs a) {
    __shared__ unsigned long long sd[kWarps][kCap];
    __shared__ int si[kWarps][kCap];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Grid g = a.g ? *a.g : a.gv;
    const int R = rings_at(a.k, g.per);
    const double est2 = radius2_at(a.k, g, g.per);
    for (int q = blockIdx.x * kWarps + w; q < a.nq; q += gridDim.x * kWarps)
        search_one(a, g, fold(a.qx[q], g.Lx), fold(a.qy[q], g.Ly), q, R, est2, sd[w], si[w], lane);
}

// The nodes that the search by cells left over, one warp each (the warp of
// their cell would take them one after another: 11,359 nodes of fourfold varying
// density, k = 61: 261 us, this way 81). Its cells are the large ones of the search by
// cells, so it starts from the density around each node, not from the mean (20,000 nodes,
// density falling a thousandfold, k = 13: 3.5 ms from the mean, 0.16). The launch costs a set that
// leaves none 2 us.
__global__ void __launch_bounds__(kWarps * 32, 8) leftover_kernel(QueryArgs a) {
    __shared__ unsigned long long sd[kWarps][kCap];
    __shared__ int si[kWarps][kCap];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int left = *a.left;
    if (left == 0) return;
    const Grid g = a.g ? *a.g : a.gv;
    for (int i = blockIdx.x * kWarps + w; i < left; i += gridDim.x * kWarps) {
        const int t = a.list[i];
        const double2 q = a.sxy[t];
        // the density around the node, from the 3 x 3 cells (none wrapped)
        const int row = cell_coord(q.y, g.y0, g.hy, g.cy) - 1 + lane;
        int count = 0, cells = 0;
        if (lane < 3 && row >= 0 && row < g.cy) {
            const int cx = cell_coord(q.x, g.x0, g.hx, g.cx);
            const int c0 = max(cx - 1, 0), c1 = min(cx + 1, g.cx - 1);
            count = a.start[row * g.cx + c1 + 1] - a.start[row * g.cx + c0];
            cells = c1 - c0 + 1;
        }
        count = __reduce_add_sync(0xffffffffu, count);
        cells = __reduce_add_sync(0xffffffffu, cells);
        const double per = static_cast<double>(count) / cells;
        const int R = min(rings_at(a.k, g.per),
                          max(1, (int)ceil(1.15 * sqrt((a.k + 1) / (3.141592653589793 * per)))));
        search_one(a, g, q.x, q.y, a.sidx[t], R, radius2_at(a.k, g, per), sd[w], si[w], lane);
    }
}

// ---- the nodes' own stencils, cell by cell ------------------------------------
constexpr int kBuckets = 128;  // of the counting sort: four a lane
// Entries of a bucket that a lane compares its own with one after another. Above,
// the distances are far from uniform over the circle (a tight cluster in a wide
// circle), and all entries are compared with all.
constexpr int kCrowded = 16;

// Shared memory of one warp: the block's candidates (coordinates, node
// indices), the kept ones (distance, node index) and the buckets.
__host__ __device__ constexpr size_t cell_smem(int cand_cap, int keep_cap) {
    return (static_cast<size_t>(cand_cap) * 20 + static_cast<size_t>(keep_cap) * 12 +
            (kBuckets + 4) * 4 + 15) & ~size_t(15);
}

// Writes the indices of the k first of the `have` entries (kd: bits of the squared distance,
// ki: node index) in the order (distance, index) to row: every entry compared
// with all, four entries a lane at a time.
__device__ __forceinline__ void rank_pairs(const unsigned long long* kd, const int* ki, int have, int k,
                                           int* row, int lane) {
    __syncwarp();
    for (int c0 = lane; c0 - lane < have; c0 += 128) {
        unsigned long long d[4];
        int id[4], rank[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int c = min(c0 + 32 * s, have - 1);
            d[s] = kd[c];
            id[s] = ki[c];
            rank[s] = 0;
        }
#pragma unroll 4
        for (int i = 0; i < have; ++i) {
            const unsigned long long o = kd[i];
            const int io = ki[i];
#pragma unroll
            for (int s = 0; s < 4; ++s) rank[s] += key_less(o, io, d[s], id[s]);
        }
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (c0 + 32 * s < have && rank[s] < k) row[rank[s]] = id[s];
    }
    __syncwarp();
}

// Ranks the `have` kept entries (kd: bits of the squared distance, ki: node
// index) by (distance, index) and writes the indices of the k first to row. scale * distance is about at most
// kBuckets.
template <int NS>
__device__ __forceinline__ void rank_kept(unsigned long long* kd, int* ki, int* hist, int have, int k,
                                          double scale, int* row, int lane) {
    unsigned long long d[NS];
    int id[NS], b[NS], at[NS];
    reinterpret_cast<int4*>(hist)[lane] = make_int4(0, 0, 0, 0);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const int c = lane + 32 * s;
        b[s] = -1;
        d[s] = 0;
        id[s] = 0;
        at[s] = 0;
        if (c < have) {
            d[s] = kd[c];
            id[s] = ki[c];
            b[s] = min(kBuckets - 1,
                       max(0, __double2int_rz(dmul(__longlong_as_double((long long)d[s]), scale))));
            at[s] = atomicAdd(hist + b[s], 1);
        }
    }
    __syncwarp();
    {
        const int4 h = reinterpret_cast<const int4*>(hist)[lane];
        if (__any_sync(0xffffffffu, max(max(h.x, h.y), max(h.z, h.w)) > kCrowded)) {
            rank_pairs(kd, ki, have, k, row, lane);
            return;
        }
        const int own = h.x + h.y + h.z + h.w;
        int incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int x = incl - own;
        reinterpret_cast<int4*>(hist)[lane] = make_int4(x, x + h.x, x + h.x + h.y, x + h.x + h.y + h.z);
        if (lane == 31) hist[kBuckets] = incl;
    }
    __syncwarp();
    int end[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        end[s] = 0;
        if (b[s] >= 0) {
            const int first = hist[b[s]];
            end[s] = hist[b[s] + 1];
            kd[first + at[s]] = d[s];  // the list was read above
            ki[first + at[s]] = id[s];
            at[s] = first;
        }
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        if (b[s] >= 0 && at[s] < k) {
            int rank = at[s];
            if (end[s] - at[s] > 1)
#pragma unroll 1
                for (int i = at[s]; i < end[s]; ++i) {
                    const unsigned long long o = kd[i];
                    rank += o < d[s] || (o == d[s] && ki[i] < id[s]);
                }
            if (rank < k) row[rank] = id[s];
        }
    }
    __syncwarp();
}

// The nodes first + i of the bits i of `which` go to leftover_kernel.
__device__ __forceinline__ void leave_over(const QueryArgs& a, int first, unsigned which, int lane) {
    int at = 0;
    if (lane == 0) at = atomicAdd(a.left, __popc(which));
    at = __shfl_sync(0xffffffffu, at, 0);
    if ((which >> lane) & 1u) a.list[at + __popc(which & ((1u << lane) - 1u))] = first + lane;
}

// One warp per cell (small sets: several), persistent over the cells. The general search
// spends 1,900 warp instructions a query, most of them on comparing every kept candidate
// with every other; here the candidate block is loaded once a cell and the
// ranking is linear in the kept ones: 530 a query at k = 21, 690 at k = 35. Bound by
// instruction issue (74 % of the issue slots at 27 warps per SM). The whole search, 1M nodes of
// a disk, k = 21: 2.24 ms by the general one, 0.52; 1M periodic, k = 35: 2.48, 0.85.
// NSMAX: kept entries a lane at most (keep_cap / 32); bounded to 8 CTAs (32
// warps, 64 registers) per SM, 6 for the largest lists.
template <bool PERIODIC, int NSMAX>
__global__ void __launch_bounds__(kWarps * 32, NSMAX > 5 ? 6 : 8) cell_query_kernel(const __grid_constant__ QueryArgs a) {
    extern __shared__ __align__(16) unsigned char knn_smem[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* base = knn_smem + w * cell_smem(a.cand_cap, a.keep_cap);
    double2* cxy = reinterpret_cast<double2*>(base);
    unsigned long long* kd = reinterpret_cast<unsigned long long*>(cxy + a.cand_cap);
    int* hist = reinterpret_cast<int*>(kd + a.keep_cap);
    int* cidx = hist + kBuckets + 4;
    int* ki = cidx + a.cand_cap;
    __shared__ Grid g;
    if (threadIdx.x == 0) g = a.g ? *a.g : a.gv;
    __syncthreads();
    const int k = a.k, items = g.cx * g.cy * a.split;
    const float want = (k + 1 + 1.9f * sqrtf(k + 1.0f)) / 3.14159265f;
    for (int item = blockIdx.x * kWarps + w; item < items; item += gridDim.x * kWarps) {
        // this warp's part of the cell's nodes
        const int cell = item / a.split, part = item - cell * a.split;
        const int first = a.start[cell], own = a.start[cell + 1] - first;
        const int q0 = first + own * part / a.split, qe = first + own * (part + 1) / a.split;
        const int q1 = min(qe, q0 + a.most);
        for (int qb = q1; qb < qe; qb += 32)
            leave_over(a, qb, qe - qb >= 32 ? 0xffffffffu : (1u << (qe - qb)) - 1u, lane);
        if (q0 == q1) continue;
        const int ccy = cell / g.cx, ccx = cell - ccy * g.cx;
        for (int qb = q0; qb < q1; qb += 32) {
            unsigned pending = q1 - qb >= 32 ? 0xffffffffu : (1u << (q1 - qb)) - 1u;
            int R = 2;
            bool shrunk = false;
            while (pending && R <= 3) {
                // the block's cells
                int xlo = ccx - R, xhi = ccx + R, ylo = ccy - R, yhi = ccy + R;
                bool fullx = false, fully = false;
                // edges of the block that nodes may lie behind
                double ex0 = -1e300, ex1 = 1e300, ey0 = -1e300, ey1 = 1e300;
                if (PERIODIC) {
                    fullx = 2 * R + 1 >= g.cx;
                    fully = 2 * R + 1 >= g.cy;
                    if (fullx) {
                        xlo = 0;
                        xhi = g.cx - 1;
                    } else {
                        ex0 = xlo * g.hx;
                        ex1 = (xhi + 1) * g.hx;
                    }
                    if (fully) {
                        ylo = 0;
                        yhi = g.cy - 1;
                    } else {
                        ey0 = ylo * g.hy;
                        ey1 = (yhi + 1) * g.hy;
                    }
                } else {
                    if (xlo > 0) ex0 = g.x0 + xlo * g.hx;
                    if (xhi < g.cx - 1) ex1 = g.x0 + (xhi + 1) * g.hx;
                    if (ylo > 0) ey0 = g.y0 + ylo * g.hy;
                    if (yhi < g.cy - 1) ey1 = g.y0 + (yhi + 1) * g.hy;
                    xlo = max(xlo, 0);
                    xhi = min(xhi, g.cx - 1);
                    ylo = max(ylo, 0);
                    yhi = min(yhi, g.cy - 1);
                }
                // its runs of consecutive cells, one a lane: the rows, and where the
                // block wraps in x the rows' second parts after them
                const int nrows = yhi - ylo + 1;
                const bool wrapx = PERIODIC && (xlo < 0 || xhi >= g.cx);
                const int nruns = wrapx ? 2 * nrows : nrows;
                int rbeg = 0, rlen = 0, own = 0;
                if (lane < nruns) {
                    const bool second = lane >= nrows;
                    int cyy = ylo + (second ? lane - nrows : lane);
                    if (PERIODIC) cyy += cyy < 0 ? g.cy : cyy >= g.cy ? -g.cy : 0;
                    int c0 = xlo, c1 = xhi;
                    if (wrapx) {
                        c0 = second ? 0 : xlo < 0 ? xlo + g.cx : xlo;
                        c1 = second ? (xlo < 0 ? xhi : xhi - g.cx) : g.cx - 1;
                    }
                    rbeg = a.start[cyy * g.cx + c0];
                    rlen = a.start[cyy * g.cx + c1 + 1] - rbeg;
                    // the run that holds the cell's own nodes
                    own = cyy == ccy && c0 <= ccx && ccx <= c1;
                }
                int incl = rlen;
#pragma unroll
                for (int o = 1; o < 16; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 15);
                const float area = static_cast<float>(nrows * (xhi - xlo + 1));
                // a dense block (by the list's capacity, at the plane's border also by its
                // density): one ring is mostly enough for k
                if (R == 2 && !shrunk && (total > a.cand_cap || total * 3.1416f > 1.6f * (k + 1) * area)) {
                    shrunk = true;
                    R = 1;
                    continue;
                }
                if (total > a.cand_cap) break;
                const int myoff = incl - rlen;
                const int ownlane = __ffs(__ballot_sync(0xffffffffu, own)) - 1;
                const int ownat = __shfl_sync(0xffffffffu, myoff - rbeg, ownlane) + qb;
#pragma unroll 1
                for (int r = 0; r < nruns; ++r) {
                    const int rb = __shfl_sync(0xffffffffu, rbeg, r);
                    const int rl = __shfl_sync(0xffffffffu, rlen, r);
                    const int ro = __shfl_sync(0xffffffffu, myoff, r);
#pragma unroll 1
                    for (int i = lane; i < rl; i += 32) {
                        cp_async16(cxy + ro + i, a.sxy + rb + i);
                        cp_async4(cidx + ro + i, a.sidx + rb + i);
                    }
                }
                cp_async_wait_all();
                for (int f = total + lane; f < ((total + 31) & ~31); f += 32)
                    cxy[f] = make_double2(INFINITY, INFINITY);
                __syncwarp();
                // differences cannot wrap when the block lies inside the box and is at
                // most half of it wide
                const bool wrap = PERIODIC && (fullx || fully || xlo < 0 || xhi >= g.cx || ylo < 0 ||
                                               yhi >= g.cy || 2 * (2 * R + 1) > g.cx ||
                                               2 * (2 * R + 1) > g.cy);
                // radius (squared) at which k + 1 nodes and 1.9 of their standard
                // deviations more are expected at the block's density
                const double est2 = g.hx * g.hy * (want * area / static_cast<float>(total));
                unsigned failed = 0;
                for (unsigned left = pending; left; left &= left - 1) {
                    const int i = __ffs(left) - 1;
                    const double2 qc = cxy[ownat + i];
                    const double b0 = qc.x - ex0, b1 = ex1 - qc.x, b2 = qc.y - ey0, b3 = ey1 - qc.y;
                    const double bx = b0 < b1 ? b0 : b1, by = b2 < b3 ? b2 : b3;
                    double bound = bx < by ? bx : by;
                    bound = bound * (1.0 - 1e-9) - 1e-15 * (fabs(qc.x) + fabs(qc.y));
                    // (a block that covers the whole domain bounds nothing)
                    const double bound2 = bound >= 1e299 ? INFINITY : bound > 0.0 ? bound * bound : 0.0;
                    double keep2 = bound2 < est2 ? bound2 : est2;
                    // a radius that keeps too few or too many entries changes by the
                    // density found, between the last that kept too few and the last
                    // that kept too many
                    float few = 0.f, many = INFINITY;
                    int have = 0;
                    for (int attempt = 0;; ++attempt) {
                        have = 0;
#pragma unroll 1
                        for (int f = lane; f - lane < total; f += 32) {
                            const double2 c = cxy[f];
                            double dx = dsub(qc.x, c.x), dy = dsub(qc.y, c.y);
                            if (wrap) {
                                dx = wrap_d(dx, g.Lx);
                                dy = wrap_d(dy, g.Ly);
                            }
                            const double d2 = dadd(dmul(dx, dx), dmul(dy, dy));
                            const bool ok = d2 < keep2;
                            const unsigned bal = __ballot_sync(0xffffffffu, ok);
                            const int pos = have + __popc(bal & ((1u << lane) - 1u));
                            if (ok && pos < a.keep_cap) {
                                kd[pos] = (unsigned long long)__double_as_longlong(d2);
                                ki[pos] = cidx[f];
                            }
                            have += __popc(bal);
                        }
                        __syncwarp();
                        const bool over = have > a.keep_cap;
                        if ((have >= k && !over) || attempt >= 5 || (!over && keep2 >= bound2)) break;
                        const float grow = fminf(4.f, 1.4f * (k + 1) / fmaxf(have, 1.f));
                        if (over)
                            many = static_cast<float>(keep2);
                        else
                            few = static_cast<float>(keep2);
                        double next = keep2 * (over ? grow : fmaxf(1.5f, grow));
                        if (!(next > few && next < many)) next = 0.5f * (few + many);
                        keep2 = next < bound2 ? next : bound2;
                    }
                    if (have < k || have > a.keep_cap) {
                        failed |= 1u << i;
                        continue;
                    }
                    // (an approximate reciprocal: the buckets only have to be monotone)
                    double scale;
                    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(scale) : "d"(keep2));
                    scale *= kBuckets;
                    int* row = a.ja + static_cast<size_t>(cidx[ownat + i]) * k;
                    if (have <= 32)
                        rank_kept<1>(kd, ki, hist, have, k, scale, row, lane);
                    else if (have <= 64)
                        rank_kept<2>(kd, ki, hist, have, k, scale, row, lane);
                    else if (have <= 96)
                        rank_kept<3>(kd, ki, hist, have, k, scale, row, lane);
                    else if (NSMAX > 3)
                        rank_kept<(NSMAX > 3 ? NSMAX : 4)>(kd, ki, hist, have, k, scale, row, lane);
                }
                pending = failed;
                ++R;
            }
            if (pending) leave_over(a, qb, pending, lane);  // what neither block completed
        }
    }
}

struct Workspace {
    size_t n_cap = 0, cells_cap = 0;
    int* cell_of = nullptr;
    int* rank = nullptr;
    Head* head = nullptr;  // followed by the cell counts (cells + 1)
    int* start = nullptr;  // cells + 1
    int* block_sums = nullptr;
    int* sidx = nullptr;
    double2* sxy = nullptr;
    Grid* grid = nullptr;
};

Workspace* ws_of(rbfb_ctx* ctx) { return static_cast<Workspace*>(ctx->knn_ws); }

void free_ws(Workspace* w) {
    cudaFree(w->cell_of); cudaFree(w->rank); cudaFree(w->sidx); cudaFree(w->sxy);
    cudaFree(w->head); cudaFree(w->start); cudaFree(w->block_sums); cudaFree(w->grid);
}

int ensure_ws(rbfb_ctx* ctx, size_t n, size_t cells) {
    if (!ctx->knn_ws) ctx->knn_ws = new Workspace();
    Workspace* w = ws_of(ctx);
    if (!w->grid) RBFB_CUDA(ctx, cudaMalloc(&w->grid, sizeof(Grid)));
    if (w->n_cap < n) {
        cudaFree(w->cell_of); cudaFree(w->rank); cudaFree(w->sidx); cudaFree(w->sxy);
        w->cell_of = w->rank = w->sidx = nullptr;
        w->sxy = nullptr;
        w->n_cap = 0;
        RBFB_CUDA(ctx, cudaMalloc(&w->cell_of, n * sizeof(int)));
        RBFB_CUDA(ctx, cudaMalloc(&w->rank, n * sizeof(int)));
        RBFB_CUDA(ctx, cudaMalloc(&w->sidx, n * sizeof(int)));
        RBFB_CUDA(ctx, cudaMalloc(&w->sxy, n * sizeof(double2)));
        w->n_cap = n;
    }
    if (w->cells_cap < cells) {
        cudaFree(w->head); cudaFree(w->start); cudaFree(w->block_sums);
        w->head = nullptr;
        w->start = w->block_sums = nullptr;
        w->cells_cap = 0;
        RBFB_CUDA(ctx, cudaMalloc(&w->head, sizeof(Head) + (cells + 1) * sizeof(int)));
        RBFB_CUDA(ctx, cudaMalloc(&w->start, (cells + 1) * sizeof(int)));
        RBFB_CUDA(ctx, cudaMalloc(&w->block_sums, ((cells + 1) / kScanBlock + 2) * sizeof(int)));
        w->cells_cap = cells;
    }
    return RBFB_OK;
}

// Mean nodes per cell. For the nodes' own stencils: larger cells share a block between
// more queries, but a block above the list's capacity (6.5 (k + 1)) falls back from two
// rings to one, in which not every query finds k. Measured for (k + 4 sqrt k) / 12.6, 10, 8, 7
// nodes a cell: 631, 614, 728, 537 us (1M disk, k = 21: a disk fills its box to 0.79, so at /
// 7 most cells take one ring), 891, 911, 951, 973 (1M periodic, k = 35), 1542, 773, 732, 676
// (300k nodes of fourfold varying density, k = 64).
// A small set takes smaller cells, towards a cell for every resident warp, down to
// 1.3 times what two rings need for k (1.0 times leaves many nodes of a varying
// density over). Arbitrary query points: kPerCell.
double per_cell(int k, int n, int sms, bool own) {
    if (!own) return kPerCell;
    const double root = std::sqrt(static_cast<double>(k));
    const double least = (k + 1 + 2.0 * root) / 8.8, most = (k + 4.0 * root) / 7.0;
    return std::max<double>(kPerCell, std::min(most, std::max(least, n / (16.0 * sms))));
}

// The cell grid over n nodes: its cells (periodic: its geometry too; open
// plane: at most that many cells, laid out on the device).
size_t plan_grid(int n, const double* period, double per, Grid& g) {
    const double cells = std::max(1.0, static_cast<double>(n) / per);
    if (!period) return static_cast<size_t>(cells);
    const double aspect = period[0] / period[1];
    const int cx = std::max(1, static_cast<int>(std::sqrt(cells * aspect)));
    const int cy = std::max(1, static_cast<int>(std::sqrt(cells / aspect)));
    g = Grid{0.0, 0.0, period[0] / cx, period[1] / cy, cx, cy, period[0], period[1], per};
    return static_cast<size_t>(cx) * cy;
}

// Enqueues the binning of the nodes into the arrays of w (one launch for a small
// set, else a memset and four launches, five in the open plane, one fewer when
// one block scans all cells); gp: the device grid (open plane) or nullptr
// (periodic: gv); *launches is increased. Returns the first error.
cudaError_t enqueue_bins(const Workspace& w, int n, const double* x, const double* y, size_t cells,
                         double per, const Grid* gp, const Grid& gv, int sms, cudaStream_t st,
                         int* launches) {
    if (n <= kSmallNodes && cells <= kSmallCells) {
        small_bins_kernel<<<1, 1024, 0, st>>>(x, y, n, static_cast<int>(cells), per, gv, gp ? w.grid : nullptr,
                                              w.head, w.start, w.sidx, w.sxy);
        *launches += 1;
        return cudaGetLastError();
    }
    const int ncell1 = static_cast<int>(cells) + 1;
    int* count = reinterpret_cast<int*>(w.head + 1);
    const cudaError_t e = cudaMemsetAsync(w.head, 0, sizeof(Head) + ncell1 * sizeof(int), st);
    if (e != cudaSuccess) return e;
    const int tpb = 256;
    const int blocks = std::max(1, std::min((n + tpb - 1) / tpb, sms * 8));
    if (gp)
        bbox_kernel<<<std::min(blocks, sms * 4), tpb, 0, st>>>(x, y, n, w.head, static_cast<int>(cells),
                                                               per, w.grid);
    cell_count_kernel<<<blocks, tpb, 0, st>>>(x, y, n, gp, gv, w.cell_of, w.rank, count);
    const int nsb = (ncell1 + kScanBlock - 1) / kScanBlock;
    scan_block_kernel<<<nsb, kScanBlock, 0, st>>>(count, w.start, ncell1, w.block_sums);
    if (nsb > 1) scan_add_kernel<<<nsb, kScanBlock, 0, st>>>(w.start, ncell1, w.block_sums);
    scatter_kernel<<<blocks, tpb, 0, st>>>(x, y, n, gp, gv, w.cell_of, w.rank, w.start, w.sidx, w.sxy);
    *launches += 3 + (gp ? 1 : 0) + (nsb > 1 ? 1 : 0);
    return cudaGetLastError();
}

QueryArgs query_args(const Workspace& w, const Grid* gp, const Grid& gv, int k, int* ja) {
    QueryArgs a{};
    a.g = gp;
    a.gv = gv;
    a.start = w.start;
    a.sidx = w.sidx;
    a.sxy = w.sxy;
    a.k = k;
    a.ja = ja;
    a.status = &w.head->status;
    a.list = w.rank;  // no longer needed
    a.left = &w.head->left;
    a.cand_cap = cand_cap_of(k);
    a.keep_cap = keep_cap_of(k);
    return a;
}

// The nodes' own stencils over the binned nodes. A small set's cells are shared by
// several warps, as many as the chip holds at once: 3,000 nodes of fourfold varying density,
// us, one warp a cell and several: k = 21 45 -> 39, k = 35 70 -> 42, k = 61 125 -> 51;
// periodic, 8,000 nodes, k = 56 three parts (one wave) 46, four 52. Above kSmallNodes about 48
// parts an SM (25,000 nodes of varying density, k = 61: 110 us, one a cell 163).
//
// A cell far above the mean would still leave its warps a long queue while the others
// are done: a warp takes 2.5 times the mean of a part, and the rest go to
// leftover_kernel, one warp each (8,000 nodes of thirtyfold varying density, k = 21:
// 112 -> 60 us; 3,000 nodes in twenty clusters, k = 28: 215 -> 75). In a grid of up to 5 x 5 cells a
// block is the whole set, and sharing it gains nothing on sets of uneven density: all nodes
// go there (200 nodes, k = 128, density falling a thousandfold: 181 us by cells, 38).
//
// A small set's list of candidates has room for a random set's 5 x 5 cells too (8,000
// nodes, k = 13: one ring was often too little, 60 -> 51 us).
constexpr int kMaxSplit = 32;
cudaError_t enqueue_cells(QueryArgs a, size_t cells, bool periodic, int sms, cudaStream_t st) {
    const bool small = a.nq <= kSmallNodes;
    if (small)
        a.cand_cap = std::min(kMaxCand, std::max(a.cand_cap, static_cast<int>(35.0 * a.nq / cells + 31) / 32 * 32));
    const size_t smem = kWarps * cell_smem(a.cand_cap, a.keep_cap);
    void (*kern)(QueryArgs) = nullptr;
    if (a.keep_cap <= 96)
        kern = periodic ? &cell_query_kernel<true, 3> : &cell_query_kernel<false, 3>;
    else if (a.keep_cap <= 160)
        kern = periodic ? &cell_query_kernel<true, 5> : &cell_query_kernel<false, 5>;
    else
        kern = periodic ? &cell_query_kernel<true, kMaxKeep / 32> : &cell_query_kernel<false, kMaxKeep / 32>;
    if (smem > 48 * 1024) {
        // the limit is the process's, not this call's: always the largest that a call
        // can ask for, or another thread's launch would be refused
        constexpr int most = static_cast<int>(kWarps * cell_smem(kMaxCand, kMaxKeep));
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return e;
    }
    // resident blocks an SM by the kernel's register bound and its shared memory
    const size_t per_sm = std::min<size_t>(a.keep_cap > 160 ? 6 : 8, (227 << 10) / (smem + 1024));
    const size_t items = static_cast<size_t>(sms) * (small ? kWarps * per_sm : 48);
    a.split = static_cast<int>(std::min<size_t>(kMaxSplit, std::max<size_t>(1, items / cells)));
    const double mean = a.nq / (static_cast<double>(cells) * a.split);
    a.most = cells <= 25 ? 0 : static_cast<int>(std::ceil(2.5 * mean)) + 1;
    const size_t want = (cells * a.split + kWarps - 1) / kWarps;
    const int blocks = static_cast<int>(std::max<size_t>(1, std::min<size_t>(want, sms * 64)));
    kern<<<blocks, kWarps * 32, smem, st>>>(a);
    const int rest = static_cast<int>(std::min<size_t>((a.nq + kWarps - 1) / kWarps, sms * 8));
    leftover_kernel<<<rest, kWarps * 32, 0, st>>>(a);
    return cudaGetLastError();
}

bool is_periodic(const double* period) { return period && period[0] > 0 && period[1] > 0; }

// Bins the nodes and finds the k nearest of every node (xq == nullptr) or of
// nq query points.
int search(rbfb_ctx* ctx, int n, const double* x, const double* y, int nq, const double* xq,
           const double* yq, int k, const double* period, int* ja, cudaStream_t st) {
    const bool periodic = is_periodic(period);
    const double per = per_cell(k, n, ctx->sms, !xq);
    Grid gv{};
    const size_t cells = plan_grid(n, periodic ? period : nullptr, per, gv);
    const int rc = ensure_ws(ctx, n, cells);
    if (rc) return rc;
    const Workspace& w = *ws_of(ctx);
    const Grid* gp = periodic ? nullptr : w.grid;
    int launches = 0;
    RBFB_CUDA(ctx, enqueue_bins(w, n, x, y, cells, per, gp, gv, ctx->sms, st, &launches));
    ctx->launches += launches;
    QueryArgs a = query_args(w, gp, gv, k, ja);
    if (!xq) {
        a.nq = n;
        RBFB_CUDA(ctx, enqueue_cells(a, cells, periodic, ctx->sms, st));
        ctx->launches += 1;
    } else {
        if (nq == 0) return RBFB_OK;
        a.nq = nq;
        a.qx = xq;
        a.qy = yq;
        const int blocks = std::max(1, std::min((nq + kWarps - 1) / kWarps, ctx->sms * 16));
        query_kernel<<<blocks, kWarps * 32, 0, st>>>(a);
        RBFB_CUDA(ctx, cudaGetLastError());
    }
    ctx->launches += 1;
    return RBFB_OK;
}

}  // namespace knn
}  // namespace rbfb

using namespace rbfb;

extern "C" {

void rbfb_release_knn(rbfb_ctx* ctx) {
    auto* w = static_cast<knn::Workspace*>(ctx->knn_ws);
    if (!w) return;
    knn::free_ws(w);
    delete w;
    ctx->knn_ws = nullptr;
}

static int knn_check(rbfb_ctx* ctx, int n, const double* x, const double* y, int k, const int* ja,
                     const double* period) {
    if (!x || !y || !ja) return fail(ctx, RBFB_EINVAL, "null pointer argument");
    if (n < 1 || k < 1 || k > n) return fail(ctx, RBFB_EINVAL, "need 1 <= k <= n");
    if (k > knn::kMaxK) return fail(ctx, RBFB_EUNSUPPORTED, "k above the search limit (128)");
    if (period && ((period[0] > 0) != (period[1] > 0)))
        return fail(ctx, RBFB_EINVAL, "periodic in both axes or neither");
    return RBFB_OK;
}

int rbfb_knn_stencils(rbfb_ctx* ctx, int n, const double* x, const double* y, int k,
                      const double* period_h, int* ja, void* stream) {
    if (!ctx) return RBFB_EINVAL;
    std::lock_guard<std::mutex> lock(ctx->mu);
    int rc = knn_check(ctx, n, x, y, k, ja, period_h);
    if (rc) return rc;
    RBFB_CUDA(ctx, cudaSetDevice(ctx->device));
    return knn::search(ctx, n, x, y, 0, nullptr, nullptr, k, period_h, ja,
                       static_cast<cudaStream_t>(stream));
}

int rbfb_knn_query(rbfb_ctx* ctx, int n, const double* x, const double* y, int nq,
                   const double* xq, const double* yq, int k, const double* period_h, int* ja,
                   void* stream) {
    if (!ctx) return RBFB_EINVAL;
    std::lock_guard<std::mutex> lock(ctx->mu);
    int rc = knn_check(ctx, n, x, y, k, ja, period_h);
    if (rc) return rc;
    if (nq < 0 || (nq > 0 && (!xq || !yq))) return fail(ctx, RBFB_EINVAL, "bad query arrays");
    RBFB_CUDA(ctx, cudaSetDevice(ctx->device));
    static const double none = 0.0;  // stands for the query arrays of an empty query
    return knn::search(ctx, n, x, y, nq, nq ? xq : &none, yq, k, period_h, ja,
                       static_cast<cudaStream_t>(stream));
}

// Status of the last search on this context's stream: 0 complete, 1 when a
// query gave up (more than 64 widenings). Synchronises `stream`.
int rbfb_knn_status(rbfb_ctx* ctx, void* stream) {
    if (!ctx || !ctx->knn_ws) return RBFB_EINVAL;
    int h = 0;
    RBFB_CUDA(ctx, cudaMemcpyAsync(&h, &knn::ws_of(ctx)->head->status, sizeof(int), cudaMemcpyDeviceToHost,
                                   static_cast<cudaStream_t>(stream)));
    RBFB_CUDA(ctx, cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
    return h;
}

}  // extern "C"

// ---- no-allocation variant: rbfb_knn_stencils_static ------------------------------
//
// Some callers may not allocate device memory once they are running: a solver
// loop that claimed all its device memory in a set-up phase and must not call
// cudaMalloc/cudaFree afterwards (those calls can synchronise the device and
// fragment the caller's pool), or a host application whose device memory is
// owned by another framework's allocator. For them this search keeps its
// scratch in a fixed array in device memory, defined below, instead of in a
// context: every GPU that loads the library holds the array until the process
// exits, and no call allocates anything.
namespace rbfb {
namespace knn {

constexpr int kStaticMaxNodes = 65536;                   // largest node set served
constexpr int kStaticMaxCells = kStaticMaxNodes / kPerCell;  // largest cell grid served
constexpr size_t al256(size_t b) { return (b + 255) & ~size_t(255); }
constexpr size_t kS_cell_of = 0;
constexpr size_t kS_rank = kS_cell_of + al256(4ull * kStaticMaxNodes);
constexpr size_t kS_head = kS_rank + al256(4ull * kStaticMaxNodes);  // and the counts
constexpr size_t kS_start = kS_head + al256(sizeof(Head) + 4ull * (kStaticMaxCells + 1));
constexpr size_t kS_bsums = kS_start + al256(4ull * (kStaticMaxCells + 1));
constexpr size_t kS_sidx = kS_bsums + al256(4ull * ((kStaticMaxCells + 1) / kScanBlock + 2));
constexpr size_t kS_sxy = kS_sidx + al256(4ull * kStaticMaxNodes);
constexpr size_t kS_grid = kS_sxy + al256(16ull * kStaticMaxNodes);
constexpr size_t kS_total = kS_grid + al256(sizeof(Grid));

// The scratch. In host code this name is only a stand-in for the device
// array, never a device address: host code takes the address with
// cudaGetSymbolAddress (per device) and passes it to the kernels.
static __device__ __align__(256) unsigned char g_knn_static[kS_total];

namespace {
std::mutex g_static_mu;
void* g_static_addr[64] = {};  // device address of the array, per device ordinal

// The array's device address on the current device: looked up once per
// device (cudaGetSymbolAddress, with that device current) and cached for the
// process. A cudaDeviceReset ends the context the address belongs to, so
// these entry points must not be used across one. nullptr on failure.
unsigned char* static_scratch(int* dev_out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    *dev_out = dev;
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_addr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_knn_static) != cudaSuccess || !p) return nullptr;
        g_static_addr[dev] = p;
    }
    return static_cast<unsigned char*>(g_static_addr[dev]);
}
}  // namespace

}  // namespace knn
}  // namespace rbfb

extern "C" int rbfb_knn_stencils_static(int n, const double* x, const double* y, int k,
                                        const double* period_h, int* ja, void* stream) {
    using namespace rbfb::knn;
    // the argument checks (and codes) of rbfb_knn_stencils
    if (!x || !y || !ja) return RBFB_EINVAL;
    if (n < 1 || k < 1 || k > n) return RBFB_EINVAL;
    if (k > kMaxK) return RBFB_EUNSUPPORTED;
    const bool periodic = period_h && period_h[0] > 0 && period_h[1] > 0;
    if (period_h && ((period_h[0] > 0) != (period_h[1] > 0))) return RBFB_EINVAL;
    if (n > kStaticMaxNodes) return RBFB_ETOOBIG;
    // the cell grid of the search, as rbfb_knn_stencils forms it
    int dev = 0;
    unsigned char* base = static_scratch(&dev);
    if (!base) return RBFB_ECUDA;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    sms = std::max(sms, 1);
    const double per = per_cell(k, n, sms, true);
    Grid gv{};
    const size_t cells = plan_grid(n, periodic ? period_h : nullptr, per, gv);
    if (cells > static_cast<size_t>(kStaticMaxCells)) return RBFB_ETOOBIG;
    Workspace w;
    w.cell_of = reinterpret_cast<int*>(base + kS_cell_of);
    w.rank = reinterpret_cast<int*>(base + kS_rank);
    w.head = reinterpret_cast<Head*>(base + kS_head);
    w.start = reinterpret_cast<int*>(base + kS_start);
    w.block_sums = reinterpret_cast<int*>(base + kS_bsums);
    w.sidx = reinterpret_cast<int*>(base + kS_sidx);
    w.sxy = reinterpret_cast<double2*>(base + kS_sxy);
    w.grid = reinterpret_cast<Grid*>(base + kS_grid);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Grid* gp = periodic ? nullptr : w.grid;
    int launches = 0;
    QueryArgs a = query_args(w, gp, gv, k, ja);
    a.nq = n;
    if (enqueue_bins(w, n, x, y, cells, per, gp, gv, sms, st, &launches) != cudaSuccess ||
        enqueue_cells(a, cells, periodic, sms, st) != cudaSuccess)
        return RBFB_ECUDA;
    return RBFB_OK;
}

// Completion status of the last rbfb_knn_stencils_static search on the
// current device: reads the status word of the fixed array into a host
// local (no allocation) and synchronises `stream`.
extern "C" int rbfb_knn_static_status(void* stream) {
    int dev = 0;
    unsigned char* base = rbfb::knn::static_scratch(&dev);
    if (!base) return RBFB_ECUDA;
    int h = 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemcpyAsync(&h, &reinterpret_cast<rbfb::knn::Head*>(base + rbfb::knn::kS_head)->status,
                        sizeof(int), cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return RBFB_ECUDA;
    return h;
}
