// asm_common.cuh -- what the assembly kernels (asm_dmma.cuh, asm_refined.cuh)
// share: the launch parameters, asynchronous copies, and the right-hand sides
// of the saddle-point system (fill_rhs, src/rbf_operators.h:116-185).
#pragma once

#include <cstdint>

#include "asm_math.cuh"

namespace rbfb {

constexpr int kMaxRhs = 8;

struct AsmParams {
    int nitems;               // stencils to process (list entries, or 0..nitems-1)
    int item_base;            // first stencil id when list is nullptr
    const int* list;          // stencil ids, or nullptr
    const int* nitems_dev;    // device-side item count (overrides nitems when set)
    const int* list_off_dev;  // device-side offset into list and fb_list, or nullptr
    const double* x;
    const double* y;
    const int* ja;  // fixed width: row s at ja + s*k; CSR: ja + ia[s]
    const int* ia;  // nullptr for fixed width
    int k;          // fixed width stencil size
    int stride;     // entries from a row to the next: k (CSR: 1, a row is its first entry)
    int row_base;   // fixed width: ja, values and info hold rows row_base.. only
    double Lx, Ly;  // periods (<= 0: open axis)
    int scale;
    int nrhs;
    int plain_ops;            // every column is Laplace, d/dx or d/dy
    int col_op[kMaxRhs];  // RBFB_OP_* of every right-hand-side column
    int col_ic[kMaxRhs];  // interpolation point index of OP_INTERP columns
    const double* xc;
    const double* yc;
    double* values[kMaxRhs];
    double* const* values_dev;  // the same table in device memory (read when set)
    int* info;
    // refinement
    int max_sweeps;
    double ir_tol;
    int* fb_list;  // stencils handed to the FP64 kernel
    int* fb_count;
    unsigned long long* sweeps_sum;
    int* sweeps_max;
    int* work;  // dynamic work counter, or nullptr for a static stride
};

// Output array of right-hand side q: from the device-resident table when the
// caller passed one (the reference's T* const* A), else from the parameters.
__device__ __forceinline__ double* out_column(const AsmParams& p, int q) {
    return p.values_dev ? p.values_dev[q] : p.values[q];
}

// Asynchronous global -> shared copies (cp.async, no register staging):
// the next stencil's data is fetched while the current one is solved.
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Right-hand sides of node row (xi, yi): every column q < nrhs, FP64, the
// PHS power r^(Q-2) shared by the derivative operators (one square root).
template <int P, int Q, int NRHS>
__device__ __forceinline__ void rhs_node(const AsmParams& p, double xi, double yi, int e,
                                         double* out) {
    const double r2 = dist2(xi, yi);
    const double rq2 = phs64<Q - 2>(r2);
    const double q = static_cast<double>(Q);
    const double qr = dmul(q, rq2);
#pragma unroll
    for (int c = 0; c < NRHS; ++c) {
        double v = 0.0;
        if (c < p.nrhs) {
            const int op = p.col_op[c];
            switch (op) {
                case kOpInterp: {
                    const double xe = scalbn(p.xc[p.col_ic[c]], -e);
                    const double ye = scalbn(p.yc[p.col_ic[c]], -e);
                    v = phs64<Q>(dist2(dsub(xe, xi), dsub(ye, yi)));
                    break;
                }
                case kOpLaplace: v = dmul(q * q, rq2); break;
                case kOpDx: v = -dmul(qr, xi); break;
                case kOpDy: v = -dmul(qr, yi); break;
                default: v = phs_op_origin<Q>(op, xi, yi); break;
            }
        }
        out[c] = v;
    }
}
template <int P>
__device__ __forceinline__ double rhs_poly(const AsmParams& p, int q, int m, int e) {
    const int op = p.col_op[q];
    if (op == kOpInterp) {
        int a, b;
        mono_exps(m, a, b);
        return mono_ab<P>(scalbn(p.xc[p.col_ic[q]], -e), scalbn(p.yc[p.col_ic[q]], -e), a, b);
    }
    return poly_op_origin(op, m);
}

}  // namespace rbfb
