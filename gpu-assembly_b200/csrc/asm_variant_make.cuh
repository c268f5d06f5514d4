// asm_variant_make.cuh -- defines one compiled shape of the assembly kernel
// (RBFB_DEFINE_VARIANT) and the Variant record the runtime launches it by.
#pragma once

#include <cuda_runtime.h>

#include "asm_dmma.cuh"
#include "asm_common.cuh"
#include "asm_refined.cuh"
#include "asm_variants.h"

namespace rbfb {

template <int NMAX, int NRHS, int P, int Q, int GPB, int MINB>
Variant make_ir_variant(const char* name) {
    using L = ir::Layout<NMAX, NRHS, NMAX - npoly(P)>;
    Variant v{};
    v.name = name;
    v.kernel = reinterpret_cast<const void*>(&ir::ir_kernel<NMAX, NRHS, P, Q, GPB, MINB>);
    v.launch = [](dim3 grid, int block, size_t smem, cudaStream_t st, const AsmParams& p) {
        ir::ir_kernel<NMAX, NRHS, P, Q, GPB, MINB><<<grid, block, smem, st>>>(p);
    };
    v.mixed = true;
    v.P = P;
    v.Q = Q;
    v.ntp = NMAX;
    v.nrhs = NRHS;
    v.group = 32;
    v.block = 32 * GPB;
    v.smem_group = L::bytes;
    v.smem_block = L::bytes * GPB;
    return v;
}

template <int NMAX, int NRHS, int P, int Q, int NW, int GPB, int MINB>
Variant make_dm_variant(const char* name) {
    using L = dm::Layout<NMAX, NRHS, NMAX - npoly(P)>;
    Variant v{};
    v.name = name;
    v.kernel = reinterpret_cast<const void*>(&dm::dm_kernel<NMAX, NRHS, P, Q, NW, GPB, MINB>);
    v.launch = [](dim3 grid, int block, size_t smem, cudaStream_t st, const AsmParams& p) {
        dm::dm_kernel<NMAX, NRHS, P, Q, NW, GPB, MINB><<<grid, block, smem, st>>>(p);
    };
    v.mixed = false;
    v.P = P;
    v.Q = Q;
    v.ntp = NMAX;
    v.nrhs = NRHS;
    v.group = 32 * NW;
    v.block = 32 * NW * GPB;
    v.smem_group = L::bytes;
    v.smem_block = L::bytes * GPB;
    return v;
}

}  // namespace rbfb

#define RBFB_DEFINE_DM_VARIANT(name, NMAX, NRHS, P, Q, NW, GPB, MINB)                           \
    namespace rbfb {                                                                           \
    Variant variant_##name() {                                                                 \
        return make_dm_variant<NMAX, NRHS, P, Q, NW, GPB, MINB>(#name);                        \
    }                                                                                          \
    }

#define RBFB_DEFINE_IR_VARIANT(name, NMAX, NRHS, P, Q, GPB, MINB)                               \
    namespace rbfb {                                                                           \
    Variant variant_##name() { return make_ir_variant<NMAX, NRHS, P, Q, GPB, MINB>(#name); }   \
    }
