// asm_variant_make.cuh -- defines one compiled shape of the assembly kernel
// (RBFB_DEFINE_VARIANT) and the Variant record the runtime launches it by.
#pragma once

#include <cuda_runtime.h>

#include "asm_blocked.cuh"
#include "asm_dmma.cuh"
#include "asm_kernel.cuh"
#include "asm_variants.h"

namespace rbfb {

template <typename T, int GR, int GC, int NTP, int NRHS, int P, int Q, bool MIXED, int BLOCK,
          int MINB, bool SMEM, bool PF>
Variant make_variant(const char* name) {
    using C = AsmCfg<T, GR, GC, NTP, NRHS, P, Q, MIXED, SMEM>;
    Variant v{};
    v.name = name;
    v.kernel =
        reinterpret_cast<const void*>(&asm_kernel<T, GR, GC, NTP, NRHS, P, Q, MIXED, BLOCK, MINB, SMEM, PF>);
    v.launch = [](dim3 grid, int block, size_t smem, cudaStream_t st, const AsmParams& p) {
        asm_kernel<T, GR, GC, NTP, NRHS, P, Q, MIXED, BLOCK, MINB, SMEM, PF><<<grid, block, smem, st>>>(p);
    };
    v.mixed = MIXED;
    v.P = P;
    v.Q = Q;
    v.ntp = NTP;
    v.nrhs = NRHS;
    v.group = C::G;
    v.block = BLOCK;
    v.smem_group = C::bytes;
    v.smem_block = C::bytes * (BLOCK / C::G);
    return v;
}

template <typename T, int NMAX, int NRHS, int P, int Q, bool MIXED, int BLOCK, int MINB, int PB,
          bool PF>
Variant make_blk_variant(const char* name) {
    using C = BlkCfg<T, NMAX, NRHS, P, Q, MIXED, PB>;
    Variant v{};
    v.name = name;
    v.kernel = reinterpret_cast<const void*>(
        &blk_kernel<T, NMAX, NRHS, P, Q, MIXED, BLOCK, MINB, PB, PF>);
    v.launch = [](dim3 grid, int block, size_t smem, cudaStream_t st, const AsmParams& p) {
        blk_kernel<T, NMAX, NRHS, P, Q, MIXED, BLOCK, MINB, PB, PF><<<grid, block, smem, st>>>(p);
    };
    v.mixed = MIXED;
    v.P = P;
    v.Q = Q;
    v.ntp = NMAX;
    v.nrhs = NRHS;
    v.group = C::G;
    v.block = BLOCK;
    v.smem_group = C::bytes;
    v.smem_block = C::bytes * (BLOCK / C::G);
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

#define RBFB_DEFINE_BLK_VARIANT(name, T, NMAX, NRHS, P, Q, MIXED, BLOCK, MINB, PB, PF)          \
    namespace rbfb {                                                                           \
    Variant variant_##name() {                                                                 \
        return make_blk_variant<T, NMAX, NRHS, P, Q, MIXED, BLOCK, MINB, PB, PF>(#name);       \
    }                                                                                          \
    }

#define RBFB_DEFINE_VARIANT(name, T, GR, GC, NTP, NRHS, P, Q, MIXED, BLOCK, MINB, SMEM, PF)    \
    namespace rbfb {                                                                           \
    Variant variant_##name() {                                                                 \
        return make_variant<T, GR, GC, NTP, NRHS, P, Q, MIXED, BLOCK, MINB, SMEM, PF>(#name);  \
    }                                                                                          \
    }
