// asm_variant_list.h -- every compiled shape of the assembly kernel, one
// line each: RBFB_VARIANT(name, T, GR, GC, NTP, NRHS, P, Q, MIXED, BLOCK, MINB, SMEM, PF)
//   T        compute type of the elimination (double: FP64, float: FP32 + FP64 refinement)
//   GR x GC  lanes per stencil (row groups x column groups), <= 32
//   NTP      padded system size (stencil size + polynomial terms <= NTP)
//   NRHS     right-hand sides compiled in; P, Q degree and PHS exponent
//   MIXED    FP32 factorisation with FP64 refinement
//   BLOCK    threads per CTA; MINB minimum resident CTAs (register budget hint)
//   SMEM     elimination on the matrix in shared memory (large systems) instead
//            of register rows
//   PF       prefetch the next stencil's neighbour data (cp.async) while the
//            current one is solved; off where the extra live state costs the
//            register-bound elimination more than the gather latency it hides
//
// RBFB_BLK_VARIANT(name, T, NMAX, NRHS, P, Q, MIXED, BLOCK, MINB, PB, PF): the
// blocked shared-memory kernel (asm_blocked.cuh), one warp per stencil, any
// system size n <= NMAX, panels of PB columns (the refined form).
//
// RBFB_DM_VARIANT(name, NMAX, NRHS, P, Q, NW, GPB, MINB): the FP64 kernel
// (asm_dmma.cuh), n <= NMAX, NW warps a stencil, GPB stencils a CTA, MINB
// resident CTAs. The first shape of a class is its default. Measured on the
// B200, 262,144 stencils (65,536 at degree 4), ms: k = 35 three one-warp
// stencils a CTA 3.40, four 3.42, one 3.52; k = 21 one a CTA 1.53, four 1.60;
// k = 64 two warps a stencil 4.09, four 4.13.
// The build compiles each line as its own translation unit.
RBFB_DM_VARIANT(b64_p2q3_n32_w1x1, 32, 3, 2, 3, 1, 1, 20)
RBFB_DM_VARIANT(b64_p2q3_n32_w1x4_r8, 32, 8, 2, 3, 1, 4, 4)
RBFB_DM_VARIANT(b64_p3q5_n45_w1x3, 45, 3, 3, 5, 1, 3, 4)
RBFB_DM_VARIANT(b64_p3q5_n45_w1x1, 45, 3, 3, 5, 1, 1, 12)
RBFB_DM_VARIANT(b64_p3q5_n48_w1x3, 48, 3, 3, 5, 1, 3, 3)
RBFB_DM_VARIANT(b64_p4q7_n64_w1, 64, 3, 4, 7, 1, 1, 6)
RBFB_DM_VARIANT(b64_p4q7_n64_w2, 64, 3, 4, 7, 2, 1, 6)
RBFB_DM_VARIANT(b64_p4q7_n80_w2, 80, 3, 4, 7, 2, 1, 4)
RBFB_DM_VARIANT(b64_p4q7_n80_w4, 80, 3, 4, 7, 4, 1, 4)
RBFB_BLK_VARIANT(bmx_p3q5_n45_pb8, float, 45, 3, 3, 5, true, 32, 1, 8, true)
RBFB_BLK_VARIANT(bmx_p3q5_n45_pb8x3, float, 45, 3, 3, 5, true, 96, 1, 8, true)
RBFB_BLK_VARIANT(bmx_p2q3_n32_pb8, float, 32, 3, 2, 3, true, 32, 1, 8, true)
RBFB_BLK_VARIANT(bmx_p4q7_n80_pb8, float, 80, 3, 4, 7, true, 32, 1, 8, true)
RBFB_VARIANT(mix_p2q3_n32_g16x1, float, 16, 1, 32, 3, 2, 3, true, 64, 1, false, true)
RBFB_VARIANT(mix_p2q3_n32_g16x2, float, 16, 2, 32, 3, 2, 3, true, 64, 1, false, true)
RBFB_VARIANT(mix_p3q5_n48_g16x2, float, 16, 2, 48, 3, 3, 5, true, 64, 4, false, true)
RBFB_VARIANT(mix_p3q5_n48_g16x1, float, 16, 1, 48, 3, 3, 5, true, 64, 1, false, true)
RBFB_VARIANT(mix_p4q7_n64_smem, float, 16, 2, 64, 3, 4, 7, true, 32, 1, true, true)
RBFB_VARIANT(mix_p4q7_n80_smem, float, 16, 2, 80, 3, 4, 7, true, 32, 1, true, true)
