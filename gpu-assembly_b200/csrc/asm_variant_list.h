// asm_variant_list.h -- every compiled shape of the assembly kernels, one
// line each, and the build compiles each line as its own translation unit. The
// first shape of a class (degree, exponent, smallest NMAX that holds the system)
// is its default.
//
// RBFB_DM_VARIANT(name, NMAX, NRHS, P, Q, NW, GPB, MINB): the FP64 kernel
// (asm_dmma.cuh): systems of n <= NMAX unknowns (stencil size + polynomial
// terms) with up to NRHS right-hand sides, degree P, PHS exponent Q, NW warps a
// stencil, GPB stencils a CTA, MINB resident CTAs. Measured on the
// B200, 262,144 stencils (65,536 at degree 4), ms: k = 35 three one-warp
// stencils a CTA 3.40, four 3.42, one 3.52; k = 21 one a CTA 1.53, four 1.60;
// k = 64 two warps a stencil 4.09, four 4.13.
//
// RBFB_IR_VARIANT(name, NMAX, NRHS, P, Q, GPB, MINB): the refined form
// (asm_refined.cuh), one warp a stencil, GPB stencils a CTA. Same counts, ms:
// k = 35 five stencils a CTA 6.40, ten 6.44, two 6.53, three (9 resident) 7.17, one
// 7.37; k = 38 nine 7.28, three 7.49; k = 21 four 2.17, one 2.19; k = 45, degree 4
// 6.63 in the 64 class, 10.46 in the 80 class; k = 64 14.5, of which the FP64 kernel
// takes 4.1 (it redoes nearly all).
RBFB_DM_VARIANT(b64_p2q3_n32_w1x1, 32, 3, 2, 3, 1, 1, 20)
RBFB_DM_VARIANT(b64_p2q3_n32_w1x4_r8, 32, 8, 2, 3, 1, 4, 4)
RBFB_DM_VARIANT(b64_p3q5_n45_w1x3, 45, 3, 3, 5, 1, 3, 4)
RBFB_DM_VARIANT(b64_p3q5_n45_w1x1, 45, 3, 3, 5, 1, 1, 12)
RBFB_DM_VARIANT(b64_p3q5_n48_w1x3, 48, 3, 3, 5, 1, 3, 3)
RBFB_DM_VARIANT(b64_p4q7_n64_w1, 64, 3, 4, 7, 1, 1, 6)
RBFB_DM_VARIANT(b64_p4q7_n64_w2, 64, 3, 4, 7, 2, 1, 6)
RBFB_DM_VARIANT(b64_p4q7_n80_w2, 80, 3, 4, 7, 2, 1, 4)
RBFB_DM_VARIANT(b64_p4q7_n80_w4, 80, 3, 4, 7, 4, 1, 4)
RBFB_IR_VARIANT(bmx_p2q3_n32_w1x4, 32, 3, 2, 3, 4, 4)
RBFB_IR_VARIANT(bmx_p2q3_n32_w1x1, 32, 3, 2, 3, 1, 16)
RBFB_IR_VARIANT(bmx_p3q5_n45_w1x5, 45, 3, 3, 5, 5, 2)
RBFB_IR_VARIANT(bmx_p3q5_n45_w1x1, 45, 3, 3, 5, 1, 9)
RBFB_IR_VARIANT(bmx_p3q5_n48_w1x9, 48, 3, 3, 5, 9, 1)
RBFB_IR_VARIANT(bmx_p3q5_n48_w1x3, 48, 3, 3, 5, 3, 3)
RBFB_IR_VARIANT(bmx_p4q7_n64_w1x5, 64, 3, 4, 7, 5, 1)
RBFB_IR_VARIANT(bmx_p4q7_n80_w1x3, 80, 3, 4, 7, 3, 1)
