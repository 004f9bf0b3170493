// Grid lengths with a compile-time two-pass factorisation N = N1 N2
// (oa_rdft.cuh): every 2-3-5 length from 12 to 160 whose two factors are at
// most 16, plus 125 = 5 x 25.  X(N, N1, N2).
//   OA_LENGTHS_LE108: lengths whose density planes fit in shared memory
//     (k_rho2_fwd / k_rho2_bwd hold two half planes)
//   OA_LENGTHS_ALL:   the z passes and the density z kernels
// N1 is a multiple of 4, for the band-pruned first DFT, where the length has
// such a pair of factors, but for 24 and 36.
// Other 2-3-5 lengths run the runtime-plan transforms (oa_fft.cuh).
#pragma once
#define OA_LENGTHS_LE108(X)                                                                              \
  X(12, 4, 3) X(15, 5, 3) X(16, 4, 4) X(18, 6, 3) X(20, 4, 5) X(24, 6, 4) X(25, 5, 5) X(27, 9, 3)        \
  X(30, 6, 5) X(32, 8, 4) X(36, 6, 6) X(40, 8, 5) X(45, 9, 5) X(48, 8, 6) X(50, 10, 5) X(54, 9, 6)       \
  X(60, 12, 5) X(64, 8, 8) X(72, 12, 6) X(75, 15, 5) X(80, 8, 10) X(81, 9, 9) X(90, 10, 9) X(96, 12, 8)  \
  X(100, 10, 10) X(108, 12, 9)
#define OA_LENGTHS_ALL(X)                                                                                \
  OA_LENGTHS_LE108(X) X(120, 12, 10) X(125, 5, 25) X(128, 16, 8) X(135, 15, 9) X(144, 12, 12)            \
  X(150, 15, 10) X(160, 16, 10)
