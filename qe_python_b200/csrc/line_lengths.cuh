// Line lengths with compile-time kernels: X(n, n1, n2, k1, k2), n = n1 n2,
// every 2-3-5 smooth n from 16 to 192 whose factors fit a small DFT
// (line_dft.cuh).  k1 <= k2: blocks of n2 values at each end of a line that
// the wave-function sphere reaches, for ecutrho near 6 and 4 ecutwfc (the
// sphere spans 0.41 and 0.5 of the grid); n1 is the factor that wastes the
// fewest rows on whole blocks, except for 36 and 144: DFT9 and DFT16 have twiddles
// of their own, and the two equal factors round less (36^3 FP64 4.5e-16 relative
// against 5.4e-16 with 4 x 9, 144^3 FP32 2.2e-7 against 2.9e-7 with 16 x 9) and
// measured faster on square planes (144^3, 96 bands FP32 1352 and 1517 us).
#pragma once

#define QEB_LINE_LENGTHS(X)                                                            \
  X(16, 4, 4, 1, 1) X(18, 3, 6, 1, 1) X(20, 4, 5, 1, 1) X(24, 4, 6, 1, 1)              \
  X(25, 5, 5, 2, 2) X(27, 3, 9, 1, 1) X(30, 6, 5, 2, 2) X(32, 4, 8, 1, 1)              \
  X(36, 6, 6, 2, 2) X(40, 8, 5, 2, 2) X(45, 9, 5, 2, 3) X(48, 8, 6, 2, 2)              \
  X(50, 10, 5, 3, 3) X(54, 9, 6, 2, 3) X(60, 12, 5, 3, 3) X(64, 8, 8, 2, 2)            \
  X(72, 8, 9, 2, 2) X(75, 15, 5, 3, 4) X(80, 8, 10, 2, 2) X(81, 9, 9, 2, 3)            \
  X(90, 10, 9, 2, 3) X(96, 12, 8, 3, 3) X(100, 10, 10, 2, 3) X(108, 12, 9, 3, 3)       \
  X(120, 12, 10, 3, 3) X(128, 16, 8, 4, 4) X(135, 15, 9, 3, 4) X(144, 12, 12, 3, 3)     \
  X(150, 15, 10, 3, 4) X(160, 16, 10, 4, 4) X(180, 15, 12, 3, 4) X(192, 16, 12, 4, 4)
