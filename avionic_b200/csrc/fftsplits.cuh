// Two-factor splits N1 N2 of the transform lengths the two-step column
// transforms are built for: those of the oversampled grids of image sizes 64
// to 160 (the smallest even sizes with factors up to 13 at 1.5 and 2 times),
// which hold the benchmark's matrix sizes too.  Other grids (above 320: images
// of more than 160 at 2 times, of more than 213 at 1.5) run the Stockham passes.
// In four lists, one per translation unit.
#pragma once

#define FFT_SPLITS_A(X) X(12, 8) X(14, 7) X(10, 10) X(13, 8) X(12, 9) X(11, 10) X(14, 8) X(12, 10) X(14, 9) X(16, 8)
#define FFT_SPLITS_B(X) \
  X(13, 10) X(12, 11) X(14, 10) X(12, 12) X(15, 10) X(14, 11) X(13, 12) X(16, 10) X(18, 9) X(14, 12) X(16, 11)
#define FFT_SPLITS_C(X) \
  X(15, 12) X(14, 13) X(16, 12) X(14, 14) X(18, 11) X(20, 10) X(16, 13) X(15, 14) X(18, 12) X(20, 11) X(16, 14)
#define FFT_SPLITS_D(X) \
  X(18, 13) X(16, 15) X(18, 14) X(16, 16) X(20, 13) X(18, 15) X(20, 14) X(18, 16) X(20, 15) X(20, 16)

