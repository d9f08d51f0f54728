// Row transforms of the Cartesian operator with two-step register FFTs (rowfft_impl.cuh).
#pragma once

#include "pd_args.cuh"

namespace avx {

// W = n1 n2 with 8 <= n2 <= n1 <= 16, or n1 = 20, or one of the short splits
// (rowfft_impl.cuh); false when W has no such split (so 216, 234, 252, 270 and
// 288, which would need n1 = 18, run the Stockham passes)
bool rowfft_split(int W, int* n1, int* n2);

// the row kernel's work (launch_rows of pd_kernels.cuh) for a length with a
// split; mode 5: Q' = row-IFFT of the sampled rows of the dense k-space in
// k.dense_in (already masked)
void launch_rowfft(const KArgs& k, int mode, cudaStream_t s);
// the attributes of length W's kernels (nothing for a length without a split)
cudaError_t configure_rowfft(int W);

}  // namespace avx
