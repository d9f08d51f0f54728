// Transforms along y as whole two-step register FFTs (yfull_impl.cuh), for frames
// with many sampled rows (see yfft.cuh for few).
#pragma once

#include "pd_args.cuh"

namespace avx {

// length of the first step when these transforms are the faster ones for
// tiles x T CTAs of height H with at most max_rows sampled rows; else 0
int yfull_n1(int W, int H, int T, int max_rows);
// tables: inv[t H + kappa] = compact row of frame t with (ky - sy) mod H =
// kappa, or -1; phase[kappa] = e^{-2 pi i sy kappa / H} / sqrt(H)
void yfull_build(int H, int T, int sy, const int* rows, const int* row_off, int* inv, float2* phase);
// launch_ydft / launch_adjoint of pd_kernels.cuh; maps in the order of
// launch_yfft_maps with n1 = yfull_n1
void launch_yfull(const KArgs& k, cudaStream_t s);
void launch_yfull_adjoint(const KArgs& k, float2* img, cudaStream_t s);
// the attributes of height H's kernels
cudaError_t configure_yfull(int H);

}  // namespace avx
