// Partial DFTs along y as one short register FFT per residue class plus a
// short sum per sampled row (yfft.cu), fp32.
//
// With H = n1 n2 and y = j + n2 i, kappa = (ky - sy) mod H,
//   sum_y e^{+2 pi i kappa (y - sy) / H} u[y]
//     = sum_j e^{+2 pi i kappa (j - sy) / H} V_j[kappa mod n1],  V_j = n1-point DFT of u[j + n2 i] over i,
// and the adjoint is the transpose: the n1-point DFT of the class sums
// sum_{kappa = k1 mod n1} e^{-2 pi i kappa (j - sy) / H} Q[kappa].  Only the
// sampled rows enter the second sum, so a column costs n2 register FFTs and
// (sampled rows) n2 multiply-adds instead of (sampled rows) H.
#pragma once

#include "pd_args.cuh"

namespace avx {

// n1 of image height H with at most max_rows sampled rows per frame; 0 when
// the height has no factor that pays (the dense transforms are used)
int yfft_n1(int H, int max_rows);
// Per-operator tables (host side).  Entry p of frame t (row_off[t] <= p <
// row_off[t + 1]) is the frame's p-th row in ascending class kappa mod n1:
//   order_cls[p] = (compact row index within the frame, class)
//   coef[p n2 + j] = e^{+2 pi i kappa (j - sy) / H} / sqrt(H)
void yfft_build(int H, int T, int sy, int n1, const int* rows, const int* row_off, int2* order_cls, float2* coef);

// the coil maps in the order the kernels' threads read them (KArgs::b1t)
size_t yfft_maps_count(int W, int H, int C, int n1);
void launch_yfft_maps(const float2* b1, float2* out, int W, int H, int C, int n1, cudaStream_t s);

// y-transform of b1 x onto the sampled rows, and the column adjoint with the
// coil combination (launch_ydft / launch_adjoint of pd_kernels.cuh)
void launch_yfft(const KArgs& k, cudaStream_t s);
void launch_yfft_adjoint(const KArgs& k, float2* img, cudaStream_t s);
// the attributes of n1's kernels
cudaError_t configure_yfft(int n1);

}  // namespace avx
