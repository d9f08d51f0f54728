// Radial grid transforms (radfft_impl.cuh): dispatch, and grid sizes 96 to 128.
#include "radfft_impl.cuh"

namespace avx {

RADFFT_DEFINE(a, FFT_SPLITS_A)

static bool run(int G, int what, const RArgs* a, int mode, float2* img, cudaStream_t s) {
  return radfft_run_a(G, what, a, mode, img, s) || radfft_run_b(G, what, a, mode, img, s) ||
         radfft_run_c(G, what, a, mode, img, s) || radfft_run_d(G, what, a, mode, img, s);
}

bool radfft_applies(const RadialGeomDev& g) {
  if (g.nw < 3 || g.nw > 5) return false;  // windows the interpolating pass is built for
  if (!run(g.Gx, 0, nullptr, 0, nullptr, 0) || !run(g.Gy, 0, nullptr, 0, nullptr, 0)) return false;
  const size_t sm = radfft_interp_smem_a(g) + radfft_interp_smem_b(g) + radfft_interp_smem_c(g) + radfft_interp_smem_d(g);
  return sm <= AVX_DYN_SMEM_MAX;
}

int radfft_forward_blocks(const RadialGeomDev& g) {
  const int srb = rad_block_sectors(g);
  return (g.nsy + srb - 1) / srb * g.C * g.T;
}

void launch_radfft_columns(const RArgs& a, cudaStream_t s) { run(a.g.Gy, 0, &a, 0, nullptr, s); }
void launch_radfft_interp(const RArgs& a, int mode, cudaStream_t s) { run(a.g.Gx, 1, &a, mode, nullptr, s); }
void launch_radfft_adjoint(const RArgs& a, float2* img, cudaStream_t s) {
  run(a.g.Gx, 2, &a, 0, nullptr, s);
  run(a.g.Gy, 3, &a, 0, img, s);
}

cudaError_t configure_radfft(const RadialGeomDev& g) {
  cudaError_t e = radfft_set_a(g);
  if (e == cudaSuccess) e = radfft_set_b(g);
  if (e == cudaSuccess) e = radfft_set_c(g);
  if (e == cudaSuccess) e = radfft_set_d(g);
  return e;
}

}  // namespace avx
