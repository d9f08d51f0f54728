// Two-step column transforms (yfull_impl.cuh): dispatch, tables, and the shorter heights.
#include <cmath>

#include "yfull_impl.cuh"

namespace avx {

YFULL_DEFINE(a, YFULL_SPLITS_A)

int yfull_n1(int W, int H, int T, int max_rows) {
  int n1 = yfull_first_a(H);
  if (!n1) n1 = yfull_first_b(H);
  if (!n1 || 2 * max_rows < 5 * n1) return 0;
  // From 2.5 n1 rows on the class sums' work (n1 terms a sample) exceeds the second step's (figures in yfull_impl.cuh).
  // The adjoint has one CTA a column tile and frame: below 8 warps an SM the class sums' CTAs, whose thread groups
  // share the coils out, fill the chip better.
  const long long warps = (long long)((W + 7) / 8) * T * ((8 * n1 + 31) / 32);
  return warps >= 148 * 8 ? n1 : 0;
}

void yfull_build(int H, int T, int sy, const int* rows, const int* row_off, int* inv, float2* phase) {
  for (int i = 0; i < T * H; ++i) inv[i] = -1;
  for (int t = 0; t < T; ++t)
    for (int r = row_off[t]; r < row_off[t + 1]; ++r) inv[(size_t)t * H + ((rows[r] - sy) % H + H) % H] = r - row_off[t];
  const double s = 1.0 / std::sqrt((double)H);
  for (int k = 0; k < H; ++k) {
    const double ang = -2.0 * M_PI * (double)((long long)sy * k % H) / H;
    phase[k] = make_float2((float)(std::cos(ang) * s), (float)(std::sin(ang) * s));
  }
}

static void run(int what, const KArgs& k, float2* img, cudaStream_t s) {
  if (!yfull_run_a(what, k, img, s)) yfull_run_b(what, k, img, s);
}
void launch_yfull(const KArgs& k, cudaStream_t s) { run(0, k, nullptr, s); }
void launch_yfull_adjoint(const KArgs& k, float2* img, cudaStream_t s) { run(1, k, img, s); }

cudaError_t configure_yfull(int H) {
  const cudaError_t e = yfull_set_a(H);
  return e == cudaSuccess ? yfull_set_b(H) : e;
}

}  // namespace avx
