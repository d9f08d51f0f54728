// Row FFT instances (rowfft_impl.cuh), first step of 8 to 12 points, and the dispatch.
#include "rowfft_impl.cuh"

namespace avx {

ROWFFT_DEFINE(8)
ROWFFT_DEFINE(9)
ROWFFT_DEFINE(10)
ROWFFT_DEFINE(11)
ROWFFT_DEFINE(12)

bool rowfft_split(int W, int* n1, int* n2) {
  // the most balanced split: the fewest threads of a row idle in either step
  for (int a : {8, 9, 10, 11, 12, 13, 14, 15, 16, 20}) {
    if (W % a) continue;
    const int b = W / a;
    if (b < 8 || b > a || b > 16) continue;
    *n1 = a;
    *n2 = b;
    return true;
  }
  return rowfft_short_split(W, n1, n2);
}

void launch_rowfft(const KArgs& k, int mode, cudaStream_t s) {
  int n1 = 0, n2 = 0;
  if (!rowfft_split(k.g.W, &n1, &n2)) return;
  if (n2 < 8) {
    rowfft_launch_short(n1, n2, k, mode, s);
    return;
  }
#define CALL_W(N) \
  case N: rowfft_launch_##N(n2, k, mode, s); break;
  switch (n1) {
    CALL_W(8)
    CALL_W(9)
    CALL_W(10)
    CALL_W(11)
    CALL_W(12)
    CALL_W(13)
    CALL_W(14)
    CALL_W(15)
    CALL_W(16)
    CALL_W(20)
    default: break;
  }
#undef CALL_W
}

cudaError_t configure_rowfft(int W) {
  int n1 = 0, n2 = 0;
  if (!rowfft_split(W, &n1, &n2)) return cudaSuccess;
  if (n2 < 8) return rowfft_configure_short(n1, n2);
#define CASE_W(N) \
  case N: return rowfft_configure_##N(n2);
  switch (n1) {
    CASE_W(8)
    CASE_W(9)
    CASE_W(10)
    CASE_W(11)
    CASE_W(12)
    CASE_W(13)
    CASE_W(14)
    CASE_W(15)
    CASE_W(16)
    CASE_W(20)
    default: return cudaSuccess;
  }
#undef CASE_W
}

}  // namespace avx
