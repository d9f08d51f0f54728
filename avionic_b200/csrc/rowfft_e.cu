// Row FFT instances (rowfft_impl.cuh), short rows.
#include "rowfft_impl.cuh"

namespace avx {

// runs F<N1, N2> for the splits of the rule below
template <int N1, int N2>
constexpr bool short_split() {
  return N2 <= N1 && ((N1 * N2 >= 20 && N1 * N2 <= 32 && N2 <= 5 && N1 <= 13) ||
                      (N1 * N2 > 32 && N1 >= 7 && N2 >= 5 && N2 <= 7));
}

bool rowfft_short_split(int W, int* n1, int* n2) {
  for (int a = 5; a <= 16; ++a) {
    if (W % a) continue;
    const int b = W / a;
    if (b > a || b < 2) continue;
    if ((W >= 20 && W <= 32 && b <= 5 && a <= 13) || (W > 32 && a >= 7 && b >= 5 && b <= 7)) {
      *n1 = a;
      *n2 = b;
      return true;
    }
  }
  return false;
}

template <int N1, int N2>
static void launch_rec(int n1, int n2, const KArgs& k, int mode, cudaStream_t s) {
  if constexpr (N1 <= 16) {
    if constexpr (N2 > 7) {
      launch_rec<N1 + 1, 2>(n1, n2, k, mode, s);
    } else {
      if constexpr (short_split<N1, N2>()) {
        if (n1 == N1 && n2 == N2) {
          rowfft_launch<N1, N2>(k, mode, s);
          return;
        }
      }
      launch_rec<N1, N2 + 1>(n1, n2, k, mode, s);
    }
  }
}
template <int N1, int N2>
static cudaError_t configure_rec(int n1, int n2) {
  if constexpr (N1 <= 16) {
    if constexpr (N2 > 7) {
      return configure_rec<N1 + 1, 2>(n1, n2);
    } else {
      if constexpr (short_split<N1, N2>()) {
        if (n1 == N1 && n2 == N2) return rowfft_configure<N1, N2>();
      }
      return configure_rec<N1, N2 + 1>(n1, n2);
    }
  }
  return cudaSuccess;
}

void rowfft_launch_short(int n1, int n2, const KArgs& k, int mode, cudaStream_t s) {
  launch_rec<5, 2>(n1, n2, k, mode, s);
}
cudaError_t rowfft_configure_short(int n1, int n2) { return configure_rec<5, 2>(n1, n2); }

}  // namespace avx
