// Row FFT instances (rowfft_impl.cuh).
#include "rowfft_impl.cuh"

namespace avx {

ROWFFT_DEFINE(13)
ROWFFT_DEFINE(14)

}  // namespace avx
