// Row FFT instances (rowfft_impl.cuh).
#include "rowfft_impl.cuh"

namespace avx {

ROWFFT_DEFINE(15)
ROWFFT_DEFINE(16)

}  // namespace avx
