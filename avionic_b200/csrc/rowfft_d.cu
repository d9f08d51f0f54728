// Row FFT instances (rowfft_impl.cuh).
#include "rowfft_impl.cuh"

namespace avx {

ROWFFT_DEFINE(20)

}  // namespace avx
