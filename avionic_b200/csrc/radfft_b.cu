// Radial grid transforms (radfft_impl.cuh): grid sizes 130 to 176.
#include "radfft_impl.cuh"

namespace avx {

RADFFT_DEFINE(b, FFT_SPLITS_B)

}  // namespace avx
