// Radial grid transforms (radfft_impl.cuh): grid sizes 234 to 320.
#include "radfft_impl.cuh"

namespace avx {

RADFFT_DEFINE(d, FFT_SPLITS_D)

}  // namespace avx
