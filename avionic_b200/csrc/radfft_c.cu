// Radial grid transforms (radfft_impl.cuh): grid sizes 180 to 224.
#include "radfft_impl.cuh"

namespace avx {

RADFFT_DEFINE(c, FFT_SPLITS_C)

}  // namespace avx
