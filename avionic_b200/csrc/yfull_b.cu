// Two-step column transforms (yfull_impl.cuh): the longer heights.
#include "yfull_impl.cuh"

namespace avx {

YFULL_DEFINE(b, YFULL_SPLITS_B)

}  // namespace avx
