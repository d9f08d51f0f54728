// Gridding of radial samples for sectors of 8 x 8 cells (spread.cu).
#pragma once

#include "radial.cuh"

namespace avx {

// the grid has sectors of 8 x 8 cells, windows of 3 to 5 points and sides of at least 32 cells, and g does not ask for
// a block per sector
bool spread8_applies(const RadialGeomDev& g);
// launch_rad_spread of radial.cuh for such a grid
void launch_spread8(const RArgs& a, const float2* samples, cudaStream_t s);
// the attributes of the kernels of g's window width
cudaError_t configure_spread8(const RadialGeomDev& g);

}  // namespace avx
