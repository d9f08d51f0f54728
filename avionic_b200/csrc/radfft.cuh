// Grid transforms of the radial operator with two-step register FFTs (radfft_impl.cuh).
#pragma once

#include "radial.cuh"

namespace avx {

// both grid sizes have a split n1 n2 the kernels are built for
bool radfft_applies(const RadialGeomDev& g);
// CTAs (and partial sums) of launch_radfft_interp
int radfft_forward_blocks(const RadialGeomDev& g);
// image -> samples: y transform of the padded, deapodised b1 (in - in2) onto
// every grid row of the image columns (into the first W columns of a.grid),
// then x transform and interpolation by blocks of grid rows; modes as
// launch_rad_interp
void launch_radfft_columns(const RArgs& a, cudaStream_t s);
void launch_radfft_interp(const RArgs& a, int mode, cudaStream_t s);
// grid -> image: x transform cropped to the image columns (in place), y
// transform cropped, deapodised and combined with conj(b1) into img
void launch_radfft_adjoint(const RArgs& a, float2* img, cudaStream_t s);
// the attributes of the kernels of g's grid sizes and window width
cudaError_t configure_radfft(const RadialGeomDev& g);

}  // namespace avx
