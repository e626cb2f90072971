// face32.cuh -- the float32 face passes (interface between face32.cu and
// kernels.cu; not part of the C ABI).
#pragma once
#include "face.cuh"

namespace astro_face32 {

// one direction's faces (a.dir), then the listed ones again in float64;
// given: the x faces with the carried z-face speeds
cudaError_t launch(const astro::FaceArgs& a, bool given, cudaStream_t s);

}  // namespace astro_face32
