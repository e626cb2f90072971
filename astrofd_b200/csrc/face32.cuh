// face32.cuh -- the float32 face passes (interface between face32.cu and
// kernels.cu; not part of the C ABI).
#pragma once
#include "face.cuh"

namespace astro_face32 {

// the faces of x, y and z (dirs[0..2]), then the listed ones again in float64;
// launched: called after each direction (the kernel timing's events)
cudaError_t launch_all(const astro::FaceArgs* dirs, int sms, void (*launched)(cudaStream_t), cudaStream_t s);
// one direction's faces (a.dir), then its listed ones, for RMHD PPM and WENO5 in
// the reference's flux mode, whose passes wait on one another; given: the x faces
// with the carried z-face speeds
cudaError_t launch_carried(const astro::FaceArgs& a, bool given, int sms, void (*launched)(cudaStream_t),
                           cudaStream_t s);

}  // namespace astro_face32
