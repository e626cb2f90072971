// face64.cuh -- the float64 face passes (interface between face64.cu and
// kernels.cu; not part of the C ABI).
#pragma once
#include "face.cuh"

namespace astro_face64 {

// the faces of up to three directions of one block in one launch
struct Args {
    const double* pr;
    int nx, ny, nz;
    astro::Bounds b;     // updated cells; the faces on both sides of each
    double* F[3];        // fluxes per direction, [nm][nc]; null: not this launch
    double* aux[3];      // sL, sR, vL, vR per direction, or null
    double* speeds_out;  // z faces: sL, sR for the carried x faces, or null
    double* FxC;         // x faces: also the fluxes with the carried speeds, or null
    const double* carried;  // those speeds (an earlier launch's speeds_out)
    int ndiss;
    bool exact;          // the general evaluation, to its last bit (RMHD "hlld_full", and
                         // PPM and WENO5 with "hlld")
    AstroParams p;
    // set by launch(): thread blocks of x, y (z follow) and faces per thread
    int blocks_x, blocks_y, seg[2];
};

// launched: called after each kernel (the launch count and the kernel timing's events)
cudaError_t launch(Args a, int sms, void (*launched)(cudaStream_t), cudaStream_t s);

}  // namespace astro_face64
