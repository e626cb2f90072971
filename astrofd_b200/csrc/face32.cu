// face32.cu -- the float32 face passes of the mixed-precision path: one thread
// per face and direction over the float32 copy of the primitives, and the
// float64 recomputation of the faces that overflow float32.
#include "face32.cuh"

using namespace astro;

namespace astro_face32 {
namespace {

// float32 face pass of one direction (the float64 passes are face64.cu's)
template <int PHYS, int RECON, int RIEMANN, bool GIVEN, int DIR>
__global__ void __launch_bounds__(128) k_face(FaceArgs a) {
    // grid: x over the (j, k) plane of the face block, y over its x layers;
    // one 32-bit split of the in-plane index per thread
    const unsigned e2 = (unsigned)a.ext[2];
    const unsigned plane = (unsigned)a.ext[1] * e2;
    const unsigned tp = blockIdx.x * blockDim.x + threadIdx.x;
    if (tp >= plane) return;
    const int c = (int)(tp % e2), bb = (int)(tp / e2);
    for (int aa = blockIdx.y; aa < a.ext[0]; aa += gridDim.y) {
        const int i = a.org[0] + aa, j = a.org[1] + bb, k = a.org[2] + c;
        const bool ok = face_at<PHYS, RECON, RIEMANN, float, float, GIVEN, DIR>(a, i, j, k);
        if (!ok && a.fix_list) {
            const unsigned slot = atomicAdd(a.fix_count, 1u);
            if (slot < a.fix_cap) a.fix_list[slot] = (unsigned)aa * plane + tp;
        }
    }
}

// whether everything face_at stored for this face (fluxes, and the speeds
// and face velocities where the pass keeps them) is finite
template <int NM>
__device__ __forceinline__ bool face_stored_finite(const FaceArgs& a, size_t nc, size_t cell) {
    bool ok = true;
    const float* F = (const float*)a.F;
#pragma unroll
    for (int v = 0; v < NM; ++v) ok &= isfinite(F[(size_t)v * nc + cell]);
    if (a.aux) {
        const float* A = (const float*)a.aux;
#pragma unroll
        for (int m = 0; m < 4; ++m) ok &= isfinite(A[(size_t)m * nc + cell]);
    }
    if (a.speeds_out) {
        const float* S = (const float*)a.speeds_out;
        ok &= isfinite(S[cell]) && isfinite(S[nc + cell]);
    }
    return ok;
}

// float64 recomputation of the faces a float32 pass listed as non-finite
// (float32 overflows where float64 does not, e.g. squared WENO smoothness
// indicators of a state whose fields have grown past ~1e9).  If more faces
// failed than the list holds (the counter keeps counting past its capacity),
// the list is incomplete: every face of the pass is then checked and the
// non-finite ones are recomputed, so no float32 failure is left in place.
template <int PHYS, int RECON, int RIEMANN, bool GIVEN, int DIR>
__global__ void __launch_bounds__(128) k_face_fix(FaceArgs a) {
    constexpr int NM = PHYS == ASTRO_SRHD ? 5 : 9;
    const unsigned cnt = *a.fix_count;
    if (cnt <= a.fix_cap) {
        for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < cnt;
             q += gridDim.x * blockDim.x) {
            const long t = a.fix_list[q];
            const int c = (int)(t % a.ext[2]);
            const long r = t / a.ext[2];
            const int bb = (int)(r % a.ext[1]);
            const int aa = (int)(r / a.ext[1]);
            face_at<PHYS, RECON, RIEMANN, double, float, GIVEN, DIR>(a, a.org[0] + aa,
                                                                    a.org[1] + bb, a.org[2] + c);
        }
        return;
    }
    const size_t nc = (size_t)a.nx * a.ny * a.nz;
    const size_t plane = (size_t)a.ext[1] * a.ext[2];
    const size_t total = (size_t)a.ext[0] * plane;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total;
         q += (size_t)gridDim.x * blockDim.x) {
        const int aa = (int)(q / plane);
        const size_t tp = q % plane;
        const int bb = (int)(tp / a.ext[2]), c = (int)(tp % a.ext[2]);
        const int i = a.org[0] + aa, j = a.org[1] + bb, k = a.org[2] + c;
        const size_t cell = ((size_t)i * a.ny + j) * a.nz + k;
        if (!face_stored_finite<NM>(a, nc, cell))
            face_at<PHYS, RECON, RIEMANN, double, float, GIVEN, DIR>(a, i, j, k);
    }
}

// direction is a template parameter so the per-direction component indices
// fold to constants and the face state stays in registers
template <int PH, int RE, int RI>
cudaError_t launch_face_dir(const FaceArgs& a, bool given, dim3 grd, dim3 blk, cudaStream_t s) {
    const dim3 fgrd(148 * 4);
    // the fix-up counter starts every pass at zero (the workspace, or the
    // shared static scratch, holds the previous pass's count)
    const cudaError_t e = cudaMemsetAsync(a.fix_count, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    if constexpr (PH == ASTRO_RMHD && RE != ASTRO_RECON_MUSCL) {
        if (given) {
            k_face<PH, RE, RI, true, 0><<<grd, blk, 0, s>>>(a);
            k_face_fix<PH, RE, RI, true, 0><<<fgrd, blk, 0, s>>>(a);
            return cudaSuccess;
        }
    }
    if (a.dir == 0) {
        k_face<PH, RE, RI, false, 0><<<grd, blk, 0, s>>>(a);
        k_face_fix<PH, RE, RI, false, 0><<<fgrd, blk, 0, s>>>(a);
    } else if (a.dir == 1) {
        k_face<PH, RE, RI, false, 1><<<grd, blk, 0, s>>>(a);
        k_face_fix<PH, RE, RI, false, 1><<<fgrd, blk, 0, s>>>(a);
    } else {
        k_face<PH, RE, RI, false, 2><<<grd, blk, 0, s>>>(a);
        k_face_fix<PH, RE, RI, false, 2><<<fgrd, blk, 0, s>>>(a);
    }
    return cudaSuccess;
}

}  // namespace

cudaError_t launch(const FaceArgs& a, bool given, cudaStream_t s) {
    // an empty cell range in any direction: no faces (checked per extent,
    // since two negative extents would give a positive product)
    if (a.ext[0] <= 0 || a.ext[1] <= 0 || a.ext[2] <= 0) return cudaSuccess;
    const unsigned plane = (unsigned)a.ext[1] * (unsigned)a.ext[2];
    const dim3 blk(128), grd((plane + 127) / 128, (unsigned)(a.ext[0] < 65535 ? a.ext[0] : 65535));
    const AstroParams& p = a.p;
    cudaError_t me = cudaSuccess;
#define FACE(PH, RE, RI) me = launch_face_dir<PH, RE, RI>(a, given, grd, blk, s)
#define RECONS(PH, RI)                                                          \
    do {                                                                        \
        if (p.recon == 0) FACE(PH, 0, RI);                                      \
        else if (p.recon == 1) FACE(PH, 1, RI);                                 \
        else FACE(PH, 2, RI);                                                   \
    } while (0)
    if (p.physics == ASTRO_SRHD) {
        if (p.riemann == 1) RECONS(ASTRO_SRHD, 1);
        else RECONS(ASTRO_SRHD, 0);
    } else {
        if (p.riemann == 2) RECONS(ASTRO_RMHD, 2);
        else if (p.riemann == 1) RECONS(ASTRO_RMHD, 1);
        else RECONS(ASTRO_RMHD, 0);
    }
#undef RECONS
#undef FACE
    if (me != cudaSuccess) return me;
    return cudaGetLastError();
}

}  // namespace astro_face32
