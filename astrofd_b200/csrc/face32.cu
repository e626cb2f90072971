// face32.cu -- the float32 face passes of the mixed-precision path: one thread
// per face and direction over the float32 copy of the primitives, and the
// float64 recomputation of the faces that overflow float32.
#include "face32.cuh"

using namespace astro;

namespace astro_face32 {
namespace {

// first place of this pass in the list of faces to recompute: behind the faces that the
// passes before it (complete by now: one stream) have counted
__device__ __forceinline__ size_t fix_base(const FaceArgs& a) {
    return (size_t)a.fix_count[-1] + a.fix_count[-2];
}

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
            const size_t slot = fix_base(a) + atomicAdd(a.fix_count, 1u);
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
// failed than the list has room for (the counter keeps counting past it), the
// pass's part of it is incomplete: every face of the pass is then checked and the
// non-finite ones are recomputed, so no float32 failure is left in place.
template <int PHYS, int RECON, int RIEMANN, bool GIVEN, int DIR>
__device__ __forceinline__ void fix_pass(const FaceArgs& a) {
    constexpr int NM = PHYS == ASTRO_SRHD ? 5 : 9;
    const unsigned cnt = *a.fix_count;
    const size_t base = fix_base(a);
    if (base + cnt <= a.fix_cap) {
        for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < cnt;
             q += gridDim.x * blockDim.x) {
            const long t = a.fix_list[base + q];
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

template <int PHYS, int RECON, int RIEMANN, bool GIVEN, int DIR>
__global__ void __launch_bounds__(128) k_face_fix(const __grid_constant__ FaceArgs a) {
    fix_pass<PHYS, RECON, RIEMANN, GIVEN, DIR>(a);
}

// all three directions' lists in one launch (blockIdx.y)
struct FaceArgs3 {
    FaceArgs d[3];
};
template <int PHYS, int RECON, int RIEMANN>
__global__ void __launch_bounds__(128) k_face_fix3(const __grid_constant__ FaceArgs3 a) {
    if (blockIdx.y == 0) fix_pass<PHYS, RECON, RIEMANN, false, 0>(a.d[0]);
    else if (blockIdx.y == 1) fix_pass<PHYS, RECON, RIEMANN, false, 1>(a.d[1]);
    else fix_pass<PHYS, RECON, RIEMANN, false, 2>(a.d[2]);
}

dim3 face_grid(const FaceArgs& a) {
    const unsigned plane = (unsigned)a.ext[1] * (unsigned)a.ext[2];
    return dim3((plane + 127) / 128, (unsigned)(a.ext[0] < 65535 ? a.ext[0] : 65535));
}

// an empty cell range in any direction: no faces (checked per extent, since two
// negative extents would give a positive product)
bool empty(const FaceArgs& a) { return a.ext[0] <= 0 || a.ext[1] <= 0 || a.ext[2] <= 0; }

// The fix-up counters start every pass at zero (the workspace, or the shared
// static scratch, holds the previous pass's count).
//
// one direction and its listed faces, for the carried order of passes
template <int RE, int RI>
struct OnePass {
    static cudaError_t run(const FaceArgs& a, bool given, int sms, cudaStream_t s) {
        constexpr int PH = ASTRO_RMHD;
        const dim3 fgrd(sms * 4), grd = face_grid(a);
        const cudaError_t e = cudaMemsetAsync(a.fix_count - 2, 0, 3 * sizeof(unsigned), s);
        if (e != cudaSuccess) return e;
        if (given) {
            k_face<PH, RE, RI, true, 0><<<grd, 128, 0, s>>>(a);
            k_face_fix<PH, RE, RI, true, 0><<<fgrd, 128, 0, s>>>(a);
        } else if (a.dir == 0) {
            k_face<PH, RE, RI, false, 0><<<grd, 128, 0, s>>>(a);
            k_face_fix<PH, RE, RI, false, 0><<<fgrd, 128, 0, s>>>(a);
        } else if (a.dir == 1) {
            k_face<PH, RE, RI, false, 1><<<grd, 128, 0, s>>>(a);
            k_face_fix<PH, RE, RI, false, 1><<<fgrd, 128, 0, s>>>(a);
        } else {
            k_face<PH, RE, RI, false, 2><<<grd, 128, 0, s>>>(a);
            k_face_fix<PH, RE, RI, false, 2><<<fgrd, 128, 0, s>>>(a);
        }
        return cudaGetLastError();
    }
};

// The three directions are independent: their listed faces are recomputed by one
// launch behind them and one clear precedes them, 5 launches instead of 9
// (SSPRK3 step of a 75 x 130 x 121 slab 1314 -> 1276 us).
template <int PH, int RE, int RI>
cudaError_t run_all(const FaceArgs3& a, int sms, void (*launched)(cudaStream_t), cudaStream_t s) {
    if (!empty(a.d[2])) {
        k_face<PH, RE, RI, false, 2><<<face_grid(a.d[2]), 128, 0, s>>>(a.d[2]);
        launched(s);
    }
    if (!empty(a.d[0])) {
        k_face<PH, RE, RI, false, 0><<<face_grid(a.d[0]), 128, 0, s>>>(a.d[0]);
        launched(s);
    }
    if (!empty(a.d[1])) k_face<PH, RE, RI, false, 1><<<face_grid(a.d[1]), 128, 0, s>>>(a.d[1]);
    k_face_fix3<PH, RE, RI><<<dim3(sms, 3), 128, 0, s>>>(a);
    launched(s);
    return cudaGetLastError();
}

template <int PH, int RE>
cudaError_t run_riemann(const FaceArgs3& a, int sms, void (*launched)(cudaStream_t), cudaStream_t s) {
    const int ri = a.d[0].p.riemann;
    if constexpr (PH == ASTRO_RMHD)
        if (ri == 2) return run_all<PH, RE, 2>(a, sms, launched, s);
    return ri == 1 ? run_all<PH, RE, 1>(a, sms, launched, s) : run_all<PH, RE, 0>(a, sms, launched, s);
}

}  // namespace

cudaError_t launch_carried(const FaceArgs& a, bool given, int sms, void (*launched)(cudaStream_t),
                           cudaStream_t s) {
    if (empty(a)) return cudaSuccess;
    const int ri = a.p.riemann;
    cudaError_t e;
    if (a.p.recon == ASTRO_RECON_PPM)
        e = ri == 2 ? OnePass<1, 2>::run(a, given, sms, s)
                    : (ri == 1 ? OnePass<1, 1>::run(a, given, sms, s) : OnePass<1, 0>::run(a, given, sms, s));
    else
        e = ri == 2 ? OnePass<2, 2>::run(a, given, sms, s)
                    : (ri == 1 ? OnePass<2, 1>::run(a, given, sms, s) : OnePass<2, 0>::run(a, given, sms, s));
    if (e == cudaSuccess) launched(s);
    return e;
}

cudaError_t launch_all(const FaceArgs* dirs, int sms, void (*launched)(cudaStream_t), cudaStream_t s) {
    // one list for the three passes in the order they run (z, x, y), the counters next to
    // each other: a third of it for each left one direction alone a rescan of its
    // whole pass at a third of the faces that it had room for
    FaceArgs3 a;
    const int order[3] = {1, 2, 0};
    for (int d = 0; d < 3; ++d) {
        a.d[d] = dirs[d];
        a.d[d].fix_count = dirs[0].fix_count + order[d];
    }
    if (empty(a.d[0]) && empty(a.d[1]) && empty(a.d[2])) return cudaSuccess;
    const cudaError_t e = cudaMemsetAsync(dirs[0].fix_count - 2, 0, 5 * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    const AstroParams& p = a.d[0].p;
    if (p.physics == ASTRO_SRHD)
        return p.recon == 0 ? run_riemann<ASTRO_SRHD, 0>(a, sms, launched, s)
                            : (p.recon == 1 ? run_riemann<ASTRO_SRHD, 1>(a, sms, launched, s)
                                            : run_riemann<ASTRO_SRHD, 2>(a, sms, launched, s));
    return p.recon == 0 ? run_riemann<ASTRO_RMHD, 0>(a, sms, launched, s)
                        : (p.recon == 1 ? run_riemann<ASTRO_RMHD, 1>(a, sms, launched, s)
                                        : run_riemann<ASTRO_RMHD, 2>(a, sms, launched, s));
}

}  // namespace astro_face32
