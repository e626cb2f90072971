// face.cuh -- one cell face: arguments of the face passes and the general
// per-face evaluation (reconstruct, floor, p2c, flux, speeds, Riemann) in the
// reference's operation order, shared by kernels.cu and face64.cu.
#pragma once
#include <cuda_runtime.h>

#include "physics.cuh"

namespace astro {

struct Bounds {
    int lo, hi[3];  // cells updated: [lo, hi[d]) per dimension
};

struct FaceArgs {
    const double* pr;
    const float* prf;    // float32 copy of the nm primitives (float32 passes)
    int nx, ny, nz;
    int dir;
    int org[3], ext[3];  // first cell and extents of the face block
    Bounds b;
    void* F;             // R[nm][nc]
    void* aux;           // R[4][nc]: sL, sR, vL, vR (or null)
    void* speeds_out;    // R[2][nc]: sL, sR (z faces, carried mode) or null
    const void* carried; // R[2][nc]: z-face speeds read by the carried x faces
    int ndiss;           // SRHD Israel-Stewart blocks: dissipation fluxes per face
    AstroParams p;
    // float32 passes: faces whose float32 result is not finite are listed here
    // and recomputed in float64 by k_face_fix.  The two words in front of the count
    // are those of the passes whose faces stand before this one's in the list, or zero
    unsigned* fix_count;
    unsigned* fix_list;
    unsigned fix_cap;
};

// One face: reconstruct, floor, p2c, flux, speeds, Riemann in arithmetic R,
// stored as RS.  Returns false when the stored flux or speeds are not finite.
template <int PHYS, int RECON, int RIEMANN, typename R, typename RS, bool GIVEN, int DIR>
__device__ __forceinline__ bool face_at(const FaceArgs& a, int i, int j, int k) {
    constexpr int NM = PHYS == ASTRO_SRHD ? 5 : 9;
    const size_t nc = (size_t)a.nx * a.ny * a.nz;
    const size_t cell = ((size_t)i * a.ny + j) * a.nz + k;
    const long stride = DIR == 0 ? (long)a.ny * a.nz : (DIR == 1 ? (long)a.nz : 1L);
    const Phys<R> P = Phys<R>::from(a.p);

    R qL[NM], qR[NM];
    constexpr int o0 = RECON == ASTRO_RECON_MUSCL ? -2 : -3;
    constexpr int o1 = RECON == ASTRO_RECON_MUSCL ? 1 : 2;
#pragma unroll
    for (int v = 0; v < NM; ++v) {
        R st[6];
        if constexpr (sizeof(R) == 4) {
            // the float32 copy: one conversion per cell and stage instead of
            // one per stencil use
            const float* base = a.prf + (size_t)v * nc + cell;
#pragma unroll
            for (int o = o0; o <= o1; ++o) st[o + 3] = __ldg(base + o * stride);
        } else {
            const double* base = a.pr + (size_t)v * nc + cell;
#pragma unroll
            for (int o = o0; o <= o1; ++o) st[o + 3] = (R)__ldg(base + o * stride);
        }
        recon_face<RECON>(st, a.p.limiter, qL[v], qR[v]);
    }
    R F[NM];
    R sL = R(-1), sR = R(1);
    if (GIVEN) {
        // previous cell of the reference's i-j-k loop, whose z-low face speeds
        // are still in (sL, sR) when this cell's x-low face is evaluated
        int pi = i, pj = j, pk = k;
        bool first = false;
        if (k > a.b.lo) pk = k - 1;
        else if (j > a.b.lo) { pj = j - 1; pk = a.b.hi[2] - 1; }
        else if (i > a.b.lo) { pi = i - 1; pj = a.b.hi[1] - 1; pk = a.b.hi[2] - 1; }
        else first = true;
        if (!first) {
            const RS* S = (const RS*)a.carried;
            const size_t pc = ((size_t)pi * a.ny + pj) * a.nz + pk;
            sL = (R)S[pc];
            sR = (R)S[nc + pc];
        }
    }
    if (PHYS == ASTRO_SRHD) {
        if (RECON == ASTRO_RECON_MUSCL && a.p.passive_offset > 5) {
            // add_pi_lr (srhd_core.py:394-398): the cells' bulk pressure on
            // the reconstructed face pressures, before the floor
            qL[4] += (R)__ldg(a.pr + 5 * nc + cell - stride);
            qR[4] += (R)__ldg(a.pr + 5 * nc + cell);
        }
        if (a.ndiss > 0) {
            R isL[10], isR[10];
#pragma unroll
            for (int m = 0; m < 10; ++m) {
                isL[m] = (R)__ldg(a.pr + (size_t)(5 + m) * nc + cell - stride);
                isR[m] = (R)__ldg(a.pr + (size_t)(5 + m) * nc + cell);
            }
            s_face<RIEMANN>(P, DIR, qL, qR, F, sL, sR, a.ndiss, isL, isR);
        } else {
            s_face<RIEMANN>(P, DIR, qL, qR, F, sL, sR);
        }
    } else {
        r_face<RIEMANN, RECON == ASTRO_RECON_MUSCL, GIVEN>(P, DIR, qL, qR, F, sL, sR);
    }
    RS* Fo = (RS*)a.F;
    bool finite = true;
#pragma unroll
    for (int v = 0; v < NM; ++v) {
        const RS f = (RS)F[v];
        finite &= isfinite(f);
        Fo[(size_t)v * nc + cell] = f;
    }
    finite &= isfinite((RS)sL) && isfinite((RS)sR);
    if (a.aux) {
        RS* A = (RS*)a.aux;
        A[cell] = (RS)sL;
        A[nc + cell] = (RS)sR;
        A[2 * nc + cell] = (RS)qL[1 + DIR];
        A[3 * nc + cell] = (RS)qR[1 + DIR];
    }
    if (a.speeds_out) {
        RS* S = (RS*)a.speeds_out;
        S[cell] = (RS)sL;
        S[nc + cell] = (RS)sR;
    }
    return finite;
}

}  // namespace astro
