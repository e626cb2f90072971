// face64.cu -- the float64 face passes of the split stages and right-hand
// sides.
//
// Reconstruction is cell-centred: both face values of a cell come from one
// evaluation (the WENO5 smoothness indicators, the PPM parabola and the MUSCL
// slope of a cell serve its low and its high face), where an evaluation per
// face (face_at) makes each of them twice.  x and y: a thread walks along the
// direction, so the high-face values of one cell are the left states of the
// next face.  z: the 32 lanes of a warp hold 32 neighbouring cells and hand
// their high-face values to the next lane (31 faces per warp).  Both pass
// them through shared memory, [variable][thread], which keeps the 18 registers
// free while the Riemann problem is solved.
//
// Divisions: the arithmetic type is fd (one reciprocal per shared
// denominator); WENO5 takes one per face value, its weights written over a
// common denominator.  A face with a result that is not finite, or whose WENO5
// denominators leave [0, 1e300], is evaluated again by the general face_at in
// float64 with IEEE divisions, so overflows end as they do there.
//
// The reference's carried x faces (core/rmhd_core.py:1445,1468) differ from the
// ordinary ones in the wave speeds alone, so both fluxes are formed from one pair of
// states instead of by two passes (HLLE; "hlld" with carried speeds is Args::exact).
//
// Bound: the float64 pipe (about 850 float64 operations per RMHD WENO5 face) at 16
// warps per SM, 128 registers.  One stage's faces of 134^3 cells, per-face passes with
// IEEE divisions against this kernel: RMHD WENO5 HLLE with carried x faces 2175 us
// and 597 us, "hlld" with its own speeds 1819 us and 558 us, MUSCL "hlld" 953 us and
// 722 us, SRHD PPM HLLC 370 us and 220 us.  (RMHD at 3 blocks per SM, which spill
// nothing, 4 % slower; at 5, 1 %.)
//
// Schemes that amplify last bits (exact_bits in kernels.cu) keep the general per-face
// evaluation, k_face_general.
#include "face64.cuh"

#include <stdint.h>
#include <string.h>

using namespace astro;

namespace astro_face64 {
namespace {

constexpr int T = 128;  // threads per block

// face_at as a call: rare, so it must not cost the caller registers
template <int PHYS, int RECON, int RIEMANN, bool GIVEN, int DIR>
__device__ __noinline__ void general_face(const Args& a, int i, int j, int k) {
    FaceArgs f;
    f.pr = a.pr;
    f.nx = a.nx; f.ny = a.ny; f.nz = a.nz;
    f.b = a.b;
    f.F = GIVEN ? a.FxC : a.F[DIR];
    f.aux = GIVEN ? nullptr : a.aux[DIR];
    f.speeds_out = DIR == 2 ? a.speeds_out : nullptr;
    f.carried = a.carried;
    f.ndiss = a.ndiss;
    f.p = a.p;
    face_at<PHYS, RECON, RIEMANN, double, double, GIVEN, DIR>(f, i, j, k);
}

// Both WENO5 face values of the cell with stencil q[0..4]: lo is the reference's
// right-biased value at its low face, hi the left-biased one at its high face.
// The smoothness indicators serve both: with the differences d_k of neighbouring
// cells the second differences are t and half the first-derivative terms h, so
// IS_k = 13/12 t^2 + h^2.  With D_k = (eps + IS_k)^2 the weights g_k / D_k / sum
// are g_k prod(D_other) / sum: one reciprocal per face value instead of six
// divisions.  Polynomials and their weighted sum follow the reference (in place of the
// middle polynomial plus weighted differences, which rounds less still, but moves
// floored cells by 4e-8 from the reference, whose roundings they amplify).  The weights'
// distance from 1, that is what the shared denominator and its reciprocal were rounded
// by, corrects the sum; as a factor, so that a polynomial across a jump does not come
// back with the last bit of 1.  L2 distance of right-hand sides of a 40 x 37 x 45 jet from
// 80-bit arithmetic, x and y momentum: 1.9e-14 and 1.5e-14; without that factor 3.7e-14
// and 3.3e-14; with the reference's six divisions 2.7e-14 and 1.7e-14.  It costs no time
// (128^3 RMHD HLLE 601 us per stage with it, 604 without; SRHD HLLC 318 and 303).
__device__ __forceinline__ void weno5_cell(const double* q, double& lo, double& hi, bool& wide) {
    const double a = q[0], b = q[1], c = q[2], d = q[3], e = q[4];
    const double d0 = b - a, d1 = c - b, d2 = d - c, d3 = e - d;
    const double t0 = d1 - d0, t1 = d2 - d1, t2 = d3 - d2;
    const double h0 = fma(0.5, t0, d1), h1 = 0.5 * (d1 + d2), h2 = fma(0.5, t2, -d2);
    constexpr double k = 13.0 / 12.0, eps = 1e-12;
    const double e0 = fma(k * t0, t0, fma(h0, h0, eps));
    const double e1 = fma(k * t1, t1, fma(h1, h1, eps));
    const double e2 = fma(k * t2, t2, fma(h2, h2, eps));
    const double D0 = e0 * e0, D1 = e1 * e1, D2 = e2 * e2;
    // weights 1, 6, 3 (the reference's 0.1, 0.6, 0.3 times ten), the outer two
    // exchanged between the faces
    const double P12 = D1 * D2, P02 = 6.0 * (D0 * D2), P01 = D0 * D1;
    const double T12 = 3.0 * P12, T01 = 3.0 * P01;
    const double denh = P12 + P02 + T01, denl = P01 + P02 + T12;
    // 1e300 by exponent (the sign is clear; infinities and NaN are above)
    wide |= __double2hiint(denh) >= 0x7e37e43c || __double2hiint(denl) >= 0x7e37e43c;
    const double rh = rcp_(fd(denh)).v, rl = rcp_(fd(denl)).v;
    const double c1 = (5.0 / 6.0) * c, c2 = (1.0 / 3.0) * c;  // of both faces
    const double h0q = fma(11.0 / 6.0, c, fma(-7.0 / 6.0, b, (1.0 / 3.0) * a));
    const double h1q = fma(1.0 / 3.0, d, fma(-1.0 / 6.0, b, c1));
    const double h2q = fma(-1.0 / 6.0, e, fma(5.0 / 6.0, d, c2));
    const double l0q = fma(11.0 / 6.0, c, fma(-7.0 / 6.0, d, (1.0 / 3.0) * e));
    const double l1q = fma(1.0 / 3.0, b, fma(-1.0 / 6.0, d, c1));
    const double l2q = fma(-1.0 / 6.0, a, fma(5.0 / 6.0, b, c2));
    // rounded before their distance from 1 is taken, not fused into it
    const double h0w = __dmul_rn(P12, rh), h1w = __dmul_rn(P02, rh), h2w = __dmul_rn(T01, rh);
    const double l0w = __dmul_rn(P01, rl), l1w = __dmul_rn(P02, rl), l2w = __dmul_rn(T12, rl);
    hi = fma(h2w, h2q, fma(h1w, h1q, h0w * h0q));
    lo = fma(l2w, l2q, fma(l1w, l1q, l0w * l0q));
    hi = fma(((1.0 - h0w) - h1w) - h2w, hi, hi);
    lo = fma(((1.0 - l0w) - l1w) - l2w, lo, lo);
}

template <int RECON>
__device__ __forceinline__ void recon_cell(const double* q, int lim, double& lo, double& hi, bool& wide) {
    if constexpr (RECON == ASTRO_RECON_MUSCL) {
        const double s = limiter(lim, fd(q[2] - q[1]), fd(q[3] - q[2])).v;
        // van Leer's denominator beyond the reciprocal's range
        wide |= lim == ASTRO_LIM_VANLEER && beyond(fd(q[3] - q[1]));
        lo = q[2] - 0.5 * s;
        hi = q[2] + 0.5 * s;
    } else if constexpr (RECON == ASTRO_RECON_PPM) {
        ppm(q[0], q[1], q[2], q[3], q[4], lo, hi);
    } else {
        weno5_cell(q, lo, hi, wide);
    }
}

// The cell (i, j, k): its face values, and the flux through its low face in
// direction DIR (when `face`) from the left states in sh[v * T + thread], which
// its own high-face values replace.  wide_left: whether the left states'
// reconstruction left its range; the cell's own on return.
template <int PHYS, int RECON, int RIEMANN, int DIR>
__device__ __forceinline__ void cell_and_face(const Args& a, double* sh, int i, int j, int k, bool face,
                                              bool& wide_left) {
    constexpr int NM = PHYS == ASTRO_SRHD ? 5 : 9;
    const int t = threadIdx.x;
    const size_t nc = (size_t)a.nx * a.ny * a.nz;
    const size_t cell = ((size_t)i * a.ny + j) * a.nz + k;
    const long stride = DIR == 0 ? (long)a.ny * a.nz : (DIR == 1 ? (long)a.nz : 1L);
    constexpr int w = RECON == ASTRO_RECON_MUSCL ? 1 : 2;
    bool wide = false;
    fd qL[NM], qR[NM];
#pragma unroll
    for (int v = 0; v < NM; ++v) {
        double q[5], lo, hi;
        const double* base = a.pr + (size_t)v * nc + cell;
#pragma unroll
        for (int o = -w; o <= w; ++o) q[o + 2] = __ldg(base + o * stride);
        recon_cell<RECON>(q, a.p.limiter, lo, hi, wide);
        qR[v] = fd(lo);
        if constexpr (DIR != 2) qL[v] = fd(sh[v * T + t]);
        sh[v * T + t] = hi;
    }
    if constexpr (DIR == 2) {
        // the lane below holds the cell below
        wide_left = __any_sync(0xffffffffu, wide);
        __syncwarp();
#pragma unroll
        for (int v = 0; v < NM; ++v) qL[v] = fd(sh[v * T + t - (t & 31 ? 1 : 0)]);
    }
    const bool wide_here = wide;
    wide |= wide_left;
    wide_left = wide_here;
    if (!face) return;
    const Phys<fd> P = Phys<fd>::from(a.p);
    fd F[NM], sL, sR;
    double* Fo = a.F[DIR];
    bool ok = !wide;
    if constexpr (PHYS == ASTRO_SRHD) {
        if (RECON == ASTRO_RECON_MUSCL && a.p.passive_offset > 5) {
            // add_pi_lr (srhd_core.py:394-398), as in face_at
            qL[4] += fd(__ldg(a.pr + 5 * nc + cell - stride));
            qR[4] += fd(__ldg(a.pr + 5 * nc + cell));
        }
        if (a.ndiss > 0) {
            fd isL[10], isR[10];
#pragma unroll
            for (int m = 0; m < 10; ++m) {
                isL[m] = fd(__ldg(a.pr + (size_t)(5 + m) * nc + cell - stride));
                isR[m] = fd(__ldg(a.pr + (size_t)(5 + m) * nc + cell));
            }
            s_face<RIEMANN>(P, DIR, qL, qR, F, sL, sR, a.ndiss, isL, isR);
        } else {
            s_face<RIEMANN>(P, DIR, qL, qR, F, sL, sR);
        }
    } else {
        constexpr bool OVR = RECON == ASTRO_RECON_MUSCL;
        fd UL[9], UR[9], FL[9], FR[9];
        r_face_states(P, DIR, qL, qR, UL, UR, FL, FR, sL, sR);
        r_riemann<RIEMANN, OVR>(P, DIR, qL, qR, UL, UR, FL, FR, sL, sR, F);
        if (DIR == 0 && !OVR && a.FxC && i < a.b.hi[0]) {
            // the x-low face of an updated cell with the z-face speeds left
            // over from the previous cell of the reference's i-j-k loop
            double cL = -1.0, cR = 1.0;
            int pi = i, pj = j, pk = k - 1;
            if (k == a.b.lo) {
                pk = a.b.hi[2] - 1;
                if (j > a.b.lo) pj = j - 1;
                else { pj = a.b.hi[1] - 1; pi = i - 1; }
            }
            if (pi >= a.b.lo) {
                const size_t pc = ((size_t)pi * a.ny + pj) * a.nz + pk;
                cL = a.carried[pc];
                cR = a.carried[nc + pc];
            }
            fd G[9];
            r_riemann<RIEMANN, OVR>(P, 0, qL, qR, UL, UR, FL, FR, fd(cL), fd(cR), G);
            bool okc = !wide && isfinite(sL.v);
#pragma unroll
            for (int v = 0; v < 9; ++v) {
                okc &= isfinite(G[v].v);
                a.FxC[(size_t)v * nc + cell] = G[v].v;
            }
            if (!okc) general_face<PHYS, RECON, RIEMANN, DIR == 0 && !OVR, 0>(a, i, j, k);
        }
    }
#pragma unroll
    for (int v = 0; v < NM; ++v) {
        ok &= isfinite(F[v].v);
        Fo[(size_t)v * nc + cell] = F[v].v;
    }
    ok &= isfinite(sL.v) && isfinite(sR.v);
    if (a.aux[DIR]) {
        double* A = a.aux[DIR];
        A[cell] = sL.v;
        A[nc + cell] = sR.v;
        A[2 * nc + cell] = qL[1 + DIR].v;
        A[3 * nc + cell] = qR[1 + DIR].v;
    }
    if (DIR == 2 && a.speeds_out) {
        a.speeds_out[cell] = sL.v;
        a.speeds_out[nc + cell] = sR.v;
    }
    if (!ok) general_face<PHYS, RECON, RIEMANN, false, DIR>(a, i, j, k);
}

// threads of direction DIR (0, 1): the plane across it, times segments of
// a.seg[DIR] faces along it
template <int PHYS, int RECON, int RIEMANN, int DIR>
__device__ __forceinline__ void walk(const Args& a, double* sh, unsigned block) {
    const int lo = a.b.lo;
    const unsigned e2 = (unsigned)(a.b.hi[2] - lo);
    const unsigned eo = (unsigned)(a.b.hi[DIR == 0 ? 1 : 0] - lo);
    const unsigned plane = e2 * eo;
    const unsigned per = (plane + T - 1) / T;  // blocks per segment
    const unsigned sg = block / per, tp = (block - sg * per) * T + threadIdx.x;
    if (tp >= plane) return;
    const int k = lo + (int)(tp % e2), o = lo + (int)(tp / e2);
    const int f0 = lo + (int)sg * a.seg[DIR];
    int f1 = f0 + a.seg[DIR];
    if (f1 > a.b.hi[DIR] + 1) f1 = a.b.hi[DIR] + 1;
    // the first turn only makes the left states of face f0
    bool wide = false;
    for (int f = f0 - 1; f < f1; ++f)
        cell_and_face<PHYS, RECON, RIEMANN, DIR>(a, sh, DIR == 0 ? f : o, DIR == 0 ? o : f, k, f >= f0,
                                                 wide);
}

// Blocks per SM: SRHD 8 (64 registers, which spill 440 to 520 bytes a thread, most of
// them for the dissipation branch: 4 blocks at 128 take 723 against 683 us for a
// 128^3 PPM step's faces, 113 against 89 us for a 64^3 MUSCL one's; 5 to 7 were not
// compared); RMHD 4 (128 registers, at most 70 bytes spilled).
template <int PHYS, int RECON, int RIEMANN>
__global__ void __launch_bounds__(T, PHYS == ASTRO_SRHD ? 8 : 4)
    k_face64(const __grid_constant__ Args a) {
    constexpr int NM = PHYS == ASTRO_SRHD ? 5 : 9;
    __shared__ double sh[NM * T];
    // the walks first: the short z blocks then fill the launch's end
    if (blockIdx.x < (unsigned)a.blocks_x) {
        walk<PHYS, RECON, RIEMANN, 0>(a, sh, blockIdx.x);
    } else if (blockIdx.x < (unsigned)(a.blocks_x + a.blocks_y)) {
        walk<PHYS, RECON, RIEMANN, 1>(a, sh, blockIdx.x - a.blocks_x);
    } else {
        // one warp per 31 z faces of a row: lane 0 only makes left states
        const int lo = a.b.lo, faces = a.b.hi[2] - lo + 1;
        const unsigned per = (unsigned)(faces + 30) / 31;
        const unsigned wp = (blockIdx.x - a.blocks_x - a.blocks_y) * (T / 32) + threadIdx.x / 32;
        const unsigned r = wp / per, ey = (unsigned)(a.b.hi[1] - lo);
        const int i = lo + (int)(r / ey), j = lo + (int)(r % ey);
        if (i >= a.b.hi[0]) return;
        const int k = lo + (int)(wp % per) * 31 + (int)(threadIdx.x & 31) - 1;
        // lanes past the last face repeat its cell, without a face
        bool wide = false;
        cell_and_face<PHYS, RECON, RIEMANN, 2>(a, sh, i, j, k < a.b.hi[2] ? k : a.b.hi[2],
                                               (threadIdx.x & 31) > 0 && k <= a.b.hi[2], wide);
    }
}

// One thread per face of one direction by the general evaluation, for steps that
// depend on its last bit (Args::exact).  Faces of a 128^3 WENO5 hlld step 6.9 ms
// against 1.9 ms above; a launch bound, a quotient of another form or both x fluxes
// in one kernel change how the compiler fuses multiplications and additions, and
// with it last bits.
template <int RECON, int RIEMANN, bool GIVEN, int DIR>
__global__ void __launch_bounds__(128) k_face_general(FaceArgs a) {
    // grid: x over the (j, k) plane of the face block, y over its x layers;
    // one 32-bit split of the in-plane index per thread
    const unsigned e2 = (unsigned)a.ext[2];
    const unsigned plane = (unsigned)a.ext[1] * e2;
    const unsigned tp = blockIdx.x * blockDim.x + threadIdx.x;
    if (tp >= plane) return;
    const int c = (int)(tp % e2), bb = (int)(tp / e2);
    for (int aa = blockIdx.y; aa < a.ext[0]; aa += gridDim.y) {
        const int i = a.org[0] + aa, j = a.org[1] + bb, k = a.org[2] + c;
        face_at<ASTRO_RMHD, RECON, RIEMANN, double, double, GIVEN, DIR>(a, i, j, k);
    }
}

// z (with the speeds the carried x faces read), x, carried x, y: of those, the ones
// this launch has buffers for
template <int RECON, int RIEMANN>
cudaError_t general_passes(const Args& a, void (*launched)(cudaStream_t), cudaStream_t s) {
    for (int pass = 0; pass < 4; ++pass) {
        const int d = pass == 0 ? 2 : (pass == 3 ? 1 : 0);
        const bool given = pass == 2;
        if (given ? !a.FxC : !a.F[d]) continue;
        FaceArgs f;
        memset(&f, 0, sizeof(f));
        f.pr = a.pr; f.nx = a.nx; f.ny = a.ny; f.nz = a.nz; f.dir = d; f.b = a.b; f.p = a.p;
        for (int e = 0; e < 3; ++e) {
            f.org[e] = a.b.lo;
            f.ext[e] = a.b.hi[e] - a.b.lo + (e == d && !given ? 1 : 0);
        }
        f.F = given ? a.FxC : a.F[d];
        f.aux = given ? nullptr : a.aux[d];
        f.speeds_out = d == 2 ? a.speeds_out : nullptr;
        f.carried = a.carried;
        f.ndiss = a.ndiss;
        const unsigned plane = (unsigned)f.ext[1] * (unsigned)f.ext[2];
        const dim3 grd((plane + 127) / 128, (unsigned)(f.ext[0] < 65535 ? f.ext[0] : 65535));
        if (given) {
            if constexpr (RECON != ASTRO_RECON_MUSCL)
                k_face_general<RECON, RIEMANN, true, 0><<<grd, 128, 0, s>>>(f);
        } else if (d == 0) k_face_general<RECON, RIEMANN, false, 0><<<grd, 128, 0, s>>>(f);
        else if (d == 1) k_face_general<RECON, RIEMANN, false, 1><<<grd, 128, 0, s>>>(f);
        else k_face_general<RECON, RIEMANN, false, 2><<<grd, 128, 0, s>>>(f);
        launched(s);
    }
    return cudaGetLastError();
}

template <int PH, int RE>
void launch_riemann(const Args& a, unsigned blocks, cudaStream_t s) {
    // "hlld_full" is always Args::exact
    if (a.p.riemann == 0) k_face64<PH, RE, 0><<<blocks, T, 0, s>>>(a);
    else k_face64<PH, RE, 1><<<blocks, T, 0, s>>>(a);
}

}  // namespace

cudaError_t launch(Args a, int sms, void (*launched)(cudaStream_t), cudaStream_t s) {
    const long e[3] = {a.b.hi[0] - a.b.lo, a.b.hi[1] - a.b.lo, a.b.hi[2] - a.b.lo};
    if (e[0] <= 0 || e[1] <= 0 || e[2] <= 0) return cudaSuccess;
    if (a.exact) {
        const bool full = a.p.riemann == ASTRO_RIEMANN_HLLD_FULL;
        if (a.p.recon == ASTRO_RECON_MUSCL) return general_passes<0, 2>(a, launched, s);
        if (a.p.recon == ASTRO_RECON_PPM)
            return full ? general_passes<1, 2>(a, launched, s) : general_passes<1, 1>(a, launched, s);
        return full ? general_passes<2, 2>(a, launched, s) : general_passes<2, 1>(a, launched, s);
    }
    long blocks[3] = {0, 0, 0};
    if (a.F[2]) blocks[2] = (e[0] * e[1] * ((e[2] + 1 + 30) / 31) + T / 32 - 1) / (T / 32);
    const long resident = (long)sms * (a.p.physics == ASTRO_SRHD ? 8 : 4);
    for (int d = 0; d < 2; ++d) {
        if (!a.F[d]) continue;
        // A longer walk repeats fewer reconstructions at its start (about 0.6 of a
        // turn per segment); more segments give more blocks.  With z blocks behind
        // them the walks are as long as leaves one block for each place on the
        // device, up to 16 faces; alone, of the lengths up to 32 the one that needs
        // the fewest turns with whole waves of blocks (128^3 RMHD x faces: 129 as 9
        // segments of 15 are 2 waves, as 19 of 7 they were 5).  Segments of equal
        // length.  Against 4 waves of walks with z first, with "hlld" and carried x
        // faces, which then were this kernel's too: PPM faces of 90 x 61 x 103 cells 174
        // -> 151 us, WENO5 of 72^3 163 -> 136 us per stage (HLLE now 134 and 133 us); SRHD
        // 128^3 PPM 228 -> 220 us.
        const long per = (e[1 - d] * e[2] + T - 1) / T, faces = e[d] + 1;
        long seg = 1;
        if (a.F[2]) {
            seg = per * faces / resident;
            seg = seg < 1 ? 1 : (seg > 16 ? 16 : seg);
        } else {
            double best = 0.0;
            for (long s = 1; s <= 32 && s <= faces; ++s) {
                const long n = per * ((faces + s - 1) / s);
                const double cost = (double)((n + resident - 1) / resident) * ((double)s + 0.6);
                if (s == 1 || cost < best) {
                    best = cost;
                    seg = s;
                }
            }
        }
        const long nseg = (faces + seg - 1) / seg;
        a.seg[d] = (int)((faces + nseg - 1) / nseg);
        blocks[d] = per * ((faces + a.seg[d] - 1) / a.seg[d]);
    }
    a.blocks_x = (int)blocks[0];
    a.blocks_y = (int)blocks[1];
    const long total = blocks[0] + blocks[1] + blocks[2];
    if (total == 0) return cudaSuccess;
    if (total > 0x7fffffffL) return cudaErrorInvalidValue;
    const unsigned n = (unsigned)total;
    if (a.p.physics == ASTRO_SRHD) {
        if (a.p.recon == 0) launch_riemann<ASTRO_SRHD, 0>(a, n, s);
        else if (a.p.recon == 1) launch_riemann<ASTRO_SRHD, 1>(a, n, s);
        else launch_riemann<ASTRO_SRHD, 2>(a, n, s);
    } else {
        if (a.p.recon == 0) launch_riemann<ASTRO_RMHD, 0>(a, n, s);
        else if (a.p.recon == 1) launch_riemann<ASTRO_RMHD, 1>(a, n, s);
        else launch_riemann<ASTRO_RMHD, 2>(a, n, s);
    }
    launched(s);
    return cudaGetLastError();
}

}  // namespace astro_face64
