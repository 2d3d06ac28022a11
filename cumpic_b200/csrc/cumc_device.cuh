// cumc_device.cuh — device-side data layout and per-cell arithmetic of the
// CUMC3D hot path on B200 (sm_100a).
//
// Layout in HBM: structure of arrays. Every field is one FP64 array over the
// ghosted box (-2:n+3)^3 with x fastest, so a warp reads 32 consecutive x
// cells (256 B) per variable. The reference keeps the 8 equations
// interleaved per cell (AoS, solver/setup.f90:257); the library transposes
// once at upload/download.
//
// Every arithmetic expression below keeps the operation order of the
// reference subroutine it cites; the parity build uses --fmad=false so that
// no multiply-add is contracted and the FP64 path reproduces the FP64 CPU
// restatement bit for bit.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "cumc_round.cuh"

namespace cumc {

constexpr int NG = 3;  // ghost layers (solver/definition.f90:54)

// Box geometry: strides of the ghosted SoA arrays.
struct Box {
    int nx, ny, nz;
    int SX, SY, SZ;  // nx+6, ny+6, nz+6
    const int* skip;  // device flag: when non-null and set, kernels return at once
                      // (the time loop has reached t_end inside a captured graph)
    __host__ __device__ __forceinline__ int idx(int j, int k, int l) const {
        return (j + 2) + SX * ((k + 2) + SY * (l + 2));
    }
    __host__ __device__ __forceinline__ long long count() const { return (long long)SX * SY * SZ; }
};

// Per-axis 1-D tables (pointers pre-offset so that t[i] is valid for
// i in -3..n+3). All values are computed on the host with the formulas of the
// reference so that the device reads the same doubles the reference would
// recompute inline.
struct AxisTabs {
    const double* f;    // face coordinate xF(i)                   (solver/coords.f90:24-32)
    const double* d;    // cell width  xF(i)-xF(i-1)               (COORD_DX, :91-93)
    const double* c;    // cell centre 0.5*(xF(i)+xF(i-1))         (GET_COORD, :63-65)
    const double* s0;   // PPM slope weight b0c of cell i          (solver/reconstruct.f90:246)
    const double* s1;   // PPM slope weight b1c of cell i          (:247)
    const double* a0;   // PPM interface weights a0p..a3p of the   (:240-243)
    const double* a1;   //   face between cell i and i+1; equal to
    const double* a2;   //   a0m..a3m of cell i+1
    const double* a3;
    const double* tcf;  // TVD_MM cf of cell i                     (:110)
    const double* tcb;  // TVD_MM cb of cell i                     (:111)
};

struct Tabs {
    AxisTabs ax[3];
    // x-axis metric factors (solver/coords.f90:173-415)
    const double* r2;     // xF(j)*xF(j)
    const double* r3d3;   // (xF(j)^3 - xF(j-1)^3)/3
    const double* rfac;   // (2*(xF(j)^3-xF(j-1)^3)/3)/(xF(j)^2-xF(j-1)^2)
    const double* hr2;    // 0.5*(xF(j)^2 - xF(j-1)^2)
    // y-axis metric factors
    const double* sinf;   // sin(yF(k))
    const double* dcos;   // cos(yF(k-1)) - cos(yF(k))
    const double* tanc;   // tan(y-centre of cell k)
    const double* sinc;   // sin(y-centre of cell k)
};

// Equation identifiers (solver/setup.f90:49-116), zero-based here.
enum { IRHO = 0, IVX = 1, IVY = 2, IVZ = 3, ITAU = 4, IBX = 5, IBY = 6, IBZ = 7 };

// ---------------------------------------------------------------------------
// reconstruction
// ---------------------------------------------------------------------------

// van Leer-limited PPM slope of a cell from its neighbours
// (solver/reconstruct.f90:254-280). The reference evaluates this three times
// per call (dmm1, dmc, dmp1); the three forms are the same expression of the
// cell's own (vm, vc, vp) and weights, so it is computed once per cell.
//
// The sweeps are bound by the FP64 pipe, so the double forms here and below
// move what they can to the integer pipe without changing a value: signs and
// minima of products and magnitudes are read from the bit patterns (a double
// orders like its bits among the non-negative ones), a product with 2 merges
// with the following sum (it is exact, so the fused sum rounds the same), and
// min(2a, 2b) = 2 min(a, b). The sign tests x > 0, x <= 0 and x < 0 are false for
// a NaN of either sign. WORDS: on the integer pipe (two or three instructions
// each), else by the FP64 pipe's compare (one). The x sweep with two cells a lane
// is faster with the first (256^3: 0.918 ms against 0.975), the walkers with the
// second (y 0.899 against 0.926, z 0.900 against 0.916).
template <bool WORDS>
__device__ __forceinline__ bool above_zero(double x) {
    if constexpr (!WORDS) return x > 0.0;
    return (unsigned)((unsigned long long)(__double_as_longlong(x) - 1) >> 32) < 0x7ff00000u;
}
template <bool WORDS>
__device__ __forceinline__ bool not_above_zero(double x) {
    if constexpr (!WORDS) return x <= 0.0;
    return !(__double_as_longlong(x) > 0 || (unsigned)__double2hiint(x) > 0xfff00000u);
}
template <bool WORDS>
__device__ __forceinline__ bool below_zero(double x) {
    if constexpr (!WORDS) return x < 0.0;
    return (unsigned)((unsigned long long)(__double_as_longlong(x) + 0x7fffffffffffffffll) >> 32) < 0x7ff00000u;
}
__device__ __forceinline__ double min_mag(double a, double b) {  // both non-negative
    return __longlong_as_double(min(__double_as_longlong(a), __double_as_longlong(b)));
}
template <bool WORDS = true, typename R>
__device__ __forceinline__ R ppm_slope(R vm, R vc, R vp, R b0, R b1) {
    const R delta = b0 * (vp - vc) + b1 * (vc - vm);
    if constexpr (sizeof(R) == 8) {
        const double up = vp - vc, dn = vc - vm;
        const double s = copysign(min_mag(fabs(delta), 2.0 * min_mag(fabs(dn), fabs(up))), delta);
        return above_zero<WORDS>(up * dn) ? s : 0.0;
    }
    if ((vp - vc) * (vc - vm) > R(0))
        return fmin(fmin(fabs(delta), R(2) * fabs(vc - vm)), R(2) * fabs(vc - vp)) * copysign(R(1), delta);
    return R(0);
}

// Unlimited PPM value at the face between cell c and c+1
// (solver/reconstruct.f90:285; identical to :286 evaluated by cell c+1).
template <typename R>
__device__ __forceinline__ R ppm_face(R vc, R vp, R dmc, R dmp, R a0, R a1, R a2, R a3) {
    return (((vc + a0 * (vp - vc)) + a1 * (vp - vc)) + a2 * dmp) + a3 * dmc;
}

// Extremum and overshoot fixes of one cell (solver/reconstruct.f90:289-307).
// The second test reads the already-modified left value, as the reference does.
template <bool WORDS = true, typename R>
__device__ __forceinline__ void ppm_fix(R vc, R vl, R vr, R& vm_out, R& vp_out) {
    if constexpr (sizeof(R) == 8) {
        const double c3 = 3.0 * vc;
        const bool flat = not_above_zero<WORDS>((vr - vc) * (vc - vl));
        const double m = below_zero<WORDS>((vr - vl) * __fma_rn(2.0, vr, vl - c3)) ? __fma_rn(-2.0, vr, c3) : vl;
        const double q = __fma_rn(-2.0, vl, c3);
        const double p = below_zero<WORDS>((vr - m) * (q - vr)) ? q : vr;
        vm_out = flat ? vc : m;
        vp_out = flat ? vc : p;
        return;
    }
    vm_out = vl;
    vp_out = vr;
    if ((vr - vc) * (vc - vl) <= R(0)) {
        vp_out = vc;
        vm_out = vc;
    } else {
        if ((vr - vl) * ((vl - R(3) * vc) + R(2) * vr) < R(0)) vm_out = R(3) * vc - R(2) * vr;
        if ((vp_out - vm_out) * ((R(3) * vc - R(2) * vl) - vr) < R(0)) vp_out = R(3) * vc - R(2) * vl;
    }
}

// TVD minmod slope of a cell (solver/reconstruct.f90:110-118).
template <typename R>
__device__ __forceinline__ R tvd_slope(R vm, R vc, R vp, R cf, R cb) {
    const R dqf = (R(2) * (vp - vc)) / cf;
    const R dqb = (R(2) * (vc - vm)) / cb;
    return (R(0.5) * (copysign(R(1), dqf) + copysign(R(1), dqb))) * fmin(fabs(dqf), fabs(dqb));
}

// The reconstruction weights of one cell and its upper face, read (and, in the
// mixed form, rounded to FP32) once for the seven fields: the sweeps store
// between fields, so the compiler would read them again for each.
template <int RECON, typename R>
struct CellWeights {  // PPM: slope weights of cell c, interface weights of the face c | c+1
    R s0, s1, a0, a1, a2, a3;
    __device__ __forceinline__ CellWeights(const AxisTabs& A, int cs, int cf)
        : s0((R)A.s0[cs]), s1((R)A.s1[cs]), a0((R)A.a0[cf]), a1((R)A.a1[cf]), a2((R)A.a2[cf]), a3((R)A.a3[cf]) {}
    static constexpr int N = 6;  // stored weights a face, in the order of the constructor below
    __device__ __forceinline__ CellWeights(const R* t, int n)
        : s0(t[0]), s1(t[n]), a0(t[2 * n]), a1(t[3 * n]), a2(t[4 * n]), a3(t[5 * n]) {}
    __device__ __forceinline__ void store(R* t, int n) const {
        t[0] = s0, t[n] = s1, t[2 * n] = a0, t[3 * n] = a1, t[4 * n] = a2, t[5 * n] = a3;
    }
    template <bool WORDS = true>
    __device__ __forceinline__ R slope(R vm, R vc, R vp) const {
        return ppm_slope<WORDS>(vm, vc, vp, s0, s1);
    }
    __device__ __forceinline__ R face(R vc, R vp, R dmc, R dmp) const {
        return ppm_face(vc, vp, dmc, dmp, a0, a1, a2, a3);
    }
};
template <typename R>
struct CellWeights<1, R> {  // TVD
    R cf, cb;
    static constexpr int N = 2;
    __device__ __forceinline__ CellWeights(const AxisTabs& A, int c) : cf((R)A.tcf[c]), cb((R)A.tcb[c]) {}
    __device__ __forceinline__ CellWeights(const R* t, int n) : cf(t[0]), cb(t[n]) {}
    __device__ __forceinline__ void store(R* t, int n) const { t[0] = cf, t[n] = cb; }
    __device__ __forceinline__ R slope(R vm, R vc, R vp) const { return tvd_slope(vm, vc, vp, cf, cb); }
};
// TVD in FP64: the quotients by cf and cb share their reciprocals over the
// fields (cumc_round.cuh; the plain operators outside the range)
template <>
struct CellWeights<1, double> {
    double cf, cb;
    Recip rf, rb;
    bool ok;
    static constexpr int N = 2;
    __device__ __forceinline__ CellWeights(const AxisTabs& A, int c) : cf(A.tcf[c]), cb(A.tcb[c]) {
        ok = range_max(cf, range_max(cb, 0u)) < RANGE_SPAN;
        rf = recip_of(cf);
        rb = recip_of(cb);
    }
    __device__ __forceinline__ double slope(double vm, double vc, double vp) const {
        const double nf = 2.0 * (vp - vc), nb = 2.0 * (vc - vm);
        const unsigned mf = magnitude(nf), mb = magnitude(nb);
        if (!ok || tiny_min(mf, tiny_min(mb, ~0u)) < TINY || max(mf, mb) >= HUGE_MAG)
            return tvd_slope(vm, vc, vp, cf, cb);
        const double dqf = quot_signed(nf, cf, rf), dqb = quot_signed(nb, cb, rb);
        // (sign(dqf) + sign(dqb))/2 min(|dqf|, |dqb|), a zero positive where the signs differ
        const bool same = (__double2hiint(dqf) >= 0) == (__double2hiint(dqb) >= 0);
        return same ? copysign(min_mag(fabs(dqf), fabs(dqb)), dqf) : 0.0;
    }
};

// ---------------------------------------------------------------------------
// HLL Riemann solver at one face (solver/rsolver.f90:43-130)
// ---------------------------------------------------------------------------

// compute_signalspeed (solver/definition.f90:394-410)
template <typename R>
__device__ __forceinline__ R signalspeed(R cs, R bn, R bt1, R bt2, R rho) {
    const R a2 = cs * cs;
    const R a4 = a2 * a2;
    const R b2n = (bn * bn) / rho;
    const R b2t1 = (bt1 * bt1) / rho;
    const R b2t2 = (bt2 * bt2) / rho;
    const R b2 = (b2n + b2t1) + b2t2;
    const R b4 = b2 * b2;
    return sqrt(R(0.5) * ((a2 + b2) + sqrt(fmax(((a4 + b4) + (R(2) * b2) * a2) - (R(4) * a2) * b2n, R(0)))));
}

// 1/x, sqrt(x) and sqrt(max(x, 0)) of the reciprocal forms. NEAR: without a
// branch, for the operands that the callers' range tests admit: the IEEE
// results, but for the few FP64 divisors whose reciprocal lies within 2^-51 of a
// unit of a rounding midpoint (cumc_round.cuh). The last Newton step counts:
// without it, a unit off half the time, a 128^3 step takes 1.916 ms instead of
// 1.926, and the density of Orszag-Tang 256^3 at t = 0.5 lies 4.0e-13 from the
// bitwise path instead of 3.0e-13. Else the IEEE operations.
template <bool NEAR>
__device__ __forceinline__ float recip_q(float x) { return NEAR ? recip_f(x) : 1.0f / x; }
template <bool NEAR>
__device__ __forceinline__ double recip_q(double x) {
    if constexpr (NEAR) return recip_of(x).y;
    return 1.0 / x;
}
template <bool NEAR>
__device__ __forceinline__ float root_q(float x) { return NEAR ? root_f(x) : sqrtf(x); }
template <bool NEAR>
__device__ __forceinline__ double root_q(double x) {
    if constexpr (NEAR) return root_of(x);
    return sqrt(x);
}
template <bool NEAR>
__device__ __forceinline__ float root_max0_q(float x) {
    if (!NEAR) return sqrtf(fmaxf(x, 0.0f));
    return x > 0.0f ? root_f(x) : 0.0f;
}
template <bool NEAR>
__device__ __forceinline__ double root_max0_q(double x) {
    if constexpr (NEAR) return root_pos(x);
    return sqrt(fmax(x, 0.0));
}

// compute_signalspeed with the quotients by rho formed as products with
// irho = 1/rho (the CUMC_FP64_FAST and mixed forms: not bit-compatible with the
// reference); square: a2 + b2, for the range test
template <bool NEAR, typename R>
__device__ __forceinline__ R signalspeed_recip(R cs, R bn, R bt1, R bt2, R irho, R& square) {
    const R a2 = cs * cs;
    const R a4 = a2 * a2;
    const R b2n = (bn * bn) * irho;
    const R b2t1 = (bt1 * bt1) * irho;
    const R b2t2 = (bt2 * bt2) * irho;
    const R b2 = (b2n + b2t1) + b2t2;
    const R b4 = b2 * b2;
    square = a2 + b2;
    return root_q<NEAR>(R(0.5) *
                        (square + root_max0_q<NEAR>(((a4 + b4) + (R(2) * b2) * a2) - (R(4) * a2) * b2n)));
}

// compute_roe (solver/definition.f90:387-392)
template <typename R>
__device__ __forceinline__ R roe_avg(R xl, R xr, R sl, R sr) {
    // sl, sr = sqrt(rhoL), sqrt(rhoR): the reference takes each DSQRT again
    // per call; the value is the same.
    return (sl * xl + sr * xr) / (sl + sr);
}

// compute_fluxhll (solver/definition.f90:380-385)
template <typename R>
__device__ __forceinline__ R fluxhll(R yl, R yr, R xl, R xr, R sl, R sr) {
    return ((sr * yl - sl * yr) + (sl * sr) * (xr - xl)) / (sr - sl);
}

// One side of the face (PtoU_MHD_face, solver/ptou_face.f90:34-88, and
// Ptof_MHD, solver/flux.f90:163-262), kept as the few scalars every conserved
// and flux component is formed from, so that the HLL combination below can
// form one component at a time (each with the reference's expression tree)
// instead of holding four 8-vectors live.
template <int DIR, typename R>
struct FaceSide {
    static constexpr int t1 = (DIR + 1) % 3, t2 = (DIR + 2) % 3;
    R rho, v[3], p, b[3], E, hb2, vdotb;
    struct GivenEps {};
    __device__ __forceinline__ FaceSide(const R w[8], R ggas)
        : FaceSide(w, (w[ITAU] / w[IRHO]) / (ggas - R(1)), GivenEps{}) {}
    // e: the side's specific internal energy, EOS_EPSILON (model/riemann/src/eos.f90:194)
    __device__ __forceinline__ FaceSide(const R w[8], R e, GivenEps) {
        rho = w[IRHO];
        v[0] = w[IVX]; v[1] = w[IVY]; v[2] = w[IVZ];
        p = w[ITAU];
        b[0] = w[IBX]; b[1] = w[IBY]; b[2] = w[IBZ];
        const R vsquare = (v[0] * v[0] + v[1] * v[1]) + v[2] * v[2];
        const R bsquare = (b[0] * b[0] + b[1] * b[1]) + b[2] * b[2];
        E = rho * (e + R(0.5) * vsquare) + R(0.5) * bsquare;
        hb2 = R(0.5) * bsquare;
        vdotb = (b[0] * v[0] + b[1] * v[1]) + b[2] * v[2];
    }
    // conserved component q
    __device__ __forceinline__ R u(int q) const {
        return q == IRHO ? rho : q <= IVZ ? v[q - IVX] * rho : q == ITAU ? E : b[q - IBX];
    }
    // flux component q along DIR (q != IBX+DIR, whose flux is 0)
    __device__ __forceinline__ R f(int q) const {
        const R vn = v[DIR], bn = b[DIR];
        if (q == IRHO) return rho * vn;
        if (q == IVX + DIR) return ((v[DIR] * rho * vn + p) + hb2) - bn * bn;
        if (q == IVX + t1) return v[t1] * rho * vn - bn * b[t1];
        if (q == IVX + t2) return v[t2] * rho * vn - bn * b[t2];
        if (q == ITAU) return (E * vn + (p + hb2) * vn) - bn * vdotb;
        if (q == IBX + t1) return vn * b[t1] - v[t1] * bn;
        return vn * b[t2] - v[t2] * bn;  // IBX + t2
    }
};

// HLL flux at a face from the left and right primitive states (8 each,
// natural order). out receives the 7 stored components: rho, rho v, E and
// the two tangential fields in natural (x, y, z) order.
template <int DIR, typename R>
__device__ __forceinline__ void hll_flux7(const R wl[8], const R wr[8], R ggas, R out[7]) {
    constexpr int ivn = IVX + DIR;
    constexpr int ibn = IBX + DIR, ibt1 = IBX + (DIR + 1) % 3, ibt2 = IBX + (DIR + 2) % 3;
    using Side = FaceSide<DIR, R>;
    const Side L(wl, ggas), Rs(wr, ggas);
    // EOS_SOUNDSPEED (model/riemann/src/eos.f90:168)
    const R csL = sqrt((ggas * wl[ITAU]) / wl[IRHO]);
    const R csR = sqrt((ggas * wr[ITAU]) / wr[IRHO]);
    const R cfsL = signalspeed(csL, wl[ibn], wl[ibt1], wl[ibt2], wl[IRHO]);
    const R cfsR = signalspeed(csR, wr[ibn], wr[ibt1], wr[ibt2], wr[IRHO]);
    const R sqL = sqrt(wl[IRHO]), sqR = sqrt(wr[IRHO]);
    const R ubar = roe_avg(wl[ivn], wr[ivn], sqL, sqR);
    const R cbar = roe_avg(cfsL, cfsR, sqL, sqR);
    const R sL = fmin(wl[ivn] - cfsL, ubar - cbar);
    const R sR = fmax(wr[ivn] + cfsR, ubar + cbar);
    constexpr int bt_a = DIR == 0 ? IBY : IBX;  // stored tangential components
    constexpr int bt_b = DIR == 2 ? IBY : IBZ;
    const int comp[7] = {IRHO, IVX, IVY, IVZ, ITAU, bt_a, bt_b};
    if (sL >= R(0)) {
#pragma unroll
        for (int c = 0; c < 7; ++c) out[c] = L.f(comp[c]);
    } else if (sL <= R(0) && sR >= R(0)) {
#pragma unroll
        for (int c = 0; c < 7; ++c)
            out[c] = fluxhll(L.f(comp[c]), Rs.f(comp[c]), L.u(comp[c]), Rs.u(comp[c]), sL, sR);
    } else {
#pragma unroll
        for (int c = 0; c < 7; ++c) out[c] = Rs.f(comp[c]);
    }
}

// hll_flux7 with the plain operators, out of line: the faces whose operands
// leave the ranges of hll_flux7_rounded
template <int DIR>
__device__ __noinline__ void hll_flux7_ieee(const double* w, double ggas, double* out) {
    double wl[8], wr[8], fx[7];
    for (int q = 0; q < 8; ++q) {
        wl[q] = w[q];
        wr[q] = w[8 + q];
    }
    hll_flux7<DIR, double>(wl, wr, ggas, fx);
    for (int q = 0; q < 7; ++q) out[q] = fx[q];
}

// Bounds of the branch-free solves. With densities and pressures in
// [2^-200, 2^200), a squared sound speed is at least 2^-400; with a2 + b2 below
// 2^500 every square, root and quotient of the speeds is a normal number (a
// faint field's share of a sum below 2^-900 vanishes beside a2, whatever its
// quotient), and with normal velocities below 2^500 so are the Roe averages. An
// overflow, an infinity or a NaN on the way leaves a2 + b2 or the velocity
// above its bound, since every word of it compares as more than any number's.
constexpr unsigned SQUARE_MAX = (1023u + 500u) << 20;   // the high word of 2^500
constexpr unsigned SPEED_MAX = SQUARE_MAX << 1;         // without the sign
__device__ __forceinline__ unsigned speed_max(double vl, double vr) {
    const unsigned l = hi_word(vl), r = hi_word(vr);
    return max(l + l, r + r);
}

// one side's fast speed and internal energy for hll_flux7_rounded; the values
// of EOS_SOUNDSPEED, compute_signalspeed and EOS_EPSILON; square: high word of
// a2 + b2
struct SideSpeed {
    double cf, sq, e;
    unsigned square;
};
__device__ __forceinline__ SideSpeed side_speed(double rho, double p, double bn2, double bt1, double bt2, double ggas,
                                                double gm1, const Recip& rg) {
    const Recip r = recip_of(rho);
    const double cs = root_of(quot(ggas * p, rho, r));
    const double a2 = cs * cs;
    const double b2n = quot(bn2, rho, r);
    const double b2 = (b2n + quot(bt1 * bt1, rho, r)) + quot(bt2 * bt2, rho, r);
    // ((a4 + b4) + (2 b2) a2) - (4 a2) b2n with the exact factors 2 and 4 merged
    const double x = __fma_rn(2.0, b2 * a2, a2 * a2 + b2 * b2);
    const double s = root_pos(__fma_rn(-4.0, a2 * b2n, x));
    return {root_of(0.5 * ((a2 + b2) + s)), root_of(rho), quot(quot(p, rho, r), gm1, rg), hi_word(a2 + b2)};
}

// hll_flux7 in FP64, bit for bit, with the quotients and roots of
// cumc_round.cuh. The sweeps are bound by the FP64 pipe and by its latency: the
// 21 quotients and 8 roots of the plain form carried a range branch each, which
// kept them from overlapping (1,414 instructions a face and warp in the y
// walker, 0.53 issued a cycle at 160^3). y and z walkers 1.17 -> 0.88 ms and the
// x sweep 1.25 -> 1.08 ms at 256^3 with the integer-pipe limiter above; the
// torus' y walker 0.193 -> 0.108 ms. Returns false where a density, a pressure,
// gamma - 1, a squared speed or a normal velocity lies outside the bounds above
// and the face needs the plain operators throughout.
template <int DIR>
__device__ __forceinline__ bool hll_flux7_rounded(const double (&wl)[8], const double (&wr)[8], double ggas,
                                                  double (&out)[7]) {
    constexpr int ivn = IVX + DIR, ibn = IBX + DIR, ibt1 = IBX + (DIR + 1) % 3, ibt2 = IBX + (DIR + 2) % 3;
    constexpr int bt_a = DIR == 0 ? IBY : IBX, bt_b = DIR == 2 ? IBY : IBZ;
    constexpr int comp[7] = {IRHO, IVX, IVY, IVZ, ITAU, bt_a, bt_b};
    const double gm1 = ggas - 1.0, bn2 = wl[ibn] * wl[ibn];
    const unsigned far =
        range_max(wl[IRHO], range_max(wr[IRHO], range_max(wl[ITAU], range_max(wr[ITAU], range_max(gm1, 0u)))));
    if (far >= RANGE_SPAN || speed_max(wl[ivn], wr[ivn]) >= SPEED_MAX) return false;
    using Side = FaceSide<DIR, double>;
    const Recip rg = recip_of(gm1);
    const SideSpeed l = side_speed(wl[IRHO], wl[ITAU], bn2, wl[ibt1], wl[ibt2], ggas, gm1, rg);
    const SideSpeed r = side_speed(wr[IRHO], wr[ITAU], bn2, wr[ibt1], wr[ibt2], ggas, gm1, rg);
    if (max(l.square, r.square) >= SQUARE_MAX) return false;
    const double sq = l.sq + r.sq;
    const Recip rs = recip_of(sq);
    const double ubar = quot(l.sq * wl[ivn] + r.sq * wr[ivn], sq, rs);
    const double cbar = quot(l.sq * l.cf + r.sq * r.cf, sq, rs);
    const double sL = fmin(wl[ivn] - l.cf, ubar - cbar);
    const double sR = fmax(wr[ivn] + r.cf, ubar + cbar);
    const Side L(wl, l.e, typename Side::GivenEps{}), Rs(wr, r.e, typename Side::GivenEps{});
    if (sL >= 0.0) {
#pragma unroll
        for (int c = 0; c < 7; ++c) out[c] = L.f(comp[c]);
    } else if (sR >= 0.0) {
        const double lr = sL * sR;
        double a[7];
#pragma unroll
        for (int c = 0; c < 7; ++c) {
            const int q = comp[c];
            a[c] = (sR * L.f(q) - sL * Rs.f(q)) + lr * (Rs.u(q) - L.u(q));
        }
        quot_group(a, sR - sL, out);
    } else {
#pragma unroll
        for (int c = 0; c < 7; ++c) out[c] = Rs.f(comp[c]);
    }
    return true;
}

// The reciprocal form (CUMC_FP64_FAST and the mixed form's all-FP32 variant, not
// bit-compatible with the reference): the 21 quotients of a face share five
// divisors (rho of either side, ggas - 1, the Roe weight sum, sR - sL), so each
// divisor's reciprocal is formed once and the quotients become products; the
// values differ from the reference's by a few units in the last place.
// NEAR (FP64): the reciprocals and roots without a branch; false where a
// density, a pressure, gamma - 1 or a squared speed is out of the bounds
// above, as in a cold fluid, where a field that fades squares to a subnormal.
template <int DIR, typename R, bool NEAR>
__device__ __forceinline__ bool hll_flux7_recip(const R (&wl)[8], const R (&wr)[8], R ggas, R (&out)[7]) {
    constexpr int ivn = IVX + DIR;
    constexpr int ibn = IBX + DIR, ibt1 = IBX + (DIR + 1) % 3, ibt2 = IBX + (DIR + 2) % 3;
    constexpr int bt_a = DIR == 0 ? IBY : IBX, bt_b = DIR == 2 ? IBY : IBZ;
    constexpr int comp[7] = {IRHO, IVX, IVY, IVZ, ITAU, bt_a, bt_b};
    using Side = FaceSide<DIR, R>;
    const R gm1 = ggas - R(1);
    if constexpr (NEAR)
        if (range_max(wl[IRHO],
                      range_max(wr[IRHO], range_max(wl[ITAU], range_max(wr[ITAU], range_max(gm1, 0u))))) >= RANGE_SPAN)
            return false;
    const R irL = recip_q<NEAR>(wl[IRHO]), irR = recip_q<NEAR>(wr[IRHO]), ig = recip_q<NEAR>(gm1);
    const Side L(wl, wl[ITAU] * irL * ig, typename Side::GivenEps{});
    const Side Rs(wr, wr[ITAU] * irR * ig, typename Side::GivenEps{});
    R squareL, squareR;
    const R csL = root_q<NEAR>((ggas * wl[ITAU]) * irL);
    const R csR = root_q<NEAR>((ggas * wr[ITAU]) * irR);
    const R cfsL = signalspeed_recip<NEAR>(csL, wl[ibn], wl[ibt1], wl[ibt2], irL, squareL);
    const R cfsR = signalspeed_recip<NEAR>(csR, wr[ibn], wr[ibt1], wr[ibt2], irR, squareR);
    if constexpr (NEAR)
        if (max(hi_word(squareL), hi_word(squareR)) >= SQUARE_MAX) return false;
    const R sqL = root_q<NEAR>(wl[IRHO]), sqR = root_q<NEAR>(wr[IRHO]);
    const R isq = recip_q<NEAR>(sqL + sqR);
    const R ubar = (sqL * wl[ivn] + sqR * wr[ivn]) * isq;
    const R cbar = (sqL * cfsL + sqR * cfsR) * isq;
    const R sL = fmin(wl[ivn] - cfsL, ubar - cbar);
    const R sR = fmax(wr[ivn] + cfsR, ubar + cbar);
    if (sL >= R(0)) {
#pragma unroll
        for (int c = 0; c < 7; ++c) out[c] = L.f(comp[c]);
    } else if (sL <= R(0) && sR >= R(0)) {
        // (at least a Roe-weighted sound speed, 2^-400, and less than 2^1000 unless
        // a velocity makes every product below infinite as well)
        const R ids = recip_q<NEAR>(sR - sL);
#pragma unroll
        for (int c = 0; c < 7; ++c) {
            const R yl = L.f(comp[c]), yr = Rs.f(comp[c]), xl = L.u(comp[c]), xr = Rs.u(comp[c]);
            out[c] = ((sR * yl - sL * yr) + (sL * sR) * (xr - xl)) * ids;
        }
    } else {
#pragma unroll
        for (int c = 0; c < 7; ++c) out[c] = Rs.f(comp[c]);
    }
    return true;
}
// its form with the IEEE operations, out of line
template <int DIR>
__device__ __noinline__ void hll_flux7_recip_ieee(const double* w, double ggas, double* out) {
    double wl[8], wr[8], fx[7];
    for (int q = 0; q < 8; ++q) {
        wl[q] = w[q];
        wr[q] = w[8 + q];
    }
    hll_flux7_recip<DIR, double, false>(wl, wr, ggas, fx);
    for (int q = 0; q < 7; ++q) out[q] = fx[q];
}

// ---------------------------------------------------------------------------
// CFL time step of one cell (finddt, solver/rungekutta.f90:201-250)
// ---------------------------------------------------------------------------

// the fast magnetosonic speed along each axis from the cell's primitives and
// bcell, then cfl * min(dx, dy, dz) / max_d(|v_d| + c_f,d); the inner square
// root has no MAX(., 0) guard, as in the reference. dxl, dyl, dzl are the
// cell's lengths along the three axes (cfl_lengths). Every caller of the CFL
// step (finddt, its fusion into stage 3, cumc_cfl_dt_static) evaluates this
// one function, so they give the same double.
__host__ __device__ __forceinline__ double cfl_cell_dt(double rho, double p, double vx, double vy, double vz,
                                                       double bcx, double bcy, double bcz, double dxl, double dyl,
                                                       double dzl, double ggas, double cfl) {
    const double cs = sqrt((ggas * p) / rho);
    const double a2 = cs * cs;
    const double a4 = a2 * a2;
    const double b2x = (bcx * bcx) / rho;
    const double b2y = (bcy * bcy) / rho;
    const double b2z = (bcz * bcz) / rho;
    const double b2 = (b2x + b2y) + b2z;
    const double b4 = b2 * b2;
    const double base = (a4 + (2.0 * a2) * b2) + b4;
    const double cfx = sqrt(0.5 * ((a2 + b2) + sqrt(base - (4.0 * a2) * b2x)));
    const double cfy = sqrt(0.5 * ((a2 + b2) + sqrt(base - (4.0 * a2) * b2y)));
    const double cfz = sqrt(0.5 * ((a2 + b2) + sqrt(base - (4.0 * a2) * b2z)));
    const double lambda = fmax(fmax(fabs(vx) + cfx, fabs(vy) + cfy), fabs(vz) + cfz);
    return (fmin(fmin(dxl, dyl), dzl) * cfl) / lambda;
}

// the cell's lengths along the axes (solver/rungekutta.f90:237-243): the
// widths, with dy -> r dy on cylindrical and spherical grids and
// dz -> r sin(theta) dz on spherical ones; xc is the cell-centre radius and
// sinyc the sine of the polar cell centre. coordinate: 1 Cartesian,
// 2 cylindrical, 3 spherical.
__host__ __device__ __forceinline__ void cfl_lengths(int coordinate, double xc, double sinyc, double& dyl,
                                                     double& dzl) {
    if (coordinate == 2) {
        dyl = xc * dyl;
    } else if (coordinate == 3) {
        dyl = xc * dyl;
        dzl = (xc * sinyc) * dzl;
    }
}

// ---------------------------------------------------------------------------
// geometry (solver/coords.f90) from the 1-D tables
// ---------------------------------------------------------------------------

// GEOM_FLUX (solver/coords.f90:231-302) for direction DIR at cell (j,k,l)
template <int COORD, int DIR>
__device__ __forceinline__ void geom_flux(const Tabs& T, int j, int k, int l, double& gp, double& gc, double& gm) {
    if (COORD == 1) {
        gp = 1.0;
        gm = 1.0;
        gc = DIR == 0 ? T.ax[0].d[j] : DIR == 1 ? T.ax[1].d[k] : T.ax[2].d[l];
    } else if (COORD == 2) {
        if (DIR == 0) { gp = T.ax[0].f[j]; gm = T.ax[0].f[j - 1]; gc = T.ax[0].c[j] * T.ax[0].d[j]; }
        else if (DIR == 1) { gp = 1.0; gm = 1.0; gc = T.ax[0].c[j] * T.ax[1].d[k]; }
        else { gp = 1.0; gm = 1.0; gc = T.ax[2].d[l]; }
    } else {
        if (DIR == 0) { gp = T.r2[j]; gm = T.r2[j - 1]; gc = T.r3d3[j]; }
        else if (DIR == 1) { gp = T.sinf[k]; gm = T.sinf[k - 1]; gc = T.rfac[j] * T.dcos[k]; }
        else { gp = 1.0; gm = 1.0; gc = ((T.rfac[j] * T.dcos[k]) * T.ax[2].d[l]) / T.ax[1].d[k]; }
    }
}

// GEOM_CT (solver/coords.f90:310-415)
struct CTf {
    double bx_ez_m, bx_ez_c, bx_ez_p, bx_ey_m, bx_ey_c, bx_ey_p;
    double by_ex_m, by_ex_c, by_ex_p, by_ez_m, by_ez_c, by_ez_p;
    double bz_ex_m, bz_ex_c, bz_ex_p, bz_ey_m, bz_ey_c, bz_ey_p;
};
template <int COORD>
__device__ __forceinline__ void geom_ct(const Tabs& T, int j, int k, int l, CTf& g) {
    const double dxl = T.ax[0].d[j], dyl = T.ax[1].d[k], dzl = T.ax[2].d[l];
    if (COORD == 1) {
        g.bx_ez_m = 1.0; g.bx_ez_c = dyl; g.bx_ez_p = 1.0;
        g.bx_ey_m = 1.0; g.bx_ey_c = dzl; g.bx_ey_p = 1.0;
        g.by_ex_m = 1.0; g.by_ex_c = dzl; g.by_ex_p = 1.0;
        g.by_ez_m = 1.0; g.by_ez_c = dxl; g.by_ez_p = 1.0;
        g.bz_ey_m = 1.0; g.bz_ey_c = dxl; g.bz_ey_p = 1.0;
        g.bz_ex_m = 1.0; g.bz_ex_c = dyl; g.bz_ex_p = 1.0;
    } else if (COORD == 2) {
        const double x = T.ax[0].c[j];
        g.bx_ez_m = 1.0; g.bx_ez_c = dyl * T.ax[0].f[j]; g.bx_ez_p = 1.0;
        g.bx_ey_m = 1.0; g.bx_ey_c = dzl; g.bx_ey_p = 1.0;
        g.by_ex_m = 1.0; g.by_ex_c = dzl; g.by_ex_p = 1.0;
        g.by_ez_m = 1.0; g.by_ez_c = dxl; g.by_ez_p = 1.0;
        g.bz_ey_m = T.ax[0].f[j - 1]; g.bz_ey_c = x * dxl; g.bz_ey_p = T.ax[0].f[j];
        g.bz_ex_m = 1.0; g.bz_ex_c = x * dyl; g.bz_ex_p = 1.0;
    } else {
        const double x = T.ax[0].c[j];
        const double dc = T.dcos[k];
        g.bx_ez_m = T.sinf[k - 1]; g.bx_ez_c = T.ax[0].f[j] * dc; g.bx_ez_p = T.sinf[k];
        g.bx_ey_m = 1.0; g.bx_ey_c = ((T.ax[0].f[j] * dc) * dzl) / dyl; g.bx_ey_p = 1.0;
        g.by_ex_m = 1.0; g.by_ex_c = (x * T.sinf[k]) * dzl; g.by_ex_p = 1.0;
        g.by_ez_m = T.ax[0].f[j - 1]; g.by_ez_c = x * dxl; g.by_ez_p = T.ax[0].f[j];
        g.bz_ey_m = T.ax[0].f[j - 1]; g.bz_ey_c = x * dxl; g.bz_ey_p = T.ax[0].f[j];
        g.bz_ex_m = 1.0; g.bz_ex_c = x * dyl; g.bz_ex_p = 1.0;
    }
}

// ---------------------------------------------------------------------------
// HLL of the mixed form (float states). The wave speeds and the two stored
// tangential-field components are formed in FP32, in the reciprocal form of
// hll_flux7_recip (five divisors, each reciprocal formed once); the five hydro
// components (rho, rho v, E) take their side fluxes, conserved values and HLL
// combination in FP64 from the FP32 states, with each side's internal energy,
// E, B^2/2 and v.B in FP64. Measured on Orszag-Tang 256^3 to t = 0.5, the
// all-FP32 form leaves the density 1.06e-5 (relative L1) from the FP64 run,
// this form 8.0e-6: the side fluxes' and the combination's FP32 rounding is
// the largest error left once the states are FP32.
//
// The FP64 quotients (by rho, by gamma-1, by sR-sL) start from the FP32
// reciprocal and take one Newton-Raphson step for 1/x, r' = r (2 - x r),
// which squares its relative error (6e-8 -> ~4e-15): FP64 accuracy without
// an FP64 division.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double rcp_newton(double x, float r0) {
    const double r = (double)r0;
    return r * (2.0 - x * r);
}

// one side's flux (F) or conserved value (U) of component q, in T from the
// FP32 side primitives and the side's derived scalars
template <typename T, int DIR>
__device__ __forceinline__ T side_f(const FaceSide<DIR, float>& s, int q, double Ex, double hb2x, double vdotbx) {
    constexpr int t1 = (DIR + 1) % 3, t2 = (DIR + 2) % 3;
    const T rho = s.rho, vn = s.v[DIR], bn = s.b[DIR], p = s.p, hb2 = (T)hb2x, E = (T)Ex, vdotb = (T)vdotbx;
    if (q == IRHO) return rho * vn;
    if (q == IVX + DIR) return ((vn * rho * vn + p) + hb2) - bn * bn;
    if (q == IVX + t1) return (T)s.v[t1] * rho * vn - bn * (T)s.b[t1];
    if (q == IVX + t2) return (T)s.v[t2] * rho * vn - bn * (T)s.b[t2];
    if (q == ITAU) return (E * vn + (p + hb2) * vn) - bn * vdotb;
    if (q == IBX + t1) return vn * (T)s.b[t1] - (T)s.v[t1] * bn;
    return vn * (T)s.b[t2] - (T)s.v[t2] * bn;
}
template <typename T, int DIR>
__device__ __forceinline__ T side_u(const FaceSide<DIR, float>& s, int q, double Ex) {
    return q == IRHO ? (T)s.rho : q <= IVZ ? (T)s.v[q - IVX] * (T)s.rho : q == ITAU ? (T)Ex : (T)s.b[q - IBX];
}

// a side's internal energy, E, B^2/2 and v.B in FP64 from its FP32 primitives
// (the FaceSide expressions); irho32, ig32: FP32 reciprocals of rho and gamma-1
struct SideScalars {
    double E, hb2, vdotb;
};
__device__ __forceinline__ SideScalars side_scalars64(const float (&w)[8], float irho32, double ig) {
    const double rho = w[IRHO], vx = w[IVX], vy = w[IVY], vz = w[IVZ], bx = w[IBX], by = w[IBY], bz = w[IBZ];
    const double e = (double)w[ITAU] * rcp_newton(rho, irho32) * ig;
    const double vsq = (vx * vx + vy * vy) + vz * vz, bsq = (bx * bx + by * by) + bz * bz;
    return {rho * (e + 0.5 * vsq) + 0.5 * bsq, 0.5 * bsq, (bx * vx + by * vy) + bz * vz};
}

// ROUNDED: the five FP32 reciprocals and eight roots without their range
// branches; false (nothing computed) where a density leaves [2^-60, 2^60), gamma
// p/rho [2^-38, 2^45), or a2 + b2 is not below 2^49 (its square then exceeds the
// roots' 2^100, or is infinite or NaN)
template <int DIR, bool ROUNDED>
__device__ __forceinline__ bool hll_flux7_mixed_form(const float (&wl)[8], const float (&wr)[8], float ggas,
                                                     float (&out)[7]) {
    constexpr int ivn = IVX + DIR;
    constexpr int ibn = IBX + DIR, ibt1 = IBX + (DIR + 1) % 3, ibt2 = IBX + (DIR + 2) % 3;
    constexpr int HYDRO = 5;  // components 0..4 in FP64
    const float irL = recip_q<ROUNDED>(wl[IRHO]), irR = recip_q<ROUNDED>(wr[IRHO]);
    float sL, sR;
    {
        const float xL = (ggas * wl[ITAU]) * irL, xR = (ggas * wr[ITAU]) * irR;
        if (ROUNDED && (range_max_f<-60>(wl[IRHO], range_max_f<-60>(wr[IRHO], 0u)) >= 120u << 23 ||
                        range_max_f<-38>(xL, range_max_f<-38>(xR, 0u)) >= 83u << 23))
            return false;
        const float csL = root_q<ROUNDED>(xL);
        const float csR = root_q<ROUNDED>(xR);
        float squareL, squareR;
        const float cfsL = signalspeed_recip<ROUNDED>(csL, wl[ibn], wl[ibt1], wl[ibt2], irL, squareL);
        const float cfsR = signalspeed_recip<ROUNDED>(csR, wr[ibn], wr[ibt1], wr[ibt2], irR, squareR);
        if (ROUNDED && max(__float_as_uint(squareL), __float_as_uint(squareR)) >= (127u + 49u) << 23) return false;
        const float sqL = root_q<ROUNDED>(wl[IRHO]), sqR = root_q<ROUNDED>(wr[IRHO]);
        const float isq = recip_q<ROUNDED>(sqL + sqR);
        const float ubar = (sqL * wl[ivn] + sqR * wr[ivn]) * isq;
        const float cbar = (sqL * cfsL + sqR * cfsR) * isq;
        sL = fminf(wl[ivn] - cfsL, ubar - cbar);
        sR = fmaxf(wr[ivn] + cfsR, ubar + cbar);
    }
    using Side = FaceSide<DIR, float>;
    const float ig = 1.0f / (ggas - 1.0f);
    const double igd = rcp_newton((double)ggas - 1.0, ig);
    const SideScalars aL = side_scalars64(wl, irL, igd), aR = side_scalars64(wr, irR, igd);
    // the FP32 side (tangential-field components only read rho, v, b)
    const Side L(wl, wl[ITAU] * irL * ig, typename Side::GivenEps{});
    const Side Rs(wr, wr[ITAU] * irR * ig, typename Side::GivenEps{});
    constexpr int bt_a = DIR == 0 ? IBY : IBX;
    constexpr int bt_b = DIR == 2 ? IBY : IBZ;
    const int comp[7] = {IRHO, IVX, IVY, IVZ, ITAU, bt_a, bt_b};
    if (sL >= 0.0f) {
#pragma unroll
        for (int q = 0; q < 7; ++q)
            out[q] = q < HYDRO ? (float)side_f<double>(L, comp[q], aL.E, aL.hb2, aL.vdotb) : L.f(comp[q]);
    } else if (sR >= 0.0f) {
        // sR - sL > 0 is at least a sound speed, 2^-19
        const float ds = sR - sL, lrf = sL * sR;
        const float idsf = ROUNDED && ds < 0x1p100f ? recip_q<ROUNDED>(ds) : 1.0f / ds;
        const double cl = sL, cr = sR, ids = rcp_newton(cr - cl, idsf), lr = cl * cr;
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            if (q < HYDRO) {
                const double yl = side_f<double>(L, comp[q], aL.E, aL.hb2, aL.vdotb);
                const double yr = side_f<double>(Rs, comp[q], aR.E, aR.hb2, aR.vdotb);
                const double xl = side_u<double>(L, comp[q], aL.E), xr = side_u<double>(Rs, comp[q], aR.E);
                out[q] = (float)(((cr * yl - cl * yr) + lr * (xr - xl)) * ids);
            } else {
                const float yl = L.f(comp[q]), yr = Rs.f(comp[q]), xl = L.u(comp[q]), xr = Rs.u(comp[q]);
                out[q] = ((sR * yl - sL * yr) + lrf * (xr - xl)) * idsf;
            }
        }
    } else {
#pragma unroll
        for (int q = 0; q < 7; ++q)
            out[q] = q < HYDRO ? (float)side_f<double>(Rs, comp[q], aR.E, aR.hb2, aR.vdotb) : Rs.f(comp[q]);
    }
    return true;
}

// the plain form out of line
template <int DIR>
__device__ __noinline__ void hll_flux7_mixed_plain(const float* w, float ggas, float* out) {
    float wl[8], wr[8], fx[7];
    for (int q = 0; q < 8; ++q) {
        wl[q] = w[q];
        wr[q] = w[8 + q];
    }
    hll_flux7_mixed_form<DIR, false>(wl, wr, ggas, fx);
    for (int q = 0; q < 7; ++q) out[q] = fx[q];
}
template <int DIR>
__device__ __forceinline__ void hll_flux7_mixed(const float (&wl)[8], const float (&wr)[8], float ggas,
                                                float (&out)[7]) {
    if (hll_flux7_mixed_form<DIR, true>(wl, wr, ggas, out)) return;
    float w[16], f[7];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        w[q] = wl[q];
        w[8 + q] = wr[q];
    }
    hll_flux7_mixed_plain<DIR>(w, ggas, f);
#pragma unroll
    for (int q = 0; q < 7; ++q) out[q] = f[q];
}


// the sweeps' HLL solve: hll_flux7's values in FP64 (RECIP: the CUMC_FP64_FAST
// form). For the mixed form's float states, RECIP selects the all-FP32
// reciprocal form (faster; density 1.06e-5 from the FP64 run at t_end above)
// and its absence hll_flux7_mixed (the default).
template <int DIR, typename R, bool RECIP>
__device__ __forceinline__ void sweep_hll(const R (&wl)[8], const R (&wr)[8], R ggas, R (&fx)[7]) {
    if constexpr (sizeof(R) == 4) {
        if constexpr (RECIP) hll_flux7_recip<DIR, R, false>(wl, wr, ggas, fx);
        else hll_flux7_mixed<DIR>(wl, wr, ggas, fx);
    } else {
        const bool done = RECIP ? hll_flux7_recip<DIR, double, true>(wl, wr, ggas, fx)
                                : hll_flux7_rounded<DIR>(wl, wr, ggas, fx);
        if (done) return;
        double w[16], f[7];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            w[q] = wl[q];
            w[8 + q] = wr[q];
        }
        if constexpr (RECIP) hll_flux7_recip_ieee<DIR>(w, ggas, f);
        else hll_flux7_ieee<DIR>(w, ggas, f);
#pragma unroll
        for (int q = 0; q < 7; ++q) fx[q] = f[q];
    }
}

}  // namespace cumc
