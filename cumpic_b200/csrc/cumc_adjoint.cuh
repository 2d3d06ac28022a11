// cumc_adjoint.cuh — hand-written discrete adjoint of the FP64 RK3 step
// (Cartesian, cylindrical and spherical grids, models NONE and RIEMANN, PPM or
// TVD reconstruction, HLL, CT, every boundary flag).
//
// The forward stage s (solver/rungekutta.f90:38-66 and the kernels of
// cumc_kernels.cuh) is, per stage,
//   P_{s-1}   primitives with ghosts (utop + boundary of the previous combine)
//   F         = sweeps(P_{s-1})             face fluxes (PPM/TVD + HLL)
//   E         = emf(F, P_{s-1})             edge EMFs
//   L         = combine's flux difference and CT curl of (F, E)
//   Upre_s    = a U0 + b U_{s-1} + c dt L   on (0:n)^3
//   (U_s,P_s) = utop(Upre_s) + boundary
// with dt frozen (recorded in the forward pass). The reverse sweep of a stage
// applies the transposes in the opposite order:
//   boundary^T   ghost adjoints folded onto the active cells they copy
//   utop^T       adjoint of Upre_s from those of U_s and P_s
//   combine^T    a, b parts to U0, U_{s-1}; c dt part to L
//   CT^T, emf^T  edge and cell-EMF adjoints
//   sweep^T      HLL^T and PPM^T per face, limiter and solver branches
//                frozen by recomputing the forward values
// Cells outside 1:n and face fields outside their live positions are
// overwritten by the forward boundary, so their adjoints are folded onto
// their sources and then zero.
#pragma once
#include "cumc_kernels.cuh"
#include "cumc_walk.cuh"

namespace cumc {

// device pointer sets passed by value
struct Arr8 {
    double* a[8];
};
struct Arr3 {
    double* a[3];
};

// adjoint of the primitive fields of one stage (with ghosts)
struct AdjPrim {
    double* w[5];   // rho, vx, vy, vz, p
    double* bc[3];  // cell-centred B
    double* eps;
};

// ---------------------------------------------------------------------------
// reconstruction transposes (branches frozen by recomputation)
// ---------------------------------------------------------------------------

// transpose of the TVD reconstruction of one cell from v[1..3] = cells
// c-1..c+1: seeds lvm, lvp on (vm_out, vp_out); adds to lv[1..3]
__device__ __forceinline__ void tvd_adj(const AxisTabs& A, int c, const double v[5], double lvm, double lvp,
                                        double lv[5]) {
    if (lvm == 0.0 && lvp == 0.0) return;
    // vm = vc - sl/2, vp = vc + sl/2, sl = minmod of dqf = 2(vp-vc)/cf, dqb = 2(vc-vm)/cb
    lv[2] += lvm + lvp;
    const double lsl = 0.5 * (lvp - lvm);
    const double cf = A.tcf[c], cb = A.tcb[c];
    const double dqf = (2.0 * (v[3] - v[2])) / cf;
    const double dqb = (2.0 * (v[2] - v[1])) / cb;
    const double sf = copysign(1.0, dqf), sb = copysign(1.0, dqb);
    if (sf != sb) return;  // slope 0
    if (fabs(dqf) <= fabs(dqb)) {  // slope = dqf
        lv[3] += 2.0 * lsl / cf;
        lv[2] -= 2.0 * lsl / cf;
    } else {  // slope = dqb
        lv[2] += 2.0 * lsl / cb;
        lv[1] -= 2.0 * lsl / cb;
    }
}

// ---------------------------------------------------------------------------
// HLL transpose (hll_flux7 of cumc_device.cuh, branches frozen)
// ---------------------------------------------------------------------------
template <int DIR>
struct SideAdj {
    // forward values here only weight derivatives, so reciprocals replace
    // the forward's divisions (no branch depends on them)
    double rho, irho, v[3], p, b[3], e, vsq, bsq, E, hb2, vdotb;
    double Lrho, Lv[3], Lp, Lb[3], LE, Lhb2, Lvdotb;
    __device__ __forceinline__ void init(const double w[8], double irho_, double ig1) {
        rho = w[IRHO];
        irho = irho_;
        v[0] = w[IVX]; v[1] = w[IVY]; v[2] = w[IVZ];
        p = w[ITAU];
        b[0] = w[IBX]; b[1] = w[IBY]; b[2] = w[IBZ];
        e = (p * irho) * ig1;
        vsq = (v[0] * v[0] + v[1] * v[1]) + v[2] * v[2];
        bsq = (b[0] * b[0] + b[1] * b[1]) + b[2] * b[2];
        E = rho * (e + 0.5 * vsq) + 0.5 * bsq;
        hb2 = 0.5 * bsq;
        vdotb = (b[0] * v[0] + b[1] * v[1]) + b[2] * v[2];
        Lrho = Lp = LE = Lhb2 = Lvdotb = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) Lv[i] = Lb[i] = 0.0;
    }
    __device__ __forceinline__ double u(int q) const {
        return q == IRHO ? rho : q <= IVZ ? v[q - IVX] * rho : q == ITAU ? E : b[q - IBX];
    }
    __device__ __forceinline__ double f(int q) const {
        constexpr int t1 = (DIR + 1) % 3, t2 = (DIR + 2) % 3;
        const double vn = v[DIR], bn = b[DIR];
        if (q == IRHO) return rho * vn;
        if (q == IVX + DIR) return ((v[DIR] * rho * vn + p) + hb2) - bn * bn;
        if (q == IVX + t1) return v[t1] * rho * vn - bn * b[t1];
        if (q == IVX + t2) return v[t2] * rho * vn - bn * b[t2];
        if (q == ITAU) return (E * vn + (p + hb2) * vn) - bn * vdotb;
        if (q == IBX + t1) return vn * b[t1] - v[t1] * bn;
        return vn * b[t2] - v[t2] * bn;
    }
    __device__ __forceinline__ void u_adj(int q, double lam) {
        if (q == IRHO) Lrho += lam;
        else if (q <= IVZ) { Lv[q - IVX] += lam * rho; Lrho += lam * v[q - IVX]; }
        else if (q == ITAU) LE += lam;
        else Lb[q - IBX] += lam;
    }
    __device__ __forceinline__ void f_adj(int q, double lam) {
        const double vn = v[DIR], bn = b[DIR];
        if (q == IRHO) {
            Lrho += lam * vn;
            Lv[DIR] += lam * rho;
        } else if (q == IVX + DIR) {
            Lv[DIR] += lam * 2.0 * rho * vn;
            Lrho += lam * vn * vn;
            Lp += lam;
            Lhb2 += lam;
            Lb[DIR] -= lam * 2.0 * bn;
        } else if (q >= IVX && q <= IVZ) {
            const int t = q - IVX;
            Lv[t] += lam * rho * vn;
            Lrho += lam * v[t] * vn;
            Lv[DIR] += lam * v[t] * rho;
            Lb[DIR] -= lam * b[t];
            Lb[t] -= lam * bn;
        } else if (q == ITAU) {
            LE += lam * vn;
            Lv[DIR] += lam * (E + p + hb2);
            Lp += lam * vn;
            Lhb2 += lam * vn;
            Lb[DIR] -= lam * vdotb;
            Lvdotb -= lam * bn;
        } else {
            const int t = q - IBX;
            Lv[DIR] += lam * b[t];
            Lb[t] += lam * vn;
            Lv[t] -= lam * bn;
            Lb[DIR] -= lam * v[t];
        }
    }
    // fold E, hb2, vdotb, e into the primitive adjoints; out[8] in natural order
    __device__ __forceinline__ void finish(double ig1, double out[8]) {
        const double Le = LE * rho;
        const double Lvsq = LE * 0.5 * rho;
        const double Lbsq = LE * 0.5 + 0.5 * Lhb2;
        Lrho += LE * (e + 0.5 * vsq);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            Lb[i] += Lvdotb * v[i] + 2.0 * b[i] * Lbsq;
            Lv[i] += Lvdotb * b[i] + 2.0 * v[i] * Lvsq;
        }
        Lp += Le * irho * ig1;
        Lrho -= Le * e * irho;
        out[IRHO] += Lrho;
        out[IVX] += Lv[0]; out[IVY] += Lv[1]; out[IVZ] += Lv[2];
        out[ITAU] += Lp;
        out[IBX] += Lb[0]; out[IBY] += Lb[1]; out[IBZ] += Lb[2];
    }
};

// one side's speeds as the forward has them (bit for bit, so that the branches
// below are the forward's), and the reciprocals that weight derivatives
template <int DIR>
struct SideWave {
    double irho, cs, cf, sq, ics_p;  // 1/rho, sound and fast speed, sqrt(rho), 1/p
    double a2, b2n, b2, is, icf;     // of compute_signalspeed; is = 1/sqrt(inner) or 0, icf = 1/cf
};
template <int DIR, bool ROUNDED>
__device__ __forceinline__ SideWave<DIR> side_wave(const double (&w)[8], double g) {
    constexpr int ibn = IBX + DIR, ibt1 = IBX + (DIR + 1) % 3, ibt2 = IBX + (DIR + 2) % 3;
    const double rho = w[IRHO], p = w[ITAU];
    SideWave<DIR> s;
    double inner, root;
    if constexpr (ROUNDED) {
        const Recip r = recip_of(rho);
        s.irho = r.y;
        s.cs = root_of(quot(g * p, rho, r));
        s.a2 = s.cs * s.cs;
        s.b2n = quot(w[ibn] * w[ibn], rho, r);
        s.b2 = (s.b2n + quot(w[ibt1] * w[ibt1], rho, r)) + quot(w[ibt2] * w[ibt2], rho, r);
        inner = __fma_rn(-4.0, s.a2 * s.b2n, __fma_rn(2.0, s.b2 * s.a2, s.a2 * s.a2 + s.b2 * s.b2));
        root = root_pos(inner);
        s.cf = root_of(0.5 * ((s.a2 + s.b2) + root));
        s.sq = root_of(rho);
        s.is = inner > 0.0 ? recip_q<true>(root) : 0.0;
        s.icf = recip_q<true>(s.cf);
        s.ics_p = recip_q<true>(p);
    } else {
        s.irho = 1.0 / rho;
        s.cs = sqrt((g * p) / rho);
        s.a2 = s.cs * s.cs;
        s.b2n = (w[ibn] * w[ibn]) / rho;
        s.b2 = (s.b2n + (w[ibt1] * w[ibt1]) / rho) + (w[ibt2] * w[ibt2]) / rho;
        inner = ((s.a2 * s.a2 + s.b2 * s.b2) + (2.0 * s.b2) * s.a2) - (4.0 * s.a2) * s.b2n;
        root = sqrt(fmax(inner, 0.0));
        s.cf = sqrt(0.5 * ((s.a2 + s.b2) + root));
        s.sq = sqrt(rho);
        s.is = inner > 0.0 ? 1.0 / root : 0.0;
        s.icf = s.cf > 0.0 ? 1.0 / s.cf : 0.0;
        s.ics_p = s.cs > 0.0 ? 1.0 / p : 0.0;
    }
    return s;
}
// the plain form, for densities and pressures outside the rounded one's range
template <int DIR>
__device__ __noinline__ SideWave<DIR> side_wave_plain(const double* wp, double g) {
    double w[8];
    for (int q = 0; q < 8; ++q) w[q] = wp[q];
    return side_wave<DIR, false>(w, g);
}

// Adjoint of out[7] = hll_flux7<DIR>(wl, wr): lout[7] -> put(side, out[8]), called
// once a side. With id = 1/(sR - sL) and ln = lout id, the wave speeds enter
// the HLL average only through the jumps dF = sum ln (fR - fL) and
// dU = sum ln (uR - uL): d/dsL = id sR (sR dU - dF), d/dsR = id sL (dF - sL dU). So the
// two sides are transposed one after the other, each with ln scaled by its two
// coefficients, and only one side's adjoints are live at a time.
template <int DIR, typename Put>
__device__ __forceinline__ void hll_adj(const double (&wl)[8], const double (&wr)[8], double g, const double (&lout)[7],
                                        Put&& put) {
    constexpr int ivn = IVX + DIR;
    constexpr int bt_a = DIR == 0 ? IBY : IBX;
    constexpr int bt_b = DIR == 2 ? IBY : IBZ;
    constexpr int comp[7] = {IRHO, IVX, IVY, IVZ, ITAU, bt_a, bt_b};
    const double ig1 = recip_q<true>(g - 1.0);
    SideWave<DIR> w[2];
    if (range_max(wl[IRHO], range_max(wr[IRHO], range_max(wl[ITAU], range_max(wr[ITAU], 0u)))) < RANGE_SPAN) {
        w[0] = side_wave<DIR, true>(wl, g);
        w[1] = side_wave<DIR, true>(wr, g);
    } else {
        double c[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) c[q] = wl[q];
        w[0] = side_wave_plain<DIR>(c, g);
#pragma unroll
        for (int q = 0; q < 8; ++q) c[q] = wr[q];
        w[1] = side_wave_plain<DIR>(c, g);
    }
    const double sqs = w[0].sq + w[1].sq;
    const Recip rs = recip_of(sqs);
    const double ubar = quot(w[0].sq * wl[ivn] + w[1].sq * wr[ivn], sqs, rs);
    const double cbar = quot(w[0].sq * w[0].cf + w[1].sq * w[1].cf, sqs, rs);
    const double aL = wl[ivn] - w[0].cf, bL = ubar - cbar;
    const double aR = wr[ivn] + w[1].cf, bR = ubar + cbar;
    const double sL = fmin(aL, bL), sR = fmax(aR, bR);
    double ln[7], kf[2], ku[2], lsL = 0.0, lsR = 0.0;
    const bool mid = !(sL >= 0.0) && sR >= 0.0;
    const double id = mid ? recip_q<true>(sR - sL) : 1.0;
#pragma unroll
    for (int c = 0; c < 7; ++c) ln[c] = lout[c] * id;
    kf[0] = mid ? sR : sL >= 0.0 ? 1.0 : 0.0;
    kf[1] = mid ? -sL : sL >= 0.0 ? 0.0 : 1.0;
    ku[1] = mid ? sL * sR : 0.0;
    ku[0] = -ku[1];
    if (mid) {
        SideAdj<DIR> L, R;
        L.init(wl, w[0].irho, ig1);
        R.init(wr, w[1].irho, ig1);
        double dF = 0.0, dU = 0.0;
#pragma unroll
        for (int c = 0; c < 7; ++c) {
            dF += ln[c] * (R.f(comp[c]) - L.f(comp[c]));
            dU += ln[c] * (R.u(comp[c]) - L.u(comp[c]));
        }
        lsL = id * sR * (sR * dU - dF);
        lsR = id * sL * (dF - sL * dU);
    }
    // sL = min(aL, bL), sR = max(aR, bR), then the Roe averages
    double lvn[2] = {0.0, 0.0}, lcf[2] = {0.0, 0.0}, lubar = 0.0, lcbar = 0.0;
    if (aL <= bL) { lvn[0] += lsL; lcf[0] -= lsL; } else { lubar += lsL; lcbar -= lsL; }
    if (aR >= bR) { lvn[1] += lsR; lcf[1] += lsR; } else { lubar += lsR; lcbar += lsR; }
    lubar *= rs.y;
    lcbar *= rs.y;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const double(&x)[8] = s == 0 ? wl : wr;
        const SideWave<DIR>& v = w[s];
        SideAdj<DIR> S;
        S.init(x, v.irho, ig1);
#pragma unroll
        for (int c = 0; c < 7; ++c) {
            S.f_adj(comp[c], kf[s] * ln[c]);
            S.u_adj(comp[c], ku[s] * ln[c]);
        }
        const double lsq = lubar * (x[ivn] - ubar) + lcbar * (v.cf - cbar);
        const double lc = lcf[s] + lcbar * v.sq;
        S.Lv[DIR] += lvn[s] + lubar * v.sq;
        S.Lrho += 0.5 * lsq * (v.sq * v.irho);  // d sqrt(rho) = d rho sqrt(rho)/(2 rho)
        // cf = sqrt((a2 + b2 + sqrt(inner))/2): signalspeed's transpose
        const double lsum = lc * 0.25 * v.icf, ls = lsum * 0.5 * v.is, ab = v.a2 + v.b2;
        const double la2 = lsum + ls * (2.0 * ab - 4.0 * v.b2n), lb2 = lsum + ls * 2.0 * ab;
        const double lb2n = lb2 - 4.0 * ls * v.a2;
        S.Lb[DIR] += 2.0 * x[IBX + DIR] * v.irho * lb2n;
        S.Lb[(DIR + 1) % 3] += 2.0 * x[IBX + (DIR + 1) % 3] * v.irho * lb2;
        S.Lb[(DIR + 2) % 3] += 2.0 * x[IBX + (DIR + 2) % 3] * v.irho * lb2;
        S.Lrho -= (v.b2n * lb2n + (v.b2 - v.b2n) * lb2) * v.irho;
        // a2 = g p / rho
        S.Lp += la2 * v.a2 * v.ics_p;
        S.Lrho -= la2 * v.a2 * v.irho;
        double out[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        S.finish(ig1, out);
        put(s, out);
    }
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
struct AdjStage {
    const double* mu[8];    // adjoint of the combine's output (Upre), live entries only
    const double* lamE[3];  // edge-EMF adjoints (k_adj_ct)
    const double* dt;       // device dt of the step
    double gam;             // combine's coefficient on dt L
};

__device__ __forceinline__ bool inside(int j, int k, int l, const Box& b) {
    return j >= 1 && j <= b.nx && k >= 1 && k <= b.ny && l >= 1 && l <= b.nz;
}
__device__ __forceinline__ bool in0n(int j, int k, int l, const Box& b) {
    return j >= 0 && j <= b.nx && k >= 0 && k <= b.ny && l >= 0 && l <= b.nz;
}

// CT^T: edge-EMF adjoints on (0:n)^3 from the field part of mu (solver/mhd.f90
// :137-148, with the GEOM_CT factors of solver/coords.f90:310-415). Each face
// field's l_rk is (E_a p - E_a' m)/c - (E_b p - E_b' m)/c over the triple's
// factors, so an edge collects p/c from its own triple and m/c from the
// triples above it.
template <int COORD>
__global__ void __launch_bounds__(256) k_adj_ct(Box b, Tabs T, AdjStage a, double* lex, double* ley, double* lez) {
    const int n0 = b.nx + 1, n1 = b.ny + 1, n2 = b.nz + 1;
    const long long total = (long long)n0 * n1 * n2;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int j = (int)(t % n0), k = (int)((t / n0) % n1), l = (int)(t / n0 / n1);
    const int i = b.idx(j, k, l);
    const int sj = 1, sk = b.SX, sl = b.SX * b.SY;
    const double cdt = a.gam * *a.dt;
    const double* mx = a.mu[IBX];
    const double* my = a.mu[IBY];
    const double* mz = a.mu[IBZ];
    // the face triple's own CT factors (the edge is its upper one) ...
    CTf g;
    geom_ct<COORD>(T, j, k, l, g);
    double ez = -(mx[i] * g.bx_ez_p) / g.bx_ez_c + (my[i] * g.by_ez_p) / g.by_ez_c;
    double ey = (mx[i] * g.bx_ey_p) / g.bx_ey_c - (mz[i] * g.bz_ey_p) / g.bz_ey_c;
    double ex = -(my[i] * g.by_ex_p) / g.by_ex_c + (mz[i] * g.bz_ex_p) / g.bz_ex_c;
    // ... and those of the triples above it, where the edge is the lower one
    if (k + 1 <= b.ny) {
        geom_ct<COORD>(T, j, k + 1, l, g);
        ez += (mx[i + sk] * g.bx_ez_m) / g.bx_ez_c;
        ex -= (mz[i + sk] * g.bz_ex_m) / g.bz_ex_c;
    }
    if (j + 1 <= b.nx) {
        geom_ct<COORD>(T, j + 1, k, l, g);
        ez -= (my[i + sj] * g.by_ez_m) / g.by_ez_c;
        ey += (mz[i + sj] * g.bz_ey_m) / g.bz_ey_c;
    }
    if (l + 1 <= b.nz) {
        geom_ct<COORD>(T, j, k, l + 1, g);
        ey -= (mx[i + sl] * g.bx_ey_m) / g.bx_ey_c;
        ex += (my[i + sl] * g.by_ex_m) / g.by_ex_c;
    }
    lex[i] = cdt * ex;
    ley[i] = cdt * ey;
    lez[i] = cdt * ez;
}

// emf^T, cell part: ecell = -v x B on (0:n+1)^3 enters four edges with -1/4
// (solver/mhd.f90:95-125); adds to the velocity and cell-field adjoints
__global__ void __launch_bounds__(256) k_adj_ecell(Box b, Prim pr, const double* lex, const double* ley,
                                                   const double* lez, AdjPrim o) {
    const int n0 = b.nx + 2, n1 = b.ny + 2, n2 = b.nz + 2;
    const long long total = (long long)n0 * n1 * n2;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int j = (int)(t % n0), k = (int)((t / n0) % n1), l = (int)(t / n0 / n1);
    const int i = b.idx(j, k, l);
    const int sj = 1, sk = b.SX, sl = b.SX * b.SY;
    auto E = [&](const double* e, int dj, int dk, int dl) -> double {
        const int jj = j - dj, kk = k - dk, ll = l - dl;
        return in0n(jj, kk, ll, b) ? e[i - dj * sj - dk * sk - dl * sl] : 0.0;
    };
    const double lx = -0.25 * (((E(lex, 0, 0, 0) + E(lex, 0, 0, 1)) + E(lex, 0, 1, 0)) + E(lex, 0, 1, 1));
    const double ly = -0.25 * (((E(ley, 0, 0, 0) + E(ley, 0, 0, 1)) + E(ley, 1, 0, 0)) + E(ley, 1, 0, 1));
    const double lz = -0.25 * (((E(lez, 0, 0, 0) + E(lez, 0, 1, 0)) + E(lez, 1, 0, 0)) + E(lez, 1, 1, 0));
    if (lx == 0.0 && ly == 0.0 && lz == 0.0) return;
    const double vx = pr.w[1][i], vy = pr.w[2][i], vz = pr.w[3][i];
    const double bx = pr.bc[0][i], by = pr.bc[1][i], bz = pr.bc[2][i];
    // ex = vz by - vy bz, ey = vx bz - vz bx, ez = vy bx - vx by
    o.w[1][i] += ly * bz - lz * by;
    o.w[2][i] += lz * bx - lx * bz;
    o.w[3][i] += lx * by - ly * bx;
    o.bc[0][i] += lz * vy - ly * vz;
    o.bc[1][i] += lx * vz - lz * vx;
    o.bc[2][i] += ly * vx - lx * vy;
}

// GEOM_SOURCE^T (solver/coords.f90:127-161) on the interior cells: the
// geometric source, added geom_repeat times to l_rk of the cell's momentum
// (and so to Upre with weight gam dt), differentiated with respect to the
// stage's primitives (rho, v, p, bcell) at the cell.
template <int COORD>
__global__ void __launch_bounds__(256) k_adj_source(Box b, Tabs T, Prim pr, AdjStage a, int repeat, AdjPrim o) {
    const long long total = (long long)b.nx * b.ny * b.nz;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int j = (int)(t % b.nx) + 1, k = (int)((t / b.nx) % b.ny) + 1, l = (int)(t / b.nx / b.ny) + 1;
    const int i = b.idx(j, k, l);
    const double f = (a.gam * *a.dt) * repeat;
    const double lx = f * a.mu[IVX][i], ly = f * a.mu[IVY][i], lz = f * a.mu[IVZ][i];
    const double rho = pr.w[0][i], vx = pr.w[1][i], vy = pr.w[2][i], vz = pr.w[3][i];
    const double bx = pr.bc[0][i], by = pr.bc[1][i], bz = pr.bc[2][i];
    const double ix = 1.0 / T.ax[0].c[j];
    double lrho, lvx, lvy, lvz, lp, lbx, lby, lbz;
    if (COORD == 2) {
        // sx = ((p + rho vy^2) + |B|^2/2 - by^2)/R, sy = -(rho vx vy - bx by)/R
        lrho = (lx * (vy * vy) - ly * (vx * vy)) * ix;
        lvx = -ly * (rho * vy) * ix;
        lvy = (lx * (2.0 * rho * vy) - ly * (rho * vx)) * ix;
        lvz = 0.0;
        lp = lx * ix;
        lbx = (lx * bx + ly * by) * ix;
        lby = (ly * bx - lx * by) * ix;
        lbz = lx * bz * ix;
    } else {
        // sx = ((2p + bx^2) + rho (vy^2 + vz^2))/r
        // sy = ((p + rho vz^2) + |B|^2/2 - bz^2)/(r tan) - (rho vx vy - bx by)/r
        // sz = -(rho vx vz - bx bz)/r - (rho vy vz - by bz)/(r tan)
        const double it = ix / T.tanc[k];
        lrho = lx * (vy * vy + vz * vz) * ix + ly * ((vz * vz) * it - (vx * vy) * ix) -
               lz * ((vx * vz) * ix + (vy * vz) * it);
        lvx = -(ly * vy + lz * vz) * rho * ix;
        lvy = lx * (2.0 * rho * vy) * ix - ly * (rho * vx) * ix - lz * (rho * vz) * it;
        lvz = lx * (2.0 * rho * vz) * ix + ly * (2.0 * rho * vz) * it - lz * ((rho * vx) * ix + (rho * vy) * it);
        lp = 2.0 * lx * ix + ly * it;
        lbx = 2.0 * lx * bx * ix + ly * (bx * it + by * ix) + lz * bz * ix;
        lby = ly * (by * it + bx * ix) + lz * bz * it;
        lbz = -ly * bz * it + lz * (bx * ix + by * it);
    }
    o.w[0][i] += lrho;
    o.w[1][i] += lvx;
    o.w[2][i] += lvy;
    o.w[3][i] += lvz;
    o.w[4][i] += lp;
    o.bc[0][i] += lbx;
    o.bc[1][i] += lby;
    o.bc[2][i] += lbz;
}

// adjoints of the reconstructed left and right states of each face (the 7
// reconstructed fields in sweep order), stored at the face's left cell
struct FaceAdj {
    double* l[7];
    double* r[7];
};

// sweep^T, pass A: per face (normal 0:n_d, transverse 0:n+1), the flux
// adjoints from mu (flux difference) and the edge adjoints (emf), the forward
// left/right states, and HLL^T. Writes the state adjoints to fa and adds the
// normal-field adjoint of the face to lambf. Four 128-thread blocks per SM
// (128 registers, 40 bytes spilled); 268 -> 178 us a launch at 128^3 with the two
// sides one after the other (hll_adj), FP64 pipe 57 % busy.
// fa holds the forward states (the forward sweep's STATES form, one
// reconstruction per cell: vp_out of cell c, vm_out of cell c+1); each face reads
// its two states and overwrites them with their adjoints.
#ifndef CUMC_ADJ_MINB
#define CUMC_ADJ_MINB 4
#endif
template <int COORD, int DIR>
__global__ void __launch_bounds__(128, CUMC_ADJ_MINB) k_adj_hll(Box b, Tabs T, Prim pr, double ggas, AdjStage a, FaceAdj fa,
                                                double* lambf) {
    const int n0 = (DIR == 0 ? b.nx : b.nx + 1) + 1;
    const int n1 = (DIR == 1 ? b.ny : b.ny + 1) + 1;
    const int n2 = (DIR == 2 ? b.nz : b.nz + 1) + 1;
    const long long total = (long long)n0 * n1 * n2;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int j = (int)(t % n0), k = (int)((t / n0) % n1), l = (int)(t / n0 / n1);
    const int base = b.idx(j, k, l);
    const int sj = 1, sk = b.SX, sl = b.SX * b.SY;
    const int s = DIR == 0 ? sj : DIR == 1 ? sk : sl;
    const int c = DIR == 0 ? j : DIR == 1 ? k : l;
    const int nd = DIR == 0 ? b.nx : DIR == 1 ? b.ny : b.nz;
    const AxisTabs A = T.ax[DIR];

    // flux adjoints
    double lf[7];
    const double cdt = a.gam * *a.dt;
    {
        const bool tin = DIR == 0 ? (k >= 1 && k <= b.ny && l >= 1 && l <= b.nz)
                                  : DIR == 1 ? (j >= 1 && j <= b.nx && l >= 1 && l <= b.nz)
                                             : (j >= 1 && j <= b.nx && k >= 1 && k <= b.ny);
        const bool lin = tin && c >= 1, rin = tin && c + 1 <= nd;
        // the face enters its left cell's flux difference as -F g+/g_c and
        // its right cell's as +F g-/g_c (Cartesian: 1/dx of each cell)
        double il = 0.0, ir = 0.0;
        if (COORD == 1) {
            il = lin ? 1.0 / A.d[c] : 0.0;
            ir = rin ? 1.0 / A.d[c + 1] : 0.0;
        } else {
            double gp, gc, gm;
            if (lin) {
                geom_flux<COORD, DIR>(T, j, k, l, gp, gc, gm);
                il = gp / gc;
            }
            if (rin) {
                geom_flux<COORD, DIR>(T, j + (DIR == 0), k + (DIR == 1), l + (DIR == 2), gp, gc, gm);
                ir = gm / gc;
            }
        }
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const double ml = lin ? a.mu[q][base] : 0.0, mr = rin ? a.mu[q][base + s] : 0.0;
            lf[q] = cdt * (mr * ir - ml * il);
        }
        auto E = [&](const double* e, int dj, int dk, int dl) -> double {
            return in0n(j - dj, k - dk, l - dl, b) ? e[base - dj * sj - dk * sk - dl * sl] : 0.0;
        };
        if (DIR == 0) {  // x faces: by enters ez (-1/2), bz enters ey (+1/2)
            lf[5] = -0.5 * (E(a.lamE[2], 0, 0, 0) + E(a.lamE[2], 0, 1, 0));
            lf[6] = 0.5 * (E(a.lamE[1], 0, 0, 0) + E(a.lamE[1], 0, 0, 1));
        } else if (DIR == 1) {  // y faces: bx enters ez (+1/2), bz enters ex (-1/2)
            lf[5] = 0.5 * (E(a.lamE[2], 0, 0, 0) + E(a.lamE[2], 1, 0, 0));
            lf[6] = -0.5 * (E(a.lamE[0], 0, 0, 0) + E(a.lamE[0], 0, 0, 1));
        } else {  // z faces: bx enters ey (-1/2), by enters ex (+1/2)
            lf[5] = -0.5 * (E(a.lamE[1], 0, 0, 0) + E(a.lamE[1], 1, 0, 0));
            lf[6] = 0.5 * (E(a.lamE[0], 0, 0, 0) + E(a.lamE[0], 0, 1, 0));
        }
    }
    bool any = false;
#pragma unroll
    for (int q = 0; q < 7; ++q) any |= lf[q] != 0.0;
    if (!any) {
#pragma unroll
        for (int v = 0; v < 7; ++v) fa.l[v][base] = fa.r[v][base] = 0.0;
        return;
    }

    constexpr int bt_a = DIR == 0 ? 1 : 0;
    constexpr int bt_b = DIR == 2 ? 1 : 2;
    const int slot[7] = {IRHO, IVX, IVY, IVZ, ITAU, IBX + bt_a, IBX + bt_b};

    double wl[8], wr[8];
#pragma unroll
    for (int v = 0; v < 7; ++v) {
        wl[slot[v]] = fa.l[v][base];
        wr[slot[v]] = fa.r[v][base];
    }
    const double bn = pr.bf[DIR][base];
    wl[IBX + DIR] = bn;
    wr[IBX + DIR] = bn;

    double lbn = 0.0;
    hll_adj<DIR>(wl, wr, ggas, lf, [&](int side, const double* out) {
        lbn += out[IBX + DIR];
        double* const* dst = side == 0 ? fa.l : fa.r;
#pragma unroll
        for (int v = 0; v < 7; ++v) dst[v][base] = out[slot[v]];
    });
    lambf[base] += lbn;
}

// field v (0..6) of a sweep along DIR: source and adjoint arrays. (v is not a
// constant here: the kernels below take their arrays as grid constants, which
// are indexed in place. As plain parameters they were copied to 272 bytes of
// stack by every thread first: k_adj_recon_x 795 us a launch at 128^3.)
template <int DIR>
__device__ __forceinline__ void sweep_field(const Prim& pr, const AdjPrim& o, int v, const double*& src, double*& dst) {
    constexpr int bt_a = DIR == 0 ? 1 : 0;
    constexpr int bt_b = DIR == 2 ? 1 : 2;
    if (v < 5) {
        src = pr.w[v];
        dst = o.w[v];
    } else {
        src = pr.bc[v == 5 ? bt_a : bt_b];
        dst = o.bc[v == 5 ? bt_a : bt_b];
    }
}

// The PPM reconstruction transpose, one slope, one interface value and one fix
// a cell. The adjoint of the interface value between two cells is the sum of
// the left one's vr and the right one's vl, so it is transposed once a face,
// and a slope's adjoint (from its two faces) once a cell. A slope's derivatives
// satisfy gc = -(gm + gp) on every branch.
struct PpmSlope {
    double d, gm, gp;
};
__device__ __forceinline__ PpmSlope ppm_slope_grad(double vm, double vc, double vp, double b0, double b1) {
    const double up = vp - vc, dn = vc - vm;
    const double delta = b0 * up + b1 * dn;
    const double m1 = fabs(delta), hd = fabs(dn), hu = fabs(up);
    const double m2 = 2.0 * hd, m3 = 2.0 * hu, m12 = min_mag(m1, m2);
    const bool on = above_zero<true>(up * dn);
    const bool by_up = m12 > m3, by_dn = !by_up && m1 > m2;  // limited by 2 |vc - vp|, by 2 |vc - vm|
    // sd 2 sign(dn); sign(up) = sign(dn) where the slope is on
    const double g = copysign(2.0, delta) * copysign(1.0, dn);
    PpmSlope s;
    s.d = on ? copysign(min_mag(m12, m3), delta) : 0.0;
    s.gm = !on || by_up ? 0.0 : by_dn ? -g : -b1;
    s.gp = !on || by_dn ? 0.0 : by_up ? g : b0;
    return s;
}
// ppm_fix's transpose at a cell with value vc and interface values vl, vr
struct PpmFixAdj {
    double c, l, r;
};
__device__ __forceinline__ PpmFixAdj ppm_fix_adj(double vc, double vl, double vr, double lvm, double lvp) {
    const double c3 = 3.0 * vc;
    const bool flat = not_above_zero<true>((vr - vc) * (vc - vl));
    const bool t1 = below_zero<true>((vr - vl) * __fma_rn(2.0, vr, vl - c3));
    const double vm = t1 ? __fma_rn(-2.0, vr, c3) : vl;
    const bool t2 = below_zero<true>((vr - vm) * (__fma_rn(-2.0, vl, c3) - vr));
    const double m1 = t1 ? lvm : 0.0, p1 = t2 ? lvp : 0.0;  // seeds that the fixes took over
    PpmFixAdj a;
    a.c = flat ? lvm + lvp : 3.0 * (m1 + p1);
    a.l = flat ? 0.0 : (lvm - m1) - 2.0 * p1;
    a.r = flat ? 0.0 : (lvp - p1) - 2.0 * m1;
    return a;
}

// sweep^T, pass B along y or z: the reconstruction transpose. One thread
// per (column, field, segment of RC_SEG cells) walks its segment: cell c's
// reconstruction (vm_out, vp_out) took its seeds from faces c-1 and c; its
// transpose adds to cells c-2..c+2, kept in registers, and a cell is
// complete once the walk has passed it by two. A segment writes cells
// c0-2 .. c1+1, so the four cells next to each end of a segment also receive
// from the neighbouring segment. The even segments run in one launch and
// the odd ones in a second (`parity`): within a launch no two threads write
// the same cell, every add is a plain one, and each cell takes its
// contributions in a fixed order, so the result is the same bits on every
// run. The next cell and face seeds are loaded one cell ahead. Against three
// slopes and two interface values a cell: 160 -> 83 us a launch at 128^3.
constexpr int RC_SEG = 32;

template <int DIR, int RECON>
__global__ void __launch_bounds__(128) k_adj_recon_col(Box b, const __grid_constant__ Tabs T, const __grid_constant__ Prim pr,
                                                       const __grid_constant__ FaceAdj fa,
                                                       const __grid_constant__ AdjPrim o, int parity) {
    using G = WalkGeom<DIR>;
    const unsigned col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= G::ncols(b)) return;
    const int v = blockIdx.y;
    const int nd = G::nd(b);
    const int c0 = (2 * (int)blockIdx.z + parity) * RC_SEG;
    if (c0 > nd + 1) return;
    const int c1 = min(c0 + RC_SEG, nd + 2);  // reconstructed cells 0..nd+1
    const int a = (int)(col % G::wa(b)), cc = (int)(col / G::wa(b));
    const int s = G::stride(b);
    const int base = G::idx(b, a, cc, 0);
    const AxisTabs A = T.ax[DIR];
    const double* src;
    double* dst;
    sweep_field<DIR>(pr, o, v, src, dst);
    src += base;
    dst += base;
    const double* fl = fa.l[v] + base;
    const double* fr = fa.r[v] + base;
    auto emit = [&](int q, double val) {
        if (val != 0.0) dst[q * s] += val;
    };
    double lvm = c0 >= 1 ? fr[(c0 - 1) * s] : 0.0;
    double lvp = c0 <= nd ? fl[c0 * s] : 0.0;
    if constexpr (RECON == 4) {
        const double xa = src[(c0 - 2) * s], xb = src[(c0 - 1) * s];
        double x0 = src[c0 * s], x1 = src[(c0 + 1) * s], x2 = src[(c0 + 2) * s];  // cells c, c+1, c+2
        PpmSlope sm = ppm_slope_grad(xa, xb, x0, A.s0[c0 - 1], A.s1[c0 - 1]);      // of cell c-1
        PpmSlope sc = ppm_slope_grad(xb, x0, x1, A.s0[c0], A.s1[c0]);              // of cell c
        double V = ppm_face(xb, x0, sm.d, sc.d, A.a0[c0 - 1], A.a1[c0 - 1], A.a2[c0 - 1], A.a3[c0 - 1]);
        double lr = 0.0, ld = 0.0;                // vr adjoint of cell c-1; slope adjoint of cell c-1
        double am = 0.0, ab = 0.0, ac = 0.0;      // value adjoints of cells c-2, c-1, c
        // the face between cells c-1 and c with adjoint L, then the slope of cell c-1
        auto close = [&](int c, double L, double& ld_c) {
            const double sL = (A.a0[c - 1] + A.a1[c - 1]) * L;
            ab += L - sL;
            ac += sL;
            const double l1 = ld + A.a3[c - 1] * L;
            ld_c = A.a2[c - 1] * L;
            am += l1 * sm.gm;
            ab -= l1 * (sm.gm + sm.gp);
            ac += l1 * sm.gp;
        };
        double d = dst[(c0 - 2) * s];  // what cell c-2 holds, read a cell ahead as well
        for (int c = c0; c < c1; ++c) {
            const double xn = c + 3 <= nd + 3 ? src[(c + 3) * s] : 0.0;
            const double lvm_n = fr[c * s];  // face c seeds vm_out of cell c+1
            const double lvp_n = c + 1 <= nd ? fl[(c + 1) * s] : 0.0;
            const double d_n = dst[(c - 1) * s];
            const PpmSlope sp = ppm_slope_grad(x0, x1, x2, A.s0[c + 1], A.s1[c + 1]);
            const double Vr = ppm_face(x0, x1, sc.d, sp.d, A.a0[c], A.a1[c], A.a2[c], A.a3[c]);
            const PpmFixAdj f = ppm_fix_adj(x0, V, Vr, lvm, lvp);
            double ld_c;
            close(c, lr + f.l, ld_c);
            ac += f.c;
            if (am != 0.0) dst[(c - 2) * s] = d + am;
            d = d_n;
            am = ab;
            ab = ac;
            ac = 0.0;
            lr = f.r;
            ld = ld_c;
            sm = sc;
            sc = sp;
            V = Vr;
            x0 = x1;
            x1 = x2;
            x2 = xn;
            lvm = lvm_n;
            lvp = lvp_n;
        }
        // the last face (c1-1 | c1), and the slopes of cells c1-1 and c1
        double ld_c;
        close(c1, lr, ld_c);
        if (am != 0.0) dst[(c1 - 2) * s] = d + am;
        emit(c1 - 1, ab + ld_c * sc.gm);
        emit(c1, ac - ld_c * (sc.gm + sc.gp));
        emit(c1 + 1, ld_c * sc.gp);
    } else {
        double x[5] = {src[(c0 - 2) * s], src[(c0 - 1) * s], src[c0 * s], src[(c0 + 1) * s], src[(c0 + 2) * s]};
        double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // cells c-2..c+2
        for (int c = c0; c < c1; ++c) {
            const double xn = c + 3 <= nd + 3 ? src[(c + 3) * s] : 0.0;
            const double lvm_n = fr[c * s];
            const double lvp_n = c + 1 <= nd ? fl[(c + 1) * s] : 0.0;
            tvd_adj(A, c, x, lvm, lvp, acc);
            emit(c - 2, acc[0]);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                acc[m] = acc[m + 1];
                x[m] = x[m + 1];
            }
            acc[4] = 0.0;
            x[4] = xn;
            lvm = lvm_n;
            lvp = lvp_n;
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) emit(c1 - 2 + m, acc[m]);
    }
}

// sweep^T, pass B along x: the reconstruction transpose with one lane per
// cell, one warp per (row, field, RX_CELLS cells). A warp covers 32 cells of a
// row and owns its middle RX_CELLS: each lane forms its own cell's slope,
// interface value and fix, and the neighbours' shares come through shuffles (a
// cell's adjoint reaches four cells to either side). Bound by issue: 269
// instructions a warp, 0.66 issued a cycle; 419 -> 255 us a launch at 128^3
// against three slopes a cell and the fields one after the other.
constexpr int RX_CELLS = 24;
inline long long recon_x_warps(const Box& b) {
    return (long long)(b.ny + 2) * (b.nz + 2) * ((b.nx + 6 + RX_CELLS - 1) / RX_CELLS);
}
template <int RECON>
__global__ void __launch_bounds__(128) k_adj_recon_x(Box b, const __grid_constant__ Tabs T, const __grid_constant__ Prim pr,
                                                     const __grid_constant__ FaceAdj fa,
                                                     const __grid_constant__ AdjPrim o) {
    constexpr unsigned FULL = 0xffffffffu;
    const int nw = (b.nx + 6 + RX_CELLS - 1) / RX_CELLS;  // warps per row
    // 32-bit index arithmetic (fewer warps than cells, fewer than 2^31 cells)
    const unsigned warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const unsigned row = warp / nw;
    const int w = (int)(warp - row * nw), k = (int)(row % (b.ny + 2)), l = (int)(row / (b.ny + 2));
    if (l > b.nz + 1) return;  // whole warp
    const int c = RX_CELLS * w + lane - 6;  // owned: lanes 4..27, from cell -2
    const AxisTabs A = T.ax[0];
    const int at = b.idx(0, k, l) + c;
    const bool mine = c >= 0 && c <= b.nx + 1;  // a reconstructed cell
    const bool owned = lane >= 4 && lane <= 27 && c <= b.nx + 3;
    const int ct = min(max(c, -1), b.nx + 1);  // table index of the lane's cell and its upper face
    const double* src;
    double* dst;
    sweep_field<0>(pr, o, (int)blockIdx.y, src, dst);
    const double x = c >= -2 && c <= b.nx + 3 ? src[at] : 0.0;
    const double lvm = mine && c >= 1 ? fa.r[blockIdx.y][at - 1] : 0.0;
    const double lvp = mine && c <= b.nx ? fa.l[blockIdx.y][at] : 0.0;
    const double held = owned ? dst[at] : 0.0;  // with the other loads, not after the arithmetic
    const double xm = __shfl_up_sync(FULL, x, 1), xp = __shfl_down_sync(FULL, x, 1);
    double tot;
    if constexpr (RECON == 4) {
        const int cs = min(max(c, -1), b.nx + 2);  // slopes exist on -1..nx+2
        const PpmSlope s = ppm_slope_grad(xm, x, xp, A.s0[cs], A.s1[cs]);
        const double a2 = A.a2[ct], a3 = A.a3[ct], as = A.a0[ct] + A.a1[ct];
        const double V = ppm_face(x, xp, s.d, __shfl_down_sync(FULL, s.d, 1), A.a0[ct], A.a1[ct], a2, a3);  // c | c+1
        const PpmFixAdj f = ppm_fix_adj(x, __shfl_up_sync(FULL, V, 1), V, lvm, lvp);
        const double L = f.r + __shfl_down_sync(FULL, f.l, 1);  // adjoint of V
        const double sL = as * L;
        // value and slope adjoints: from the face above (L) and the one below
        const double ld = a3 * L + __shfl_up_sync(FULL, a2 * L, 1);
        tot = (f.c + (L - sL)) + __shfl_up_sync(FULL, sL, 1) - ld * (s.gm + s.gp);
        tot += __shfl_down_sync(FULL, ld * s.gm, 1) + __shfl_up_sync(FULL, ld * s.gp, 1);
    } else {
        double lv[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        const double v[5] = {0.0, xm, x, xp, 0.0};
        if (mine) tvd_adj(A, c, v, lvm, lvp, lv);
        tot = lv[2] + __shfl_down_sync(FULL, lv[1], 1) + __shfl_up_sync(FULL, lv[3], 1);
    }
    if (owned && tot != 0.0) dst[at] = held + tot;
}

// boundary^T: the transpose of k_boundary, in gather form. k_boundary copies
// each ghost from one source (an active cell, or a live face), with the
// parity sign, and sets the ghost pressure p = rho eps (gamma-1)
// (solver/update.f90:27-35). So the transpose adds to each source the signed
// adjoints of every ghost copied from it, each ghost's density and eps
// adjoints first taking in its pressure adjoint. k_adj_boundary_gather runs
// one thread per possible source and enumerates its ghost images direction
// by direction (at most 6 per direction), so there are no atomics and the
// summation order is fixed. k_adj_boundary_clear then zeroes every ghost
// adjoint that was moved. fw holds the forward primitives of the stage.

// ghost indices along one direction whose gmap source is a; count returned
__device__ __forceinline__ int ghost_images(int a, int n, int fin, int fout, int* g, int* side) {
    int c = 0;
    if (a < 1 || a > n) return 0;
#pragma unroll
    for (int t = 0; t < 6; ++t) {
        const int i = t < 3 ? t - 2 : n + t - 2;
        int src, sd;
        gmap(i, n, fin, fout, src, sd);
        if (src == a) {
            g[c] = i;
            side[c] = sd;
            ++c;
        }
    }
    return c;
}

// parity factor of a ghost image (side < 0: identity)
__device__ __forceinline__ int bsign(const BoundArgs& fw, int dir, int side, int q) {
    if (side < 0 || fw.flag[2 * dir + side] < 2) return 1;
    return fw.fac[2 * dir + side][q];
}

// A ghost's source lies within three cells of a face, so only cells with an
// index in the face set 0..3, n-2..n of some direction are visited: one thread
// a box cell spent 119 us at 128^3, half its warps on the few such cells of
// every row.
__host__ __device__ __forceinline__ int face_set(int n) { return n + 1 < 7 ? n + 1 : 7; }  // its size
__device__ __forceinline__ int face_set_index(int s, int n) { return n + 1 < 7 || s < 4 ? s : n - 6 + s; }
inline long long face_set_cells(const Box& b) {
    const long long n0 = b.nx + 1, n1 = b.ny + 1, n2 = b.nz + 1;
    const long long i0 = n0 - face_set(b.nx), i1 = n1 - face_set(b.ny), i2 = n2 - face_set(b.nz);
    return n0 * n1 * n2 - i0 * i1 * i2;
}

__global__ void __launch_bounds__(256) k_adj_boundary_gather(Box b, const __grid_constant__ BoundArgs fw,
                                                             const __grid_constant__ AdjPrim o, double* lbx,
                                                             double* lby, double* lbz) {
    // the planes l in the face set, then the rows k in it of the other planes,
    // then the cells j in it of the other rows (the seven of a row on
    // consecutive threads)
    const int n0 = b.nx + 1, n1 = b.ny + 1, fx = face_set(b.nx), fy = face_set(b.ny), fz = face_set(b.nz);
    const unsigned nz = (unsigned)fz * n0 * n1, ny = (unsigned)(b.nz + 1 - fz) * fy * n0;
    unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    int j, k, l;
    if (t < nz) {
        j = (int)(t % n0);
        k = (int)((t / n0) % n1);
        l = face_set_index((int)(t / n0 / n1), b.nz);
    } else if ((t -= nz) < ny) {
        j = (int)(t % n0);
        k = face_set_index((int)((t / n0) % fy), b.ny);
        l = 4 + (int)(t / n0 / fy);
    } else {
        t -= ny;
        const unsigned rows = (unsigned)(n1 - fy) * (b.nz + 1 - fz);
        if (t >= rows * fx) return;
        j = face_set_index((int)(t % fx), b.nx);
        k = 4 + (int)((t / fx) % (n1 - fy));
        l = 4 + (int)(t / fx / (n1 - fy));
    }
    const int i = b.idx(j, k, l);
    // index lists per direction: entry 0 is the identity, then the ghost images
    int gx[7], sx[7], gy[7], sy[7], gz[7], sz[7], gye[7], sye[7];
    gx[0] = j, gy[0] = k, gz[0] = l, gye[0] = k;
    sx[0] = sy[0] = sz[0] = sye[0] = -1;
    const int cx = 1 + ghost_images(j, b.nx, fw.flag[0], fw.flag[1], gx + 1, sx + 1);
    const int cy = 1 + ghost_images(k, b.ny, fw.flag[2], fw.flag[3], gy + 1, sy + 1);
    const int cz = 1 + ghost_images(l, b.nz, fw.flag[4], fw.flag[5], gz + 1, sz + 1);
    const int cye = 1 + ghost_images(k, b.ny, fw.flag[2], fw.eps_yout, gye + 1, sye + 1);
    if (cx == 1 && cy == 1 && cz == 1 && cye == 1) return;
    const double gm1 = fw.ggas - 1.0;
    if (j >= 1 && k >= 1 && l >= 1) {  // cell-centred quantities
        double acc[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int z = 0; z < cz; ++z)
            for (int y = 0; y < cy; ++y)
                for (int x = 0; x < cx; ++x) {
                    if (x == 0 && y == 0 && z == 0) continue;
                    const int g = b.idx(gx[x], gy[y], gz[z]);
                    const double lp = o.w[4][g];
                    const double lw[7] = {o.w[0][g] + lp * fw.eps[g] * gm1, o.w[1][g], o.w[2][g], o.w[3][g],
                                          o.bc[0][g], o.bc[1][g], o.bc[2][g]};
#pragma unroll
                    for (int q = 0; q < 7; ++q) {
                        const int qq = q < 4 ? q : IBX + q - 4;
                        const int s = bsign(fw, 0, sx[x], qq) * bsign(fw, 1, sy[y], qq) * bsign(fw, 2, sz[z], qq);
                        acc[q] += s * lw[q];
                    }
                }
        double acce = 0.0;
        for (int z = 0; z < cz; ++z)
            for (int y = 0; y < cye; ++y)
                for (int x = 0; x < cx; ++x) {
                    if (x == 0 && y == 0 && z == 0) continue;
                    const int g = b.idx(gx[x], gye[y], gz[z]);
                    acce += o.eps[g] + o.w[4][g] * fw.w[0][g] * gm1;
                }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (acc[q] != 0.0) o.w[q][i] += acc[q];
#pragma unroll
        for (int q = 0; q < 3; ++q)
            if (acc[4 + q] != 0.0) o.bc[q][i] += acc[4 + q];
        if (acce != 0.0) o.eps[i] += acce;
    }
    // face fields: only the components tangential to a ghost direction move
    if (k >= 1 && l >= 1 && (cy > 1 || cz > 1)) {
        double acc = 0.0;
        for (int z = 0; z < cz; ++z)
            for (int y = 0; y < cy; ++y)
                if (y || z) acc += (bsign(fw, 1, sy[y], IBX) * bsign(fw, 2, sz[z], IBX)) * lbx[b.idx(j, gy[y], gz[z])];
        if (acc != 0.0) lbx[i] += acc;
    }
    if (j >= 1 && l >= 1 && (cx > 1 || cz > 1)) {
        double acc = 0.0;
        for (int z = 0; z < cz; ++z)
            for (int x = 0; x < cx; ++x)
                if (x || z) acc += (bsign(fw, 0, sx[x], IBY) * bsign(fw, 2, sz[z], IBY)) * lby[b.idx(gx[x], k, gz[z])];
        if (acc != 0.0) lby[i] += acc;
    }
    if (j >= 1 && k >= 1 && (cx > 1 || cy > 1)) {
        double acc = 0.0;
        for (int y = 0; y < cy; ++y)
            for (int x = 0; x < cx; ++x)
                if (x || y) acc += (bsign(fw, 0, sx[x], IBZ) * bsign(fw, 1, sy[y], IBZ)) * lbz[b.idx(gx[x], gy[y], l)];
        if (acc != 0.0) lbz[i] += acc;
    }
}

// zero the ghost adjoints k_adj_boundary_gather moved (one thread per ghost,
// the ghost order of k_boundary)
__global__ void __launch_bounds__(256) k_adj_boundary_clear(Box b, BoundArgs fw, AdjPrim o, double* lbx, double* lby,
                                                            double* lbz) {
    const unsigned zp = (unsigned)b.SX * b.SY, yp = (unsigned)b.SX * b.nz, xp = (unsigned)b.ny * b.nz;
    unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    int j, k, l;
    if (t < 6u * zp) {
        const int s = (int)(t / zp), r = (int)(t % zp);
        l = s < 3 ? s - 2 : b.nz + s - 2;
        k = r / b.SX - 2;
        j = r % b.SX - 2;
    } else if ((t -= 6u * zp) < 6u * yp) {
        const int s = (int)(t / yp), r = (int)(t % yp);
        k = s < 3 ? s - 2 : b.ny + s - 2;
        l = r / b.SX + 1;
        j = r % b.SX - 2;
    } else if ((t -= 6u * yp) < 6u * xp) {
        const int s = (int)(t / xp), r = (int)(t % xp);
        j = s < 3 ? s - 2 : b.nx + s - 2;
        l = r / b.ny + 1;
        k = r % b.ny + 1;
    } else {
        return;
    }
    const int i = b.idx(j, k, l);
    const bool gx = j < 1 || j > b.nx, gy = k < 1 || k > b.ny, gz = l < 1 || l > b.nz;
#pragma unroll
    for (int q = 0; q < 5; ++q) o.w[q][i] = 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) o.bc[q][i] = 0.0;
    o.eps[i] = 0.0;
    if (j >= 0 && j <= b.nx && (gy || gz)) lbx[i] = 0.0;
    if (k >= 0 && k <= b.ny && (gx || gz)) lby[i] = 0.0;
    if (l >= 0 && l <= b.nz && (gx || gy)) lbz[i] = 0.0;
}

// the primitives (before the boundary fill) and face fields of a taped combine
// output src, into a scratch state: k_utop on the tape's own arrays, without a
// copy of them first. The scratch state's hydro cons are not read.
template <int MODEL>
__global__ void __launch_bounds__(256) k_adj_prims(Box b, Arr8 src, UtopArgs a) {
    int j, k, l, i;
    if (!box1_index(b, j, k, l, i)) return;
    const bool interior = j >= 1 && k >= 1 && l >= 1;
    const int off[3] = {1, b.SX, b.SX * b.SY};
    double uh[5], bc[3];
#pragma unroll
    for (int q = 0; q < 5; ++q) uh[q] = src.a[q][i];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double f = src.a[IBX + q][i];
        a.u[IBX + q][i] = f;
        bc[q] = interior ? 0.5 * (f + src.a[IBX + q][i - off[q]]) : a.bc[q][i];
        if (interior) a.bc[q][i] = bc[q];
    }
    const CellConv o =
        utop_of<MODEL, true, true>(uh, interior, bc[0], bc[1], bc[2], a.ggas, a.rho_floor, a.eps_floor);
#pragma unroll
    for (int q = 0; q < 4; ++q) a.w[q][i] = o.w[q];
    a.eps[i] = o.eps;
    if (interior) {
        a.w[4][i] = o.p;
        if (o.bad) atomicOr(a.flag, 1u);
    }
}

// utop^T on the active cells: from the adjoints of the re-derived conserved
// hydro variables (lu) and of the primitives (o), the adjoint of the
// combine's output Upre (hydro part, mu) and of the cell-centred field
// (lb, folded onto the faces by k_adj_bface). FROMUTORVE, CHECKRHO (RIEMANN:
// eps >= 0, branch frozen), FROMRVETOU and UPDATE's pressure
// (solver/fromrvetou.f90:21-127, solver/update.f90:27-35). FROM_CONS=false is
// initial_update, whose inputs are the uploaded rho, v and eps: mu then
// receives (rho, vx, vy, vz, eps) adjoints.
template <int MODEL, bool FROM_CONS>
__global__ void __launch_bounds__(256) k_adj_utop(Box b, Arr8 u, Arr8 w0, const double* eps0, Arr8 lu,
                                                  AdjPrim o, double ggas, Arr8 mu, Arr3 lb, double alpha,
                                                  double beta, Arr8 lam0, bool first) {
    const int n0 = b.nx + 1, n1 = b.ny + 1, n2 = b.nz + 1;
    const long long total = (long long)n0 * n1 * n2;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int j = (int)(t % n0), k = (int)((t / n0) % n1), l = (int)(t / n0 / n1);
    const int i = b.idx(j, k, l);
    if (!(j >= 1 && k >= 1 && l >= 1)) {
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            mu.a[q][i] = 0.0;
            if (beta != 0.0) lu.a[q][i] = 0.0;
            if (FROM_CONS && first) lam0.a[q][i] = 0.0;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) lb.a[q][i] = 0.0;
        return;
    }
    const double bx = 0.5 * (u.a[IBX][i] + u.a[IBX][i - 1]);
    const double by = 0.5 * (u.a[IBY][i] + u.a[IBY][i - b.SX]);
    const double bz = 0.5 * (u.a[IBZ][i] + u.a[IBZ][i - b.SX * b.SY]);
    const double bsquare = (bx * bx + by * by) + bz * bz;
    double rho, vx, vy, vz, e_raw, ir = 0.0, eb = 0.0;  // ir = 1/rho, eb = (E - bsq/2)/rho
    if (FROM_CONS) {
        rho = u.a[IRHO][i];
        ir = 1.0 / rho;
        const double n[4] = {u.a[IVX][i], u.a[IVY][i], u.a[IVZ][i], u.a[ITAU][i] - 0.5 * bsquare};
        double q[4];
        quot_group(n, rho, q);  // the forward's values: e_raw decides a branch
        vx = q[0];
        vy = q[1];
        vz = q[2];
        eb = q[3];
        e_raw = eb - 0.5 * ((vx * vx + vy * vy) + vz * vz);
    } else {
        rho = w0.a[0][i];
        vx = w0.a[1][i];
        vy = w0.a[2][i];
        vz = w0.a[3][i];
        e_raw = eps0[i];
    }
    const bool clamped = MODEL == 1 && !(e_raw >= 0.0);
    const double e = clamped ? 0.0 : e_raw;
    const double vsquare = (vx * vx + vy * vy) + vz * vz;
    const double g1 = ggas - 1.0;
    // adjoint inputs
    const double lu0 = lu.a[IRHO][i], lu1 = lu.a[IVX][i], lu2 = lu.a[IVY][i], lu3 = lu.a[IVZ][i], lu4 = lu.a[ITAU][i];
    const double lp = o.w[4][i];
    double Lrho = lu0 + o.w[0][i] + lu1 * vx + lu2 * vy + lu3 * vz + lu4 * (e + 0.5 * vsquare) + lp * e * g1;
    double Lvx = o.w[1][i] + lu1 * rho, Lvy = o.w[2][i] + lu2 * rho, Lvz = o.w[3][i] + lu3 * rho;
    double Le = o.eps[i] + lu4 * rho + lp * rho * g1;
    double Lvsq = lu4 * 0.5 * rho;
    double Lbsq = 0.5 * lu4;
    if (clamped) Le = 0.0;
    if (FROM_CONS) {
        // e_raw = (E - bsq/2)/rho - vsq/2
        const double LE = Le * ir;
        Lbsq -= 0.5 * LE;
        Lrho -= LE * eb;
        Lvsq -= 0.5 * Le;
        Lvx += 2.0 * vx * Lvsq;
        Lvy += 2.0 * vy * Lvsq;
        Lvz += 2.0 * vz * Lvsq;
        // v = m / rho
        mu.a[IVX][i] = Lvx * ir;
        mu.a[IVY][i] = Lvy * ir;
        mu.a[IVZ][i] = Lvz * ir;
        Lrho -= (Lvx * vx + Lvy * vy + Lvz * vz) * ir;
        mu.a[IRHO][i] = Lrho;
        mu.a[ITAU][i] = LE;
    } else {
        Lvx += 2.0 * vx * Lvsq;
        Lvy += 2.0 * vy * Lvsq;
        Lvz += 2.0 * vz * Lvsq;
        mu.a[0][i] = Lrho;
        mu.a[1][i] = Lvx;
        mu.a[2][i] = Lvy;
        mu.a[3][i] = Lvz;
        mu.a[4][i] = Le;  // adjoint of the uploaded eps
    }
    lb.a[0][i] = o.bc[0][i] + 2.0 * bx * Lbsq;
    lb.a[1][i] = o.bc[1][i] + 2.0 * by * Lbsq;
    lb.a[2][i] = o.bc[2][i] + 2.0 * bz * Lbsq;
    // combine^T of the hydro part: Upre = alpha U0 + beta U_prev + ...; the
    // adjoint of U_prev replaces lu (read above by this thread only)
    if (FROM_CONS && (alpha != 0.0 || beta != 0.0)) {
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const double m = mu.a[q][i];
            lam0.a[q][i] = first ? alpha * m : lam0.a[q][i] + alpha * m;
            if (beta != 0.0) lu.a[q][i] = beta * m;
        }
    }
    // the primitive adjoints are spent (the boundary's transpose has cleared the
    // ghosts'): cleared here for the next stage to add to
    if (FROM_CONS) {
#pragma unroll
        for (int q = 0; q < 5; ++q) o.w[q][i] = 0.0;
#pragma unroll
        for (int q = 0; q < 3; ++q) o.bc[q][i] = 0.0;
        o.eps[i] = 0.0;
    }
}

// face-field adjoint on (0:n)^3: the pass-through adjoint of the live face
// values plus half the adjoints of the two active cells whose bcell average
// reads the face (solver/fromrvetou.f90:97-107); zero on every other entry
__global__ void __launch_bounds__(256) k_adj_bface(Box b, Arr3 lbf, Arr3 lb, Arr3 out, double alpha, double beta,
                                                   Arr3 lam0, bool first) {
    const int n0 = b.nx + 1, n1 = b.ny + 1, n2 = b.nz + 1;
    const long long total = (long long)n0 * n1 * n2;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int j = (int)(t % n0), k = (int)((t / n0) % n1), l = (int)(t / n0 / n1);
    const int i = b.idx(j, k, l);
    const int st[3] = {1, b.SX, b.SX * b.SY};
    const int own[3] = {j, k, l};
    const int nn[3] = {b.nx, b.ny, b.nz};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        bool live = true;
#pragma unroll
        for (int e = 0; e < 3; ++e)
            if (e != d && (own[e] < 1 || own[e] > nn[e])) live = false;
        double v = 0.0;
        if (live) {
            v = lbf.a[d][i];
            const double left = own[d] >= 1 ? lb.a[d][i] : 0.0;
            const double right = own[d] + 1 <= nn[d] ? lb.a[d][i + st[d]] : 0.0;
            v += 0.5 * (left + right);
        }
        out.a[d][i] = v;
        // combine^T of the field part (lbf, read above by this thread only,
        // becomes the adjoint of the previous stage's face field)
        if (alpha != 0.0) lam0.a[d][i] = first ? alpha * v : lam0.a[d][i] + alpha * v;
        if (beta != 0.0) lbf.a[d][i] = beta * v;
    }
}

// objective at the final state, per-block partial sums (deterministic order)
// and its adjoint seed. kind 1: magnetic energy 0.5 sum |bcell|^2 dV; kind 2:
// kinetic energy 0.5 sum rho |v|^2 dV; kind 3: sum of weights . cons over the
// live entries (weights in lamu on entry).
__global__ void __launch_bounds__(256) k_adj_objective(Box b, Tabs T, int coord, Prim pr, Arr8 u, int kind, AdjPrim o,
                                                       Arr8 lamu, double* partial) {
    const long long total = (long long)b.nx * b.ny * b.nz;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    double acc = 0.0;
    if (t < total) {
        const int j = (int)(t % b.nx) + 1, k = (int)((t / b.nx) % b.ny) + 1, l = (int)(t / b.nx / b.ny) + 1;
        const int i = b.idx(j, k, l);
        // cell volume: dx dy dz; R dR dphi dz; (r^3)/3 d(-cos theta) dphi
        const double dv = coord == CUMC_CARTESIAN     ? (T.ax[0].d[j] * T.ax[1].d[k]) * T.ax[2].d[l]
                          : coord == CUMC_CYLINDRICAL ? ((T.ax[0].c[j] * T.ax[0].d[j]) * T.ax[1].d[k]) * T.ax[2].d[l]
                                                      : (T.r3d3[j] * T.dcos[k]) * T.ax[2].d[l];
        if (kind == 1) {
            const double bx = pr.bc[0][i], by = pr.bc[1][i], bz = pr.bc[2][i];
            acc = 0.5 * ((bx * bx + by * by) + bz * bz) * dv;
            o.bc[0][i] += bx * dv;
            o.bc[1][i] += by * dv;
            o.bc[2][i] += bz * dv;
        } else if (kind == 2) {
            const double rho = pr.w[0][i], vx = pr.w[1][i], vy = pr.w[2][i], vz = pr.w[3][i];
            const double vsq = (vx * vx + vy * vy) + vz * vz;
            acc = 0.5 * rho * vsq * dv;
            o.w[0][i] += 0.5 * vsq * dv;
            o.w[1][i] += rho * vx * dv;
            o.w[2][i] += rho * vy * dv;
            o.w[3][i] += rho * vz * dv;
        } else {
            for (int q = 0; q < 5; ++q) acc += lamu.a[q][i] * u.a[q][i];
            // face fields: the cell's own faces (index 1:n) plus the lower boundary faces (index 0)
            const int st[3] = {1, b.SX, b.SX * b.SY};
            const int own[3] = {j, k, l};
            for (int d = 0; d < 3; ++d) {
                acc += lamu.a[IBX + d][i] * u.a[IBX + d][i];
                if (own[d] == 1) acc += lamu.a[IBX + d][i - st[d]] * u.a[IBX + d][i - st[d]];
            }
        }
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
    __shared__ double red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += red[w];
        partial[blockIdx.x] = v;
    }
}

// clears the weights of a linear objective off its live entries
__global__ void __launch_bounds__(256) k_adj_mask_live(Box b, Arr8 lamu) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= b.count()) return;
    const int j = (int)(t % b.SX) - 2, k = (int)((t / b.SX) % b.SY) - 2, l = (int)(t / b.SX / b.SY) - 2;
    const int own[3] = {j, k, l};
    const int nn[3] = {b.nx, b.ny, b.nz};
    const bool cell = inside(j, k, l, b);
    for (int q = 0; q < 5; ++q)
        if (!cell) lamu.a[q][t] = 0.0;
    for (int d = 0; d < 3; ++d) {
        bool live = own[d] >= 0 && own[d] <= nn[d];
        for (int e = 0; e < 3; ++e)
            if (e != d && (own[e] < 1 || own[e] > nn[e])) live = false;
        if (!live) lamu.a[IBX + d][t] = 0.0;
    }
}

// one block: sum of n partial sums in a fixed order
__global__ void __launch_bounds__(256) k_adj_sum(const double* partial, int n, double* out) {
    double acc = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) acc += partial[i];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
    __shared__ double red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += red[w];
        *out = v;
    }
}

}  // namespace cumc
