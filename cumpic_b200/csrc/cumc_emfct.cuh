// cumc_emfct.cuh — edge EMFs and the constrained-transport update of the
// face fields in one kernel (the EMF sums of GET_FLUXES,
// solver/spatial.f90:190-203,268-281,346-359, flux_ct's ecell/ecorn,
// solver/mhd.f90:95-125, its curl, :130-153, and the RK combine of the face
// fields, solver/rungekutta.f90:41-51,75-85,109-119).
//
// k_emf writes the three edge-EMF arrays and k_ct reads them back at six
// neighbouring edges a face triple. Here a block owns a tile of 32 x 4 face
// triples (x fastest) and marches in z over a segment of planes. Per plane
// it forms, in shared memory, the cell EMFs E = -v x B of the cells the
// plane's edges average, then the edge EMFs of the tile and of the halo row
// and column its CT reads (Ez at j-1 and k-1; Ey at j-1; Ex at k-1), and
// keeps the x and y edge EMFs of the previous plane (the l-1 edges of CT).
// Each cell EMF is formed at most 1.6 times, each edge EMF 1.3 times.
// Edges with an index of -1 are zero, as the never-written entries of the
// edge arrays are for k_ct. Every value is the same expression, in the same
// order, as in k_emf and k_ct, so the result is bit for bit theirs.
#pragma once
#include "cumc_kernels.cuh"

namespace cumc {

// Face triples of a tile. Smaller tiles form more halo edges and cells (1.29
// and 1.59 a triple at 32 x 4, 1.16 and 1.33 at 32 x 8), but a block waits at
// its barriers for fewer warps. 32 x 8 -> 32 x 4: 0.717 -> 0.675 ms a stage at
// 256^3, 0.115 -> 0.091 on the 192x128x64 torus, 0.027 -> 0.023 at 64^3; 32 x 2
// takes 0.76, 0.098 and 0.025.
#ifndef CUMC_EC_TY
#define CUMC_EC_TY 4
#endif
constexpr int EC_TX = 32, EC_TY = CUMC_EC_TY;
constexpr int EC_CX = EC_TX + 2, EC_CY = EC_TY + 2;  // cells j0-1..j0+32, k0-1..k0+4
constexpr int EC_EX = EC_TX + 1, EC_EY = EC_TY + 1;  // edges j0-1..j0+31, k0-1..k0+3

__host__ __device__ __forceinline__ int ec_tiles_x(const Box& b) { return (b.nx + 1 + EC_TX - 1) / EC_TX; }

// shared memory of a tile; R is the EMFs' type (double, or float in the
// mixed form)
template <typename R>
struct EmfCtSmemT {
    R ec[2][3][EC_CY][EC_CX];   // cell EMFs of two planes (ring by plane parity)
    R ex[2][EC_EY][EC_EX];      // x edge EMFs of two planes (ring by plane parity)
    R ey[2][EC_EY][EC_EX];      // y edge EMFs of two planes
    R ez[EC_EY][EC_EX];         // z edge EMFs of the current plane
};
using EmfCtSmem = EmfCtSmemT<double>;

// cell EMFs of plane l for the tile's cells (zero outside -1..n+1)
template <typename R>
__device__ __forceinline__ void ec_cells(const Box& b, const PrimT<R>& pr, EmfCtSmemT<R>& S, int j0, int k0, int l) {
    const int slot = l & 1;
    for (int t = threadIdx.x; t < EC_CX * EC_CY; t += EC_TX * EC_TY) {
        const int cj = t % EC_CX, ck = t / EC_CX;
        const int j = j0 - 1 + cj, k = k0 - 1 + ck;
        R x = R(0), y = R(0), z = R(0);
        if (j <= b.nx + 1 && k <= b.ny + 1 && l >= -1 && l <= b.nz + 1) {
            const int i = b.idx(j, k, l);
            x = ecell_x(pr, i);
            y = ecell_y(pr, i);
            z = ecell_z(pr, i);
        }
        S.ec[slot][0][ck][cj] = x;
        S.ec[slot][1][ck][cj] = y;
        S.ec[slot][2][ck][cj] = z;
    }
}

// edge EMFs of plane l (x and y edges into their ring slot; z edges with `z`)
template <typename R>
__device__ __forceinline__ void ec_edges(const Box& b, const FaceFluxT<R>& fx, const FaceFluxT<R>& fy,
                                         const FaceFluxT<R>& fz, EmfCtSmemT<R>& S, int j0, int k0, int l, bool z) {
    const int sj = 1, sk = b.SX, sl = b.SX * b.SY;
    const R q = R(0.25);
    const int c0 = l & 1, c1 = (l + 1) & 1;  // cell-EMF slots of planes l and l+1
    const int e = l & 1;
    for (int t = threadIdx.x; t < EC_EX * EC_EY; t += EC_TX * EC_TY) {
        const int ej = t % EC_EX, ek = t / EC_EX;  // edge (j0 - 1 + ej, k0 - 1 + ek)
        const int j = j0 - 1 + ej, k = k0 - 1 + ek;
        const bool live = j >= 0 && k >= 0 && l >= 0 && j <= b.nx && k <= b.ny && l <= b.nz;
        const int i = live ? b.idx(j, k, l) : 0;
        // cell (j, k) of the edge is cell slot (ck, cj) = (ek, ej): the edge sits
        // at the upper faces of cells j and k
        const int cj = ej, ck = ek;
        R ex = R(0), ey = R(0), ez = R(0);
        if (live) {
            ex = R(0) + q * (-fy.f[6][i] - fy.f[6][i + sl]);
            ex = ex + q * (fz.f[6][i] + fz.f[6][i + sk]);
            ey = R(0) + q * (fx.f[6][i] + fx.f[6][i + sl]);
            ey = ey + q * (-fz.f[5][i] - fz.f[5][i + sj]);
            // k_emf's sums: cells (j,k,l), (j,k,l+1), (j,k+1,l), (j,k+1,l+1) for Ex;
            // (j,k,l), (j,k,l+1), (j+1,k,l), (j+1,k,l+1) for Ey; (j,k), (j,k+1),
            // (j+1,k), (j+1,k+1) of plane l for Ez
            ex = ex * R(2) - q * (((S.ec[c0][0][ck][cj] + S.ec[c1][0][ck][cj]) + S.ec[c0][0][ck + 1][cj]) +
                                 S.ec[c1][0][ck + 1][cj]);
            ey = ey * R(2) - q * (((S.ec[c0][1][ck][cj] + S.ec[c1][1][ck][cj]) + S.ec[c0][1][ck][cj + 1]) +
                                 S.ec[c1][1][ck][cj + 1]);
            if (z) {
                ez = R(0) + q * (-fx.f[5][i] - fx.f[5][i + sk]);
                ez = ez + q * (fy.f[5][i] + fy.f[5][i + sj]);
                ez = ez * R(2) - q * (((S.ec[c0][2][ck][cj] + S.ec[c0][2][ck + 1][cj]) + S.ec[c0][2][ck][cj + 1]) +
                                     S.ec[c0][2][ck + 1][cj + 1]);
            }
        }
        S.ex[e][ek][ej] = ex;
        S.ey[e][ek][ej] = ey;
        if (z) S.ez[ek][ej] = ez;
    }
}

// the flux half of one edge's three EMFs (the first two sums of each, k_emf's
// order); the cell-EMF half is added once the plane's cell EMFs are in
// shared memory (ec_edge_finish)
template <typename R>
struct EdgePart {
    R x, y, z;
};
template <typename R>
__device__ __forceinline__ EdgePart<R> ec_edge_part(const Box& b, const FaceFluxT<R>& fx, const FaceFluxT<R>& fy,
                                                    const FaceFluxT<R>& fz, int j0, int k0, int l, int t) {
    const int sj = 1, sk = b.SX, sl = b.SX * b.SY;
    const R q = R(0.25);
    const int j = j0 - 1 + t % EC_EX, k = k0 - 1 + t / EC_EX;
    EdgePart<R> e{R(0), R(0), R(0)};
    if (j >= 0 && k >= 0 && j <= b.nx && k <= b.ny && l <= b.nz) {
        const int i = b.idx(j, k, l);
        e.x = R(0) + q * (-fy.f[6][i] - fy.f[6][i + sl]);
        e.x = e.x + q * (fz.f[6][i] + fz.f[6][i + sk]);
        e.y = R(0) + q * (fx.f[6][i] + fx.f[6][i + sl]);
        e.y = e.y + q * (-fz.f[5][i] - fz.f[5][i + sj]);
        e.z = R(0) + q * (-fx.f[5][i] - fx.f[5][i + sk]);
        e.z = e.z + q * (fy.f[5][i] + fy.f[5][i + sj]);
    }
    return e;
}
template <typename R>
__device__ __forceinline__ void ec_edge_finish(const Box& b, EmfCtSmemT<R>& S, const EdgePart<R>& e, int j0, int k0,
                                               int l, int t) {
    const R q = R(0.25);
    const int ej = t % EC_EX, ek = t / EC_EX;
    const int j = j0 - 1 + ej, k = k0 - 1 + ek;
    const bool live = j >= 0 && k >= 0 && j <= b.nx && k <= b.ny && l <= b.nz;
    const int c0 = l & 1, c1 = (l + 1) & 1, cj = ej, ck = ek;
    R ex = R(0), ey = R(0), ez = R(0);
    if (live) {
        ex = e.x * R(2) - q * (((S.ec[c0][0][ck][cj] + S.ec[c1][0][ck][cj]) + S.ec[c0][0][ck + 1][cj]) +
                               S.ec[c1][0][ck + 1][cj]);
        ey = e.y * R(2) - q * (((S.ec[c0][1][ck][cj] + S.ec[c1][1][ck][cj]) + S.ec[c0][1][ck][cj + 1]) +
                               S.ec[c1][1][ck][cj + 1]);
        ez = e.z * R(2) - q * (((S.ec[c0][2][ck][cj] + S.ec[c0][2][ck + 1][cj]) + S.ec[c0][2][ck][cj + 1]) +
                               S.ec[c0][2][ck + 1][cj + 1]);
    }
    S.ex[l & 1][ek][ej] = ex;
    S.ey[l & 1][ek][ej] = ey;
    S.ez[ek][ej] = ez;
}

// ct_lrk (solver/mhd.f90:137-148) from the nine edge EMFs around a face triple:
// the six quotients of ct_lrk, bit for bit, through quot_group (on Cartesian
// grids two share each width)
template <int COORD>
__device__ __forceinline__ void ct_curl(const CTf& g, double Ex, double Ex_lm, double Ex_km, double Ey, double Ey_lm,
                                        double Ey_jm, double Ez, double Ez_km, double Ez_jm, double (&L)[3]) {
    const double nxz = Ez * g.bx_ez_p - Ez_km * g.bx_ez_m, nxy = Ey * g.bx_ey_p - Ey_lm * g.bx_ey_m;
    const double nyx = Ex * g.by_ex_p - Ex_lm * g.by_ex_m, nyz = Ez * g.by_ez_p - Ez_jm * g.by_ez_m;
    const double nzy = Ey * g.bz_ey_p - Ey_jm * g.bz_ey_m, nzx = Ex * g.bz_ex_p - Ex_km * g.bz_ex_m;
    double qx[2], qy[2], qz[2];  // by the widths along x, y, z
    if constexpr (COORD == 1) {
        const double ax[2] = {nyz, nzy}, ay[2] = {nxz, nzx}, az[2] = {nxy, nyx};
        quot_group(ax, g.by_ez_c, qx);
        quot_group(ay, g.bx_ez_c, qy);
        quot_group(az, g.bx_ey_c, qz);
    } else {
        auto one = [](double a, double b) {
            const double n[1] = {a};
            double q[1];
            quot_group(n, b, q);
            return q[0];
        };
        qx[0] = one(nyz, g.by_ez_c);
        qx[1] = one(nzy, g.bz_ey_c);
        qy[0] = one(nxz, g.bx_ez_c);
        qy[1] = one(nzx, g.bz_ex_c);
        qz[0] = one(nxy, g.bx_ey_c);
        qz[1] = one(nyx, g.by_ex_c);
    }
    L[0] = -(qy[0] - qz[0]);
    L[1] = -(qz[1] - qx[0]);
    L[2] = -(qx[1] - qy[1]);
}

// Per plane a thread first issues its global loads (the flux half of its
// edges, u_old and u of its face triple, the cell fields of its cells of the
// next plane), so that one memory latency a plane is exposed instead of
// three. Two barriers a plane: the next plane's cell EMFs overwrite the slot
// of plane l-1's cells, read only before this plane's second barrier, and
// its edges overwrite slots that CT reads, which every thread has finished
// before it reaches the next plane's first barrier.
#ifndef CUMC_EC_MINB
#define CUMC_EC_MINB 8
#endif
template <int COORD, int STAGE>
__global__ void __launch_bounds__(EC_TX * EC_TY, CUMC_EC_MINB) k_emf_ct(Box b, Tabs T, Prim pr, FaceFlux fx,
                                                                      FaceFlux fy, FaceFlux fz, CombineArgs a,
                                                                      int seg) {
    extern __shared__ __align__(16) unsigned char ec_raw[];
    EmfCtSmem& S = *reinterpret_cast<EmfCtSmem*>(ec_raw);
    if (b.skip && *b.skip) return;
    constexpr int NE = EC_EX * EC_EY, NT = EC_TX * EC_TY;
    static_assert(NE > NT && NE <= 2 * NT, "two edges a thread at most");
    const int tx = ec_tiles_x(b), j0 = (int)(blockIdx.x % tx) * EC_TX, k0 = (int)(blockIdx.x / tx) * EC_TY;
    const int l0 = blockIdx.y * seg, l1 = min(l0 + seg, b.nz + 1);
    const int tj = threadIdx.x % EC_TX, tk = threadIdx.x / EC_TX;
    const int j = j0 + tj, k = k0 + tk;
    const bool mine = j <= b.nx && k <= b.ny;
    const int e0 = threadIdx.x, e1 = threadIdx.x + NT;  // the thread's edges (e1 < NE for some)
    const double dt = *a.dt;

    // prologue: the x and y edges of plane l0 - 1 (zero for l0 = 0)
    ec_cells(b, pr, S, j0, k0, l0 - 1);
    ec_cells(b, pr, S, j0, k0, l0);
    __syncthreads();
    ec_edges(b, fx, fy, fz, S, j0, k0, l0 - 1, false);
    __syncthreads();
    for (int l = l0; l < l1; ++l) {
        const EdgePart<double> p0 = ec_edge_part(b, fx, fy, fz, j0, k0, l, e0);
        const EdgePart<double> p1 = e1 < NE ? ec_edge_part(b, fx, fy, fz, j0, k0, l, e1) : EdgePart<double>{0.0, 0.0, 0.0};
        double u0v[3] = {0.0, 0.0, 0.0}, ucv[3] = {0.0, 0.0, 0.0};
        const int i = b.idx(j, k, l);
        if (mine) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                u0v[c] = a.u0[IBX + c][i];
                if (STAGE != 1) ucv[c] = a.uc[IBX + c][i];
            }
        }
        ec_cells(b, pr, S, j0, k0, l + 1);  // replaces plane l - 1's cells
        __syncthreads();
        ec_edge_finish(b, S, p0, j0, k0, l, e0);
        if (e1 < NE) ec_edge_finish(b, S, p1, j0, k0, l, e1);
        __syncthreads();
        if (mine) {
            // ct_lrk (solver/mhd.f90:137-148) on the shared-memory edges; the tile's
            // (tj, tk) is edge (tj + 1, tk + 1)
            const int ej = tj + 1, ek = tk + 1, e = l & 1, em = (l - 1) & 1;
            const double Ez = S.ez[ek][ej], Ez_km = S.ez[ek - 1][ej], Ez_jm = S.ez[ek][ej - 1];
            const double Ey = S.ey[e][ek][ej], Ey_lm = S.ey[em][ek][ej], Ey_jm = S.ey[e][ek][ej - 1];
            const double Ex = S.ex[e][ek][ej], Ex_lm = S.ex[em][ek][ej], Ex_km = S.ex[e][ek - 1][ej];
            CTf g;
            geom_ct<COORD>(T, j, k, l, g);
            double L[3];
            ct_curl<COORD>(g, Ex, Ex_lm, Ex_km, Ey, Ey_lm, Ey_jm, Ez, Ez_km, Ez_jm, L);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double r = rk_point<STAGE>(u0v[c], ucv[c], dt, L[c]);
                a.ud[IBX + c][i] = r;
                if (a.tape[IBX + c]) a.tape[IBX + c][i] = r;
            }
        }
    }
}

// Grid of a tiled EMF + CT launch and the planes a block marches over: the
// segment length that makes (rounds of `slots` resident blocks) x (planes + 1)
// least; each segment repeats one plane of cell and edge EMFs. Against 32 planes
// halved down to 4 (and the plain quotients in the curl): 192x128x64 torus 0.129
// -> 0.115 ms, the 90x26x75 one 0.029 -> 0.019, a 512x4x4 tube 0.020 -> 0.011,
// 256^3 0.73 -> 0.72.
// (x tile fastest, then y, in the grid's first dimension: the others end at
// 65,535.)
inline dim3 emf_ct_grid(const Box& b, long long slots, int* seg) {
    const long long tiles = (long long)ec_tiles_x(b) * ((b.ny + 1 + EC_TY - 1) / EC_TY);
    int count;
    *seg = segment_length(b.nz + 1, tiles, slots, 1, 1, b.nz + 1, &count);
    return dim3((unsigned)tiles, (unsigned)count);
}

}  // namespace cumc
