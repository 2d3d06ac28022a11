// cumc_walk.cuh — column-walking directional sweeps
// (GET_FLUXES interpolate + RIEMANN, solver/spatial.f90:170-324).
//
// Each thread owns one column (a fixed pair of transverse indices) and walks
// along the sweep direction over a segment of faces. A sliding window of
// five values per reconstructed field is carried from face f to face f+1:
//   v(f+1), v(f+2), the limited slope of cell f+1, the interface value
//   between cells f and f+1, and vp_out(f).
// Per face the thread loads one new cell per field, forms one limited slope,
// one interface value and one extremum fix, and solves one HLL problem. Every
// quantity the reference evaluates several times per cell
// (solver/reconstruct.f90:254-307) is formed exactly once, with the
// reference's expression trees, so the fluxes are bit-identical to the
// per-face evaluation. Only the segment prologue (three slopes, two interface
// values, one fix) is repeated per segment.
//
// Two storage forms of the window:
//   k_sweep_walk     window in registers (168 registers a thread in FP64,
//                    which caps residency near 12 warps per SM);
//   k_sweep_walk_sm  window in shared memory, one private slot column per
//                    thread ([slot][field][thread], so a warp's accesses are
//                    conflict-free), which frees about 70 registers a thread.
// Along y and z consecutive threads hold consecutive x, so every load is
// coalesced. Along x consecutive threads hold consecutive y rows; each load
// touches one 32-byte sector per row, which the following three faces reuse
// from L1.
#pragma once
#include "cumc_kernels.cuh"

namespace cumc {

constexpr int WK_THREADS = 64;
// resident blocks per SM the walker and the lane-per-cell x sweep are compiled
// for (the register budget a thread gets); build-time tunables. The walker's 9
// blocks of 64 get 96 registers, and 10 fit: 0.90 ms a stage at 256^3, FP64 pipe
// 60 % busy; 7 and 8 blocks (128 registers) take 0.91, 11 and 12 (80) 0.93-0.94.
#ifndef CUMC_WALK_MINB
#define CUMC_WALK_MINB 9
#endif
#ifndef CUMC_XWARP_MINB
#define CUMC_XWARP_MINB 8
#endif
constexpr int WK_FIELDS = 7;  // rho, vx, vy, vz, p and the two tangential cell fields

template <int DIR>
struct WalkGeom {
    static_assert(DIR >= 0 && DIR <= 2, "sweep direction");
    __host__ __device__ static int nd(const Box& b) { return DIR == 0 ? b.nx : DIR == 1 ? b.ny : b.nz; }
    // transverse widths: a is the fast column index, c the slow one (each 0:n+1)
    __host__ __device__ static int wa(const Box& b) { return DIR == 0 ? b.ny + 2 : b.nx + 2; }
    __host__ __device__ static int wc(const Box& b) { return DIR == 2 ? b.ny + 2 : b.nz + 2; }
    __host__ __device__ static int stride(const Box& b) { return DIR == 0 ? 1 : DIR == 1 ? b.SX : b.SX * b.SY; }
    __host__ __device__ static long long ncols(const Box& b) { return (long long)wa(b) * wc(b); }
    __device__ static int idx(const Box& b, int a, int c, int f) {
        return DIR == 0 ? b.idx(f, a, c) : DIR == 1 ? b.idx(a, f, c) : b.idx(a, c, f);
    }
};

// Segments of a walk along DIR over `ncols` columns. Equal blocks run in
// rounds of the WK_RESIDENT blocks a SM that fit (96 registers and 17.5 KB of
// shared memory a 64-thread block with PPM, 14 KB with TVD), and a segment costs its faces plus a
// prologue (three slopes, two interface values and a fix a field, and a
// memory latency: about one and a half faces), so the count is taken that
// makes rounds x (faces + 1.5) least. Against about 64 faces, halved down to
// 8 while the grid gave fewer than 32 warps a SM: 64^3 0.036 -> 0.029 ms a
// walk, the 90x26x75 torus 0.029 -> 0.023, a 512x4x4 tube 0.021 -> 0.013; 256^3
// unchanged (0.90). In a step's graph, where the three sweeps run side by side,
// ms a step with that rule, this one, and this one with a third of the GPU a
// sweep: 64^3 0.331, 0.328, 0.340; tube 0.125, 0.111, 0.111; 90x26x75 0.271,
// 0.263, 0.266; 192x128x64 torus 1.720, 1.713, 1.702; 128^3 reciprocal solve
// 1.760, 1.770, 1.781.
constexpr int WK_RESIDENT = 10, WK_SEG_MAX = 64;  // (64 faces: 1.5 KB of FP32 weights a mixed block)
template <int DIR>
inline int walk_segment_for(const Box& b, long long ncols, int sm_count, int* nseg) {
    const int faces = WalkGeom<DIR>::nd(b) + 1;
    const long long blocks = (ncols + WK_THREADS - 1) / WK_THREADS, slots = (long long)sm_count * WK_RESIDENT;
    return segment_length(faces, blocks, slots, 2, 3, WK_SEG_MAX, nseg);
}

// cell index 0 (along DIR) of column `col` of the block's grid, clamped to
// the last column so that the spare threads of the last block stay in bounds
template <int DIR>
__device__ __forceinline__ int walk_base(const Box& b, long long col) {
    using G = WalkGeom<DIR>;
    col = min(col, G::ncols(b) - 1);
    return G::idx(b, (int)(col % G::wa(b)), (int)(col / G::wa(b)), 0);
}

// column set-up shared by both window forms. Every thread of a block stays
// to the end (the x sweep synchronises the block); threads past the last
// column walk a copy of it and store nothing. The columns are those whose
// slow transverse index is c_lo, c_lo + c_step, .. (c_cnt of them; c_cnt < 0:
// all).
template <int DIR, typename R>
struct WalkCol {
    int base, s, f0, f1, nd;
    bool active;
    const R* src[WK_FIELDS];
    int slot[WK_FIELDS];
    const R* bn;
    __device__ bool init(const Box& b, const PrimT<R>& pr, int seg, int c_lo = 0, int c_cnt = -1, int c_step = 1) {
        using G = WalkGeom<DIR>;
        if (b.skip && *b.skip) return false;
        if (c_cnt < 0) c_cnt = G::wc(b);
        const long long ncols = (long long)G::wa(b) * c_cnt;
        const long long col = (long long)blockIdx.x * WK_THREADS + threadIdx.x;
        active = col < ncols;
        nd = G::nd(b);
        f0 = blockIdx.y * seg;
        if (f0 > nd) return false;
        f1 = min(f0 + seg, nd + 1);
        s = G::stride(b);
        const unsigned cc = (unsigned)min(col, ncols - 1);  // fewer columns than cells: 32-bit division
        base = G::idx(b, (int)(cc % G::wa(b)), c_lo + c_step * (int)(cc / G::wa(b)), 0);
        // tangential cell fields: (by, bz) for x, (bx, bz) for y, (bx, by) for z
        constexpr int ta = DIR == 0 ? 1 : 0;
        constexpr int tb = DIR == 2 ? 1 : 2;
        const R* s7[WK_FIELDS] = {pr.w[0], pr.w[1], pr.w[2], pr.w[3], pr.w[4], pr.bc[ta], pr.bc[tb]};
        const int q7[WK_FIELDS] = {IRHO, IVX, IVY, IVZ, ITAU, IBX + ta, IBX + tb};
#pragma unroll
        for (int v = 0; v < WK_FIELDS; ++v) {
            src[v] = s7[v] + base;
            slot[v] = q7[v];
        }
        bn = pr.bf[DIR] + base;
        return true;
    }
};

// x-sweep staging. Along x a thread's column is a row of the array, so a
// direct load by a warp touches 32 rows. Instead the block stages its 64
// rows through shared memory in chunks of XS_CELLS = 4 cells (one 32-byte
// sector a row): each warp load then covers 8 rows x 4 consecutive cells.
// A chunk holds cells cb..cb+3 of the 7 reconstructed fields and the normal
// field on faces fc..fc+3; layout [field][row][5] (one pad entry a row keeps
// a warp's 8-byte reads conflict-free).
constexpr int XS_CELLS = 4;
constexpr int XS_PITCH = XS_CELLS + 1;
template <typename R>
constexpr size_t xstage_smem() {
    return (size_t)(WK_FIELDS + 1) * WK_THREADS * XS_PITCH * sizeof(R);
}

//
// The 7 flux components of face f go back into the slots of field 0..6 at
// position (f - fc): by then the thread has consumed its own cells there.
// flush() writes a chunk's fluxes out in the same sector-sized pieces.
template <typename R>
struct XStage {
    R* buf;
    int rowbase[4];  // cell 0 of the rows this thread loads: tid/4 + 16 m
    bool rowok[4];   // the row is a real column (not a spare of the last block)
    const R* fld[WK_FIELDS + 1];
    __device__ void init(const Box& b, const PrimT<R>& pr, R* smem) {
        buf = smem;
        const R* f8[WK_FIELDS + 1] = {pr.w[0], pr.w[1], pr.w[2], pr.w[3], pr.w[4], pr.bc[1], pr.bc[2], pr.bf[0]};
#pragma unroll
        for (int v = 0; v <= WK_FIELDS; ++v) fld[v] = f8[v];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const long long col = (long long)blockIdx.x * WK_THREADS + (threadIdx.x >> 2) + 16 * m;
            rowbase[m] = walk_base<0>(b, col);
            rowok[m] = col < WalkGeom<0>::ncols(b);
        }
    }
    // fluxes of faces fc..fc+3 (only those < fend)
    __device__ void flush(int fc, int fend, FaceFluxT<R>& out) const {
        const int j = threadIdx.x & 3;
        const int face = fc + j;
        if (face >= fend) return;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            if (!rowok[m]) continue;
            const int row = (threadIdx.x >> 2) + 16 * m;
#pragma unroll
            for (int v = 0; v < WK_FIELDS; ++v) out.f[v][rowbase[m] + face] = buf[(v * WK_THREADS + row) * XS_PITCH + j];
        }
    }
    __device__ void put(int v, int j, R x) { buf[(v * WK_THREADS + threadIdx.x) * XS_PITCH + j] = x; }
    // cells cb..cb+3 (only those <= last, the last ghost cell) and faces
    // fc..fc+3 (only those < fend)
    __device__ void load(int cb, int last, int fc, int fend) {
        const int j = threadIdx.x & 3;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int row = (threadIdx.x >> 2) + 16 * m;
#pragma unroll
            for (int v = 0; v <= WK_FIELDS; ++v) {
                const int cell = (v < WK_FIELDS ? cb : fc) + j;
                const bool ok = v < WK_FIELDS ? cell <= last : cell < fend;
                buf[(v * WK_THREADS + row) * XS_PITCH + j] = ok ? fld[v][rowbase[m] + cell] : R(0);
            }
        }
    }
    __device__ R get(int v, int j) const { return buf[(v * WK_THREADS + threadIdx.x) * XS_PITCH + j]; }
};

// segment prologue for one field: returns vp_out(f0), the slope of cell
// f0+1 and the interface value between f0 and f0+1 (PPM)
template <int RECON, typename R>
__device__ __forceinline__ void walk_prologue(const AxisTabs& A, int f0, R x0, R x1, R x2, R x3, R x4, R& vpf, R& d1,
                                              R& Vf) {
    if (RECON == 4) {
        const R dm0 = ppm_slope<false>(x0, x1, x2, (R)A.s0[f0 - 1], (R)A.s1[f0 - 1]);
        const R dmc = ppm_slope<false>(x1, x2, x3, (R)A.s0[f0], (R)A.s1[f0]);
        const R dmp = ppm_slope<false>(x2, x3, x4, (R)A.s0[f0 + 1], (R)A.s1[f0 + 1]);
        const R Vm = ppm_face(x1, x2, dm0, dmc, (R)A.a0[f0 - 1], (R)A.a1[f0 - 1], (R)A.a2[f0 - 1], (R)A.a3[f0 - 1]);
        const R Vp = ppm_face(x2, x3, dmc, dmp, (R)A.a0[f0], (R)A.a1[f0], (R)A.a2[f0], (R)A.a3[f0]);
        R vm, vp;
        ppm_fix<false>(x2, Vm, Vp, vm, vp);
        vpf = vp;
        d1 = dmp;
        Vf = Vp;
    } else {
        vpf = x2 + R(0.5) * tvd_slope(x1, x2, x3, (R)A.tcf[f0], (R)A.tcb[f0]);
        d1 = R(0);
        Vf = R(0);
    }
}

// the weights of the step at face f: PPM forms the slope of cell f+2 and the
// interface value between f+1 and f+2, TVD the slope of cell f+1
template <int RECON, typename R>
__device__ __forceinline__ CellWeights<RECON, R> walk_weights(const AxisTabs& A, int f) {
    if constexpr (RECON == 4) return CellWeights<RECON, R>(A, f + 2, f + 1);
    else return CellWeights<RECON, R>(A, f + 1);
}

// one window step for one field at face f: from v(f) (TVD), v(f+1), v(f+2),
// the new cell x = v(f+3), the carried slope d1 and interface Vf, returns
// vm_out(f+1), vp_out(f+1) and updates d1, Vf
template <int RECON, typename R>
__device__ __forceinline__ void walk_step(const CellWeights<RECON, R>& W, R v0, R v1, R v2, R x, R& d1, R& Vf, R& vm1,
                                          R& vp1) {
    if constexpr (RECON == 4) {
        const R d2 = W.template slope<false>(v1, v2, x);
        const R Vn = W.face(v1, v2, d1, d2);
        ppm_fix<false>(v1, Vf, Vn, vm1, vp1);
        d1 = d2;
        Vf = Vn;
    } else {
        const R sl = W.slope(v0, v1, v2);
        vm1 = v1 - R(0.5) * sl;
        vp1 = v1 + R(0.5) * sl;
    }
}

// HLL at face f; the x sweep parks the fluxes in the staging slots (j)
template <int DIR, typename R, bool RECIP = false>
__device__ __forceinline__ void walk_flux(const WalkCol<DIR, R>& C, int f, R (&wl)[8], R (&wr)[8], R ggas,
                                          FaceFluxT<R>& out, R bn, XStage<R>& X, int j) {
    wl[IBX + DIR] = bn;
    wr[IBX + DIR] = bn;
    R fx[7];
    sweep_hll<DIR, R, RECIP>(wl, wr, ggas, fx);
    if (DIR == 0) {
#pragma unroll
        for (int i = 0; i < 7; ++i) X.put(i, j, fx[i]);
        return;
    }
    if (!C.active) return;
    const int o = C.base + f * C.s;
#pragma unroll
    for (int i = 0; i < 7; ++i) out.f[i][o] = fx[i];
}

// x sweep, at the first face f of a chunk: write out the previous chunk's
// fluxes, then stage cells f+4..f+7 and faces f..f+3
template <int DIR, typename R>
__device__ __forceinline__ void walk_chunk(const WalkCol<DIR, R>& C, int f, XStage<R>& X, FaceFluxT<R>& out) {
    __syncthreads();
    if (f > C.f0) X.flush(f - XS_CELLS, C.f1, out);
    X.load(f + 4, C.nd + 3, f, C.f1);
    __syncthreads();
}

// x sweep, after the last face: write out the last chunk
template <int DIR, typename R>
__device__ __forceinline__ void walk_last(const WalkCol<DIR, R>& C, XStage<R>& X, FaceFluxT<R>& out) {
    __syncthreads();
    X.flush(C.f0 + ((C.f1 - 1 - C.f0) & ~(XS_CELLS - 1)), C.f1, out);
}

template <int DIR, int RECON, typename R>
__global__ void __launch_bounds__(WK_THREADS, 5) k_sweep_walk(Box b, Tabs T, PrimT<R> pr, R ggas, FaceFluxT<R> out,
                                                             int seg) {
    extern __shared__ __align__(16) unsigned char wk_raw[];
    WalkCol<DIR, R> C;
    if (!C.init(b, pr, seg)) return;
    const AxisTabs A = T.ax[DIR];
    const int s = C.s, f0 = C.f0;
    XStage<R> X;
    if (DIR == 0) X.init(b, pr, reinterpret_cast<R*>(wk_raw));

    R v0[WK_FIELDS], v1[WK_FIELDS], v2[WK_FIELDS], d1[WK_FIELDS], Vf[WK_FIELDS], vpf[WK_FIELDS], nxt[WK_FIELDS];
#pragma unroll
    for (int v = 0; v < WK_FIELDS; ++v) {
        const R* q = C.src[v];
        const R x0 = q[(f0 - 2) * s], x1 = q[(f0 - 1) * s], x2 = q[f0 * s], x3 = q[(f0 + 1) * s],
                x4 = q[(f0 + 2) * s];
        walk_prologue<RECON>(A, f0, x0, x1, x2, x3, x4, vpf[v], d1[v], Vf[v]);
        v0[v] = x2;
        v1[v] = x3;
        v2[v] = x4;
        nxt[v] = q[(f0 + 3) * s];
    }

    for (int f = f0; f < C.f1; ++f) {
        R wl[8], wr[8];
        const int j = (f - f0) & (XS_CELLS - 1);
        if (DIR == 0 && j == 0) walk_chunk(C, f, X, out);
        const R bn = DIR == 0 ? X.get(WK_FIELDS, j) : C.bn[f * s];
        const auto W = walk_weights<RECON, R>(A, f);
#pragma unroll
        for (int v = 0; v < WK_FIELDS; ++v) {
            const R x = nxt[v];
            R vm1, vp1;
            walk_step<RECON>(W, v0[v], v1[v], v2[v], x, d1[v], Vf[v], vm1, vp1);
            wl[C.slot[v]] = vpf[v];  // vp_out of cell f
            wr[C.slot[v]] = vm1;     // vm_out of cell f+1
            vpf[v] = vp1;
            v0[v] = v1[v];
            v1[v] = v2[v];
            v2[v] = x;
        }
        // prefetch the next cell (f+4 <= nd+3 while f+1 < f1)
        if (f + 1 < C.f1) {
#pragma unroll
            for (int v = 0; v < WK_FIELDS; ++v) nxt[v] = DIR == 0 ? X.get(v, j) : C.src[v][(f + 4) * s];
        }
        walk_flux<DIR>(C, f, wl, wr, ggas, out, bn, X, j);
    }
    if (DIR == 0) walk_last(C, X, out);
}

// shared-memory window. PPM steps from v(f+1), v(f+2), the carried slope and
// interface value: a ring of two cell values and three slots; TVD from v(f),
// v(f+1), v(f+2): a ring of three and one slot. The last slot is vp_out(f).
template <int RECON>
struct WalkSlots {
    static constexpr int RING = RECON == 4 ? 2 : 3, D1 = RING, VF = RING + 1, VP = RECON == 4 ? RING + 2 : RING,
                         COUNT = VP + 1;
};
// The mixed form's walkers also keep the weights of the segment's faces, rounded
// to FP32 once a block: 0.541 -> 0.527 (y) and 0.520 ms (z) at 256^3. In FP64 the
// weights come from global memory at every face, the same 0.90 ms.
template <typename R>
constexpr bool WALK_TAB = sizeof(R) == 4;
// the window, then the weights (CellWeights::store), then the x staging
template <typename R>
inline size_t walk_smem(int dir, bool ppm, int seg) {
    const int w = !WALK_TAB<R> ? 0 : ppm ? CellWeights<4, R>::N : CellWeights<1, R>::N;
    return ((size_t)(ppm ? WalkSlots<4>::COUNT : WalkSlots<1>::COUNT) * WK_FIELDS * WK_THREADS + (size_t)w * seg) *
               sizeof(R) +
           (dir == 0 ? xstage_smem<R>() : 0);
}
constexpr int WK_SLOTS = 6;  // slots of the fused walkers (cumc_fused.cuh): a ring of three, slope, interface, vp_out

// STATES (y and z only): instead of solving HLL, store each face's
// reconstructed states, left in out and right in out_r (field order of the
// sweep, at the face's left cell), for the adjoint's HLL transpose.
// c_lo, c_cnt, c_step: the columns walked (WalkCol; c_cnt < 0 for all)
// RECIP: the HLL solve's quotients as products with reciprocals (hll_flux7_recip)
template <int DIR, int RECON, typename R, bool STATES = false, bool RECIP = false>
__global__ void __launch_bounds__(WK_THREADS, CUMC_WALK_MINB) k_sweep_walk_sm(Box b, Tabs T, PrimT<R> pr, R ggas, FaceFluxT<R> out,
                                                             int seg, FaceFluxT<R> out_r, int c_lo, int c_cnt, int c_step) {
    static_assert(!STATES || DIR != 0, "face states along y and z");
    extern __shared__ __align__(16) unsigned char wk_raw[];
    R* const sm = reinterpret_cast<R*>(wk_raw) + threadIdx.x;
    auto at = [&](int slot, int v) -> R& { return sm[(slot * WK_FIELDS + v) * WK_THREADS]; };
    WalkCol<DIR, R> C;
    if (!C.init(b, pr, seg, c_lo, c_cnt, c_step)) return;
    const AxisTabs A = T.ax[DIR];
    const int s = C.s, f0 = C.f0;
    XStage<R> X;
    using W = WalkSlots<RECON>;
    R* const tab = reinterpret_cast<R*>(wk_raw) + W::COUNT * WK_FIELDS * WK_THREADS;
    if constexpr (WALK_TAB<R>)
        for (int n = threadIdx.x; n < C.f1 - f0; n += WK_THREADS) walk_weights<RECON, R>(A, f0 + n).store(tab + n, seg);
    if (DIR == 0) X.init(b, pr, tab + (WALK_TAB<R> ? CellWeights<RECON, R>::N * seg : 0));

    R nxt[WK_FIELDS];
    // ring positions of v(f), v(f+1), v(f+2) for f = f0 (a ring of two has no v(f))
    int r0 = f0 % W::RING, r1 = (f0 + 1) % W::RING, r2 = (f0 + 2) % W::RING;
#pragma unroll
    for (int v = 0; v < WK_FIELDS; ++v) {
        const R* q = C.src[v];
        const R x0 = q[(f0 - 2) * s], x1 = q[(f0 - 1) * s], x2 = q[f0 * s], x3 = q[(f0 + 1) * s],
                x4 = q[(f0 + 2) * s];
        R vpf, d1, Vf;
        walk_prologue<RECON>(A, f0, x0, x1, x2, x3, x4, vpf, d1, Vf);
        if (RECON != 4) at(r0, v) = x2;
        at(r1, v) = x3;
        at(r2, v) = x4;
        if (RECON == 4) {
            at(W::D1, v) = d1;
            at(W::VF, v) = Vf;
        }
        at(W::VP, v) = vpf;
        nxt[v] = q[(f0 + 3) * s];
    }
    // the mixed form fetches the normal field a face ahead too (its faces are short
    // enough to wait for it: z 0.519 -> 0.484 ms); FP64 has no register for it
    constexpr bool AHEAD = DIR > 0 && sizeof(R) == 4;
    R bn_next = AHEAD ? C.bn[f0 * s] : R(0);
    if constexpr (WALK_TAB<R>) __syncthreads();

    for (int f = f0; f < C.f1; ++f) {
        R wl[8], wr[8];
        const int j = (f - f0) & (XS_CELLS - 1);
        if (DIR == 0 && j == 0) walk_chunk(C, f, X, out);
        const R bn = DIR == 0 ? X.get(WK_FIELDS, j) : AHEAD ? bn_next : C.bn[f * s];
        auto weights = [&] {
            if constexpr (WALK_TAB<R>) return CellWeights<RECON, R>(tab + (f - f0), seg);
            else return walk_weights<RECON, R>(A, f);
        };
        const CellWeights<RECON, R> cw = weights();
#pragma unroll
        for (int v = 0; v < WK_FIELDS; ++v) {
            const R x = nxt[v];
            R d1 = RECON == 4 ? at(W::D1, v) : R(0), Vf = RECON == 4 ? at(W::VF, v) : R(0);
            R vm1, vp1;
            walk_step<RECON>(cw, RECON == 4 ? R(0) : at(r0, v), at(r1, v), at(r2, v), x, d1, Vf, vm1, vp1);
            wl[C.slot[v]] = at(W::VP, v);  // vp_out of cell f
            wr[C.slot[v]] = vm1;           // vm_out of cell f+1
            at(W::VP, v) = vp1;
            if (RECON == 4) {
                at(W::D1, v) = d1;
                at(W::VF, v) = Vf;
            }
            at(RECON == 4 ? r1 : r0, v) = x;  // v(f+3) takes the place of the oldest value
        }
        if (RECON == 4) {
            const int r = r1;
            r1 = r2;
            r2 = r;
        } else {
            const int r = r0;
            r0 = r1;
            r1 = r2;
            r2 = r;
        }
        if (f + 1 < C.f1) {
#pragma unroll
            for (int v = 0; v < WK_FIELDS; ++v) nxt[v] = DIR == 0 ? X.get(v, j) : C.src[v][(f + 4) * s];
            if (AHEAD) bn_next = C.bn[(f + 1) * s];
        }
        if (STATES) {
            if (C.active) {
                const int o = C.base + f * s;
#pragma unroll
                for (int v = 0; v < WK_FIELDS; ++v) {
                    out.f[v][o] = wl[C.slot[v]];
                    out_r.f[v][o] = wr[C.slot[v]];
                }
            }
        } else {
            walk_flux<DIR, R, RECIP>(C, f, wl, wr, ggas, out, bn, X, j);
        }
    }
    if (DIR == 0) walk_last(C, X, out);
}

}  // namespace cumc

namespace cumc {

// ---------------------------------------------------------------------------
// x sweep with one lane per cell (GET_FLUXES x sweep, solver/spatial.f90:131-168).
// A warp holds 32 consecutive cells x0 .. x0+31 of one row. Each lane forms
// its own cell's limited slope, the interface value with the next cell and
// the extremum fix once, taking the neighbours' values through warp shuffles
// (the same expressions and operand order as the per-face kernel, so the
// fluxes are bit-identical); lanes 2..28 then solve HLL at their faces. A
// warp yields 27 faces; consecutive warps overlap by 5 cells. Loads and
// stores are one 256-byte row segment per field.
// Eight 128-thread blocks per SM (64 registers, a few spilled to L1). The mixed
// form's x sweep (bound by issue, 0.75 a cycle, and by its conversions: 0.70 ->
// 0.66 ms a stage at 256^3 with branch-free roots) and the adjoint's face states;
// in FP64 the two-cell form below is the default.
// ---------------------------------------------------------------------------
constexpr int XW_FACES = 27;

// STATES: store each face's reconstructed states (left in out, right in
// out_r, field order of the sweep) instead of solving HLL.
// The rows are those of the z planes l_lo .. l_lo + l_cnt - 1 (l_cnt < 0: all).
template <int RECON, typename R, bool STATES = false, bool RECIP = false>
__global__ void __launch_bounds__(128, CUMC_XWARP_MINB) k_sweep_xwarp(Box b, Tabs T, PrimT<R> pr, R ggas, FaceFluxT<R> out,
                                                        FaceFluxT<R> out_r, int l_lo, int l_cnt) {
    constexpr unsigned FULL = 0xffffffffu;
    const int nw = (b.nx + 1 + XW_FACES - 1) / XW_FACES;  // warps per row
    const unsigned warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (l_cnt < 0) l_cnt = b.nz + 2;
    const long long rows = (long long)(b.ny + 2) * l_cnt;
    if (warp >= rows * nw || (b.skip && *b.skip)) return;  // uniform over the warp
    const int w = (int)(warp % nw);
    const unsigned row = warp / nw;
    const int k = (int)(row % (b.ny + 2)), l = l_lo + (int)(row / (b.ny + 2));
    const int c = w * XW_FACES - 2 + lane;  // this lane's cell; its face is c | c+1
    const bool inb = c >= -2 && c <= b.nx + 3;
    const int ct = min(max(c, -2), b.nx + 3);  // table index kept in range for spare lanes
    const int base = b.idx(0, k, l);
    const AxisTabs A = T.ax[0];
    const R* src[7] = {pr.w[0], pr.w[1], pr.w[2], pr.w[3], pr.w[4], pr.bc[1], pr.bc[2]};
    const int slot[7] = {IRHO, IVX, IVY, IVZ, ITAU, IBY, IBZ};
    R wl[8], wr[8];
#pragma unroll
    for (int v = 0; v < 7; ++v) {
        const R x = inb ? src[v][base + c] : R(0);
        const R xm = __shfl_up_sync(FULL, x, 1), xp = __shfl_down_sync(FULL, x, 1);
        R vm, vp;
        if (RECON == 4) {
            const R d = ppm_slope(xm, x, xp, (R)A.s0[ct], (R)A.s1[ct]);
            const R dp = __shfl_down_sync(FULL, d, 1);
            const R V = ppm_face(x, xp, d, dp, (R)A.a0[ct], (R)A.a1[ct], (R)A.a2[ct], (R)A.a3[ct]);  // c | c+1
            const R Vm = __shfl_up_sync(FULL, V, 1);                                                // c-1 | c
            ppm_fix(x, Vm, V, vm, vp);
        } else {
            const R sl = tvd_slope(xm, x, xp, (R)A.tcf[ct], (R)A.tcb[ct]);
            vm = x - R(0.5) * sl;
            vp = x + R(0.5) * sl;
        }
        wl[slot[v]] = vp;                             // vp_out of cell c
        wr[slot[v]] = __shfl_down_sync(FULL, vm, 1);  // vm_out of cell c+1
    }
    if (lane < 2 || lane > 28 || c < 0 || c > b.nx) return;
    if (STATES) {
#pragma unroll
        for (int v = 0; v < 7; ++v) {
            out.f[v][base + c] = wl[slot[v]];
            out_r.f[v][base + c] = wr[slot[v]];
        }
        return;
    }
    const R bn = pr.bf[0][base + c];
    wl[IBX] = bn;
    wr[IBX] = bn;
    R fx[7];
    sweep_hll<0, R, RECIP>(wl, wr, ggas, fx);
#pragma unroll
    for (int i = 0; i < 7; ++i) out.f[i][base + c] = fx[i];
}

inline long long xwarp_threads(const Box& b, int l_cnt = -1) {
    return (long long)(b.ny + 2) * (l_cnt < 0 ? b.nz + 2 : l_cnt) * ((b.nx + 1 + XW_FACES - 1) / XW_FACES) * 32;
}

// ---------------------------------------------------------------------------
// x sweep with two cells a lane (the default in FP64). The rows 0:n+1 of a plane are
// taken as one line of SX (ny + 2) cells: a warp holds 64 consecutive cells of
// it, lane i the cells 2i and 2i+1, forms each cell's slope, interface value
// and extremum fix once (five shuffled values a field and two cells, against
// eight in k_sweep_xwarp) and solves HLL at 58 faces, so that 58 of 64 lanes'
// work counts instead of 27 of 32, and a row that is no multiple of 27 faces
// costs nothing but its five faces that straddle the row's end, which are
// skipped. The pair's states wait in shared memory between the reconstruction
// and the two solves (one body, run twice), which keeps the registers to the
// walkers' 96. VEC: with SX even a pair starts on a 16-byte boundary and moves as
// one vector.
// ---------------------------------------------------------------------------
constexpr int XP_FACES = 58, XP_THREADS = 128;
#ifndef CUMC_XPAIR_MINB
#define CUMC_XPAIR_MINB 5
#endif
template <bool VEC>
__device__ __forceinline__ double2 ld_pair(const double* p, int i) {
    if constexpr (VEC) return *reinterpret_cast<const double2*>(p + i);
    return make_double2(p[i], p[i + 1]);
}
template <bool VEC>
__device__ __forceinline__ void st_pair(double* p, int i, double a, double b, bool oka, bool okb) {
    if (VEC && oka && okb) {
        *reinterpret_cast<double2*>(p + i) = make_double2(a, b);
    } else {
        if (oka) p[i] = a;
        if (okb) p[i + 1] = b;
    }
}

__host__ __device__ __forceinline__ unsigned xpair_blocks(const Box& b) {
    const unsigned warps = (unsigned)(b.SX * (b.ny + 2) - 2 + XP_FACES - 1) / XP_FACES;
    return (warps + XP_THREADS / 32 - 1) / (XP_THREADS / 32);
}

// cell c's weights; TVD slopes count on 0..n+1 only, and beyond it the weights
// of the nearest such cell keep them on the rounded path
template <int RECON>
__device__ __forceinline__ CellWeights<RECON, double> xpair_weights(const AxisTabs& A, int c, int n) {
    if constexpr (RECON == 4) return CellWeights<RECON, double>(A, c, c);
    else return CellWeights<RECON, double>(A, min(max(c, 0), n + 1));
}

template <int RECON, bool RECIP, bool VEC>
__global__ void __launch_bounds__(XP_THREADS, CUMC_XPAIR_MINB) k_sweep_xpair(Box b, Tabs T, Prim pr, double ggas,
                                                                           FaceFlux out, int l_lo, int l_step) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ double sm[28][XP_THREADS];  // states of the pair's two faces: left 7, right 7 each
    const int cells = b.SX * (b.ny + 2);
    const unsigned bpp = xpair_blocks(b), plane = blockIdx.x / bpp;  // blocks a plane
    const int w = (int)(blockIdx.x - plane * bpp) * (XP_THREADS / 32) + (int)(threadIdx.x >> 5);
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    if (w * XP_FACES + 2 >= cells || (b.skip && *b.skip)) return;  // uniform over the warp
    const int m = w * XP_FACES + 2 * lane;  // position of the lane's first cell in the plane's line
    const int g = b.idx(-2, 0, l_lo + l_step * (int)plane) + m;
    const int j0 = m % b.SX - 2, j1 = j0 == b.nx + 3 ? -2 : j0 + 1;
    const bool faces = lane >= 1 && lane <= 29;
    const bool ok0 = faces && m < cells && j0 >= 0 && j0 <= b.nx;
    const bool ok1 = faces && m + 1 < cells && j1 >= 0 && j1 <= b.nx;
    const AxisTabs A = T.ax[0];
    const double* src[7] = {pr.w[0], pr.w[1], pr.w[2], pr.w[3], pr.w[4], pr.bc[1], pr.bc[2]};
    const auto W0 = xpair_weights<RECON>(A, j0, b.nx), W1 = xpair_weights<RECON>(A, j1, b.nx);
#pragma unroll
    for (int v = 0; v < 7; ++v) {
        const double2 x = ld_pair<VEC>(src[v], g);
        const double xm = __shfl_up_sync(FULL, x.y, 1), xp = __shfl_down_sync(FULL, x.x, 1);
        double vm0, vp0, vm1, vp1;
        if constexpr (RECON == 4) {
            const double d0 = W0.slope(xm, x.x, x.y), d1 = W1.slope(x.x, x.y, xp);
            const double d2 = __shfl_down_sync(FULL, d0, 1);
            const double V0 = W0.face(x.x, x.y, d0, d1), V1 = W1.face(x.y, xp, d1, d2);
            const double Vm = __shfl_up_sync(FULL, V1, 1);
            ppm_fix(x.x, Vm, V0, vm0, vp0);
            ppm_fix(x.y, V0, V1, vm1, vp1);
        } else {
            const double s0 = W0.slope(xm, x.x, x.y), s1 = W1.slope(x.x, x.y, xp);
            vm0 = x.x - 0.5 * s0;
            vp0 = x.x + 0.5 * s0;
            vm1 = x.y - 0.5 * s1;
            vp1 = x.y + 0.5 * s1;
        }
        sm[v][tid] = vp0;  // face 2i | 2i+1: vp_out of its left cell, vm_out of its right cell
        sm[7 + v][tid] = vm1;
        sm[14 + v][tid] = vp1;
        sm[21 + v][tid] = __shfl_down_sync(FULL, vm0, 1);
    }
    if (!ok0 && !ok1) return;
    const double2 bn = ld_pair<VEC>(pr.bf[0], g);
    double fx[7];
#pragma unroll 1
    for (int f = 0; f < 2; ++f) {
        if (f == 0 ? ok0 : ok1) {
            constexpr int slot[7] = {IRHO, IVX, IVY, IVZ, ITAU, IBY, IBZ};
            double wl[8], wr[8];
#pragma unroll
            for (int v = 0; v < 7; ++v) {
                wl[slot[v]] = sm[14 * f + v][tid];
                wr[slot[v]] = sm[14 * f + 7 + v][tid];
            }
            wl[IBX] = wr[IBX] = f == 0 ? bn.x : bn.y;
            sweep_hll<0, double, RECIP>(wl, wr, ggas, fx);
        }
        if (f == 0) {
#pragma unroll
            for (int i = 0; i < 7; ++i) sm[i][tid] = fx[i];
        }
    }
#pragma unroll
    for (int i = 0; i < 7; ++i) st_pair<VEC>(out.f[i], g, sm[i][tid], fx[i], ok0, ok1);
}

// the vector form's conditions: every pair aligned to its own size
inline bool xpair_vec(const Box& b, const Prim& pr, const FaceFlux& out) {
    uintptr_t at = (uintptr_t)pr.bc[1] | (uintptr_t)pr.bc[2] | (uintptr_t)pr.bf[0];
    for (int q = 0; q < 5; ++q) at |= (uintptr_t)pr.w[q];
    for (int q = 0; q < 7; ++q) at |= (uintptr_t)out.f[q];
    return b.SX % 2 == 0 && at % 16 == 0;
}
inline dim3 xpair_grid(const Box& b, int l_cnt) { return dim3(xpair_blocks(b) * (unsigned)l_cnt); }

}  // namespace cumc
