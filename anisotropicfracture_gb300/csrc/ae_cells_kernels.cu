// Kernels of the batched periodic-cell solve.  Every stencil kernel walks a work table with a
// grid-stride loop (a persistent grid sized by the tuner); each entry is a run of `chunk`
// consecutive nodes of one solve's level, one node per thread.  Entries of solves that are not
// active (converged, failed, or without that level) are skipped by the whole block.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "ae_cell.cuh"
#include "ae_cells.h"
#include "ae_kernels.cuh"

namespace ae {

namespace {

template <class R>
__device__ __forceinline__ const CellVec<R>& vec_of(const SolveDev& S, int m) {
    if constexpr (sizeof(R) == 8) return S.v64[m];
    else return S.v32[m];
}
template <class R>
__device__ __forceinline__ const R* cfield(const CellLevelDev& L) {
    if constexpr (sizeof(R) == 8) return L.C64;
    else return L.C32;
}
template <class R>
__device__ __forceinline__ const R* ifield(const CellLevelDev& L) {
    if constexpr (sizeof(R) == 8) return L.I64;
    else return L.I32;
}
template <class R>
__device__ __forceinline__ const SCoef<R>& kfield(const CellLevelDev& L) {
    if constexpr (sizeof(R) == 8) return L.K64;
    else return L.K32;
}
template <class R>
__device__ __forceinline__ const R* tabfield(const CellLevelDev& L) {
    if constexpr (sizeof(R) == 8) return L.tab64;
    else return L.tab32;
}
template <class R>
__device__ __forceinline__ const R* itabfield(const CellLevelDev& L) {
    if constexpr (sizeof(R) == 8) return L.itab64;
    else return L.itab32;
}

// (converted on the host: a conversion holds the FP64 pipe for 64 clocks a warp)
template <class R>
__device__ __forceinline__ R omega_of(const CellArgs& A) {
    if constexpr (sizeof(R) == 8) return A.omega;
    else return A.omega32;
}

// Which finest-level representation a launch serves: GR = true the grain tables (entries of
// cells without them are skipped), GR = false the per-node arrays (on the finest level, entries
// of cells with grain tables are skipped).  Coarser levels always use the per-node arrays.
__device__ __forceinline__ bool rep_skips(bool GR, int m, const CellLevelDev& L) {
    return GR ? (m != 0 || L.gid == nullptr) : (m == 0 && L.gid != nullptr);
}

// A u = row_factor f at node t of level m
template <int M, class R, bool GR>
__device__ __forceinline__ void level_apply(const CellLevelDev& L, int uniform, const R* U, int t, const POff& o,
                                            R f[3]) {
    if constexpr (GR) cell_apply_grains<M, R>(kfield<R>(L), uniform, L.gid, tabfield<R>(L), L.rows64, U, L.nn, t, o, f);
    else cell_apply<M, R>(kfield<R>(L), uniform, cfield<R>(L), L.nn, U, L.nn, t, o, f);
}

constexpr int kCellThreads = 256;
// Resident blocks per SM requested for the FP32 cell sweeps (smoother, correction residual);
// 0: the compiler's choice.  On a 512-cell mixed batch:
//   finest level on a grain map: 4 blocks (64 registers), 482 solves/s, against 444 with the
//     compiler's 80 registers;
//   per-node levels: 3 blocks (80 registers, about 100 B of spills), 507 solves/s, against 482
//     with the compiler's 118 registers.
#ifndef AE_CELL_SMOOTH_BLOCKS
#define AE_CELL_SMOOTH_BLOCKS 4
#endif
// FP64 on a grain map: 2 blocks (128 registers, 34 KB of tables and queue each)
#ifndef AE_CELL_GRAIN64_BLOCKS
#define AE_CELL_GRAIN64_BLOCKS 2
#endif
#ifndef AE_CELL_SMOOTH_BLOCKS_PERNODE
#define AE_CELL_SMOOTH_BLOCKS_PERNODE 3
#endif
template <int M, class R, bool GR>
constexpr int cell_min_blocks() {
    // FP64, 21 slots per node: two blocks need 128 registers; the compiler took 186 for the smoother, one block:
    // 19 cells of 64^3, fixed cycles, 58.5 ms, with two 56.3
    if (M == MM && sizeof(R) == 8 && !GR) return 2;
    return sizeof(R) != 4 ? 0 : GR ? AE_CELL_SMOOTH_BLOCKS : AE_CELL_SMOOTH_BLOCKS_PERNODE;
}

// one damped-Jacobi sweep of the correction at level m: from2 = 0 reads cor and writes cor2,
// from2 = 1 the reverse.  ZERO: the input is the zero vector (the first sweep of a V-cycle).
template <int M, class R, bool ZERO, bool GR>
__global__ void __launch_bounds__(kCellThreads, cell_min_blocks<M, R, GR>()) kb_smooth(CellArgs A, const Work* __restrict__ tab, int ntab, int m,
                                                          int from2) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        if (m >= S.nlev - 1 || !S.st->active) continue;
        const CellLevelDev& L = A.cells[S.cell].lv[m];
        if (rep_skips(GR, m, L)) continue;
        if (GR && !ZERO && sizeof(R) == 4 && L.march) continue;  // kb_grain_march's
        const int t = w.start + threadIdx.x;
        const int nn = L.nn;
        if (t >= nn) continue;
        const CellVec<R>& V = vec_of<R>(S, m);
        const R* __restrict__ xin = from2 ? V.cor2 : V.cor;
        R* __restrict__ xout = from2 ? V.cor : V.cor2;
        const R* __restrict__ b = V.res;
        const R omega = omega_of<R>(A);
        // grain tables on the finest level of a Voronoi cell, per-node arrays otherwise
        constexpr bool grains = GR;
        const int g3 = grains ? 3 * (int)__ldg(L.gid + t) : 0;
        const R* __restrict__ invD = grains ? itabfield<R>(L) + g3 : ifield<R>(L) + t;
        const int ds = grains ? 1 : nn;  // component stride of invD / D
        if (ZERO) {
#pragma unroll
            for (int p = 0; p < 3; ++p) xout[p * nn + t] = jacobi_update<R>(R(0), b[p * nn + t], invD[p * ds], omega);
            continue;
        }
        int i, j, k;
        cell_ijk(L.n, t, i, j, k);
        const POff o = cell_offsets(L.n, i, j, k);
        R f[3];
        level_apply<M, R, GR>(L, A.uniform, xin, t, o, f);
        const R sc = row_factor(kfield<R>(L));
#pragma unroll
        for (int p = 0; p < 3; ++p)
            xout[p * nn + t] = jacobi_update<R>(xin[p * nn + t], row_residual(b[p * nn + t], sc, f[p]), invD[p * ds], omega);
    }
}

template <class R>
__global__ void __launch_bounds__(kCellThreads) kb_copy2(CellArgs A, const Work* __restrict__ tab, int ntab, int m,
                                                         int fill0) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        if (m >= S.nlev - 1 || !S.st->active) continue;
        const int nn = A.cells[S.cell].lv[m].nn;
        const int t = w.start + threadIdx.x;
        if (t >= nn) continue;
        const CellVec<R>& V = vec_of<R>(S, m);
#pragma unroll
        for (int p = 0; p < 3; ++p) V.cor[p * nn + t] = fill0 ? R(0) : V.cor2[p * nn + t];
    }
}

// rescor = res - A cor at level m (inplace: into res)
template <int M, class R, bool GR>
__global__ void __launch_bounds__(kCellThreads, cell_min_blocks<M, R, GR>()) kb_rescor(CellArgs A, const Work* __restrict__ tab, int ntab, int m,
                                                          int inplace) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        // the cycle's residual skips the bottom level; the in-place update between inner cycles
        // (top level) also runs on single-level cells
        if ((!inplace && m >= S.nlev - 1) || !S.st->active) continue;
        const CellLevelDev& L = A.cells[S.cell].lv[m];
        if (rep_skips(GR, m, L)) continue;
        if (GR && sizeof(R) == 4 && L.march) continue;  // kb_grain_march's
        const int t = w.start + threadIdx.x;
        const int nn = L.nn;
        if (t >= nn) continue;
        const CellVec<R>& V = vec_of<R>(S, m);
        int i, j, k;
        cell_ijk(L.n, t, i, j, k);
        const POff o = cell_offsets(L.n, i, j, k);
        R f[3];
        level_apply<M, R, GR>(L, A.uniform, V.cor, t, o, f);
        R* out = inplace ? V.res : V.rescor;
        const R sc = row_factor(kfield<R>(L));
#pragma unroll
        for (int p = 0; p < 3; ++p) out[p * nn + t] = row_residual(V.res[p * nn + t], sc, f[p]);
    }
}

// res_{m+1} = R rescor_m over the level m+1 nodes of solves that have level m+1
template <class R>
__global__ void __launch_bounds__(kCellThreads) kb_restrict(CellArgs A, const Work* __restrict__ tab, int ntab,
                                                            int m) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        if (m + 1 > S.nlev - 1 || !S.st->active) continue;
        const CellLevelDev& Lf = A.cells[S.cell].lv[m];
        const CellLevelDev& Lc = A.cells[S.cell].lv[m + 1];
        const int t = w.start + threadIdx.x;
        if (t >= Lc.nn) continue;
        int I, J, K;
        cell_ijk(Lc.n, t, I, J, K);
        const R* fine = vec_of<R>(S, m).rescor;
        R* crse = vec_of<R>(S, m + 1).res;
#pragma unroll
        for (int p = 0; p < 3; ++p) crse[p * Lc.nn + t] = cell_restrict<R>(fine + p * Lf.nn, Lf.n, I, J, K);
    }
}

// cor_m += I cor_{m+1} over the level m nodes
template <class R>
__global__ void __launch_bounds__(kCellThreads) kb_interp(CellArgs A, const Work* __restrict__ tab, int ntab, int m) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        if (m >= S.nlev - 1 || !S.st->active) continue;
        const CellLevelDev& Lf = A.cells[S.cell].lv[m];
        const CellLevelDev& Lc = A.cells[S.cell].lv[m + 1];
        const int t = w.start + threadIdx.x;
        if (t >= Lf.nn) continue;
        int i, j, k;
        cell_ijk(Lf.n, t, i, j, k);
        R* fine = vec_of<R>(S, m).cor;
        const R* crse = vec_of<R>(S, m + 1).cor;
#pragma unroll
        for (int p = 0; p < 3; ++p) fine[p * Lf.nn + t] += cell_interp<R>(crse + p * Lc.nn, Lc.n, i, j, k);
    }
}

// ------------------------------------------------------------------ bottom (one CTA per solve)
// The bordered cell problem on the coarsest level: Krylov on the mean-projected operator.
template <int M, bool LDG>
struct CellBottomOps {
    int n[3];
    int nn;
    SCoef<double> K;
    const double* C;
    const double* D;
    const double* I;
    int uniform;
    int sweeps;
    double omega;
    __device__ void apply_raw(const double* x, double* out) const {
        for (int t = threadIdx.x; t < nn; t += blockDim.x) {
            int i, j, k;
            cell_ijk(n, t, i, j, k);
            const POff o = cell_offsets(n, i, j, k);
            double f[3];
            cell_apply<M, double, LDG>(K, uniform, C, nn, x, nn, t, o, f);
#pragma unroll
            for (int p = 0; p < 3; ++p) out[t + p * nn] = mul_rn(K.i2[0], f[p]);
        }
        __syncthreads();
    }
    __device__ void project(double* v, BlkRed& sh) const {
#pragma unroll 1
        for (int p = 0; p < 3; ++p) {
            double s = 0.0;
            for (int t = threadIdx.x; t < nn; t += blockDim.x) s += v[p * nn + t];
            const double mean = blk_sum(s, sh) / (double)nn;
            for (int t = threadIdx.x; t < nn; t += blockDim.x) v[p * nn + t] -= mean;
        }
        __syncthreads();
    }
    __device__ void apply(const double* x, double* out, BlkRed& sh) const {
        apply_raw(x, out);
        project(out, sh);
    }
    __device__ void residual(const double* x, const double* b, double* r, BlkRed& sh) const {
        apply_raw(x, r);
        for (int t = threadIdx.x; t < 3 * nn; t += blockDim.x) r[t] = b[t] - r[t];
        __syncthreads();
        project(r, sh);
    }
    __device__ double dot(const double* x, const double* y, BlkRed& sh) const {
        double s = 0.0;
        for (int t = threadIdx.x; t < 3 * nn; t += blockDim.x) s += x[t] * y[t];
        return blk_sum(s, sh);
    }
    __device__ double ninf(const double* x, BlkRed& sh) const {
        double s = 0.0;
        for (int t = threadIdx.x; t < 3 * nn; t += blockDim.x) s = fmax(s, fabs(x[t]));
        return blk_max(s, sh);
    }
    __device__ void smooth(double* x, const double* b, double* tmp, BlkRed&) const {
        for (int s = 0; s < sweeps; ++s) {
            apply_raw(x, tmp);
            for (int t = threadIdx.x; t < 3 * nn; t += blockDim.x) {
                const double xv = x[t];
                const double rx = tmp[t] - xv * D[t];
                x[t] = (1.0 - omega) * xv + omega * (b[t] - rx) * I[t];
            }
            __syncthreads();
        }
    }
};

__host__ __device__ constexpr long long cell_bottom_smem_doubles(int nc, long long nn) { return (nc + 36) * nn; }

template <int M, class R>
__global__ void __launch_bounds__(kBottomThreads) kb_bottom(CellArgs A, KrylovParams kp, int dyn_bytes) {
    __shared__ BlkRed sh;
    extern __shared__ double smem[];
    constexpr int NC = NCoef<M>::value;
    const SolveDev& S = A.solves[blockIdx.x];
    if (!S.st->active) return;
    const int m = S.nlev - 1;
    const CellLevelDev& L = A.cells[S.cell].lv[m];
    const int nn = L.nn;
    const long long N = 3LL * nn;
    const bool fits = cell_bottom_smem_doubles(NC, nn) * (long long)sizeof(double) <= dyn_bytes;
    const double* Cp = L.C64;
    const double* Dp = L.D64;
    const double* Ip = L.I64;
    double* b = S.bwork + 8 * N;
    double* x = b + N;
    double* work = S.bwork;
    if (fits) {
        double* sC = smem;
        double* sD = sC + NC * nn;
        double* sI = sD + N;
        b = sI + N;
        x = b + N;
        work = x + N;
        for (int t = threadIdx.x; t < NC * nn; t += blockDim.x) sC[t] = L.C64[t];
        for (int t = threadIdx.x; t < N; t += blockDim.x) {
            sD[t] = L.D64[t];
            sI[t] = L.I64[t];
        }
        Cp = sC; Dp = sD; Ip = sI;
    }
    const CellVec<R>& V = vec_of<R>(S, m);
    for (int t = threadIdx.x; t < N; t += blockDim.x) {
        b[t] = (double)V.res[t];
        x[t] = 0.0;
    }
    __syncthreads();
    int ret;
    if (fits) {
        const CellBottomOps<M, false> ops{{L.n[0], L.n[1], L.n[2]}, nn, L.K64, Cp, Dp, Ip, A.uniform, A.sweeps,
                                          A.omega};
        ret = krylov_bottom(ops, kp, N, x, b, work, sh);
    } else {
        const CellBottomOps<M, true> ops{{L.n[0], L.n[1], L.n[2]}, nn, L.K64, Cp, Dp, Ip, A.uniform, A.sweeps,
                                         A.omega};
        ret = krylov_bottom(ops, kp, N, x, b, work, sh);
    }
    if (ret != 0 && ret != 9 && threadIdx.x == 0) S.st->bfail += 1;
    for (int t = threadIdx.x; t < N; t += blockDim.x) V.cor[t] = (R)x[t];
}

// ------------------------------------------------------------------ FP64 top level
// block sums of up to kPartStride values per thread, in a fixed tree, into S.part[chunk]
template <int NQ>
__device__ __forceinline__ void block_partials(double (&v)[NQ], double* dst) {
    __shared__ double red[kCellThreads / 32][NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        double s = v[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][q] = s;
    }
    __syncthreads();
    if (threadIdx.x < NQ) {
        double s = 0.0;
        for (int wq = 0; wq < (int)(blockDim.x >> 5); ++wq) s += red[wq][threadIdx.x];
        dst[threadIdx.x] = s;
    }
    __syncthreads();
}

// r = b - A x at level 0 with per-chunk sums of r (tab: one kRedChunk run per entry)
template <int M, bool GR>
__global__ void __launch_bounds__(kCellThreads, cell_min_blocks<M, double, GR>()) kb_resid_top(CellArgs A, const Work* __restrict__ tab, int ntab) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        if (!S.st->active) continue;
        const CellLevelDev& L = A.cells[S.cell].lv[0];
        if (rep_skips(GR, 0, L)) continue;
        const int t = w.start + threadIdx.x;
        const int nn = L.nn;
        double v[3] = {0.0, 0.0, 0.0};
        if (t < nn) {
            int i, j, k;
            cell_ijk(L.n, t, i, j, k);
            const POff o = cell_offsets(L.n, i, j, k);
            double f[3];
            level_apply<M, double, GR>(L, A.uniform, S.x, t, o, f);
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                v[p] = row_residual(S.b[p * nn + t], L.K64.i2[0], f[p]);
                S.r[p * nn + t] = v[p];
            }
        }
        block_partials<3>(v, S.part + (size_t)(w.start / kRedChunk) * kPartStride);
    }
}

// ------------------------------------------------------------------ finest level on a grain map
// The smoother, the correction residual and the top residual of Voronoi cells in FP64.  A block takes its run
// of nodes in two passes: every node's row without the grad C term, then, packed into as few warps as hold
// them, the nodes whose neighbours lie in different grains, which get that term added.  In one pass nearly
// every warp holds such a node and pays three columns of operations for all its lanes.  The grains' numbers
// are in shared memory (up to kGrainTabs; loaded when a block comes to another cell): rows of an odd number
// of words, so that lanes in different grains hit different banks.  The row's 36 numbers come from a table
// instead of being formed from the 21 slots (60 operations).  The arithmetic is that of cell_apply on the
// equivalent per-node field; a direction whose two neighbours lie in the same grain has an exactly zero
// stiffness difference, so its column is zero.
//
// 128 cells of 16 to 64 nodes an edge: residual 5.14 -> 3.71 ms a call.  In FP32 two passes are slower than
// one (0.444 against 0.415 ms): those sweeps march (kb_grain_march) or take one pass (kb_smooth, kb_rescor).
constexpr int kGrainTabs = 56;
template <int M, class R>
constexpr int grain_words() {  // slots, 1 / D, row numbers (FP64)
    const int n = NCoef<M>::value + 3 + (sizeof(R) == 8 ? RowN<M>::value : 0);
    return n | 1;
}
enum CellOp { CELL_SMOOTH, CELL_RESCOR, CELL_RESID };
template <int M, int OP>
__global__ void __launch_bounds__(kCellThreads, AE_CELL_GRAIN64_BLOCKS)
    kb_grain_sweep(CellArgs A, const Work* __restrict__ tab, int ntab, int flag) {
    using R = double;
    constexpr int NC = NCoef<M>::value, TS = grain_words<M, R>();
    __shared__ R ts[kGrainTabs * TS];
    __shared__ R qf[3][kCellThreads];
    __shared__ unsigned char qt[kCellThreads];
    __shared__ int qn;
    int have = -1;  // the cell whose numbers are in ts
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        if ((OP == CELL_SMOOTH || (OP == CELL_RESCOR && !flag)) && S.nlev <= 1) continue;
        if (!S.st->active) continue;
        const CellLevelDev& L = A.cells[S.cell].lv[0];
        if (rep_skips(true, 0, L)) continue;
        const int nn = L.nn;
        const bool in_smem = L.ngrains <= kGrainTabs;
        __syncthreads();  // the block is done with the queue and the numbers
        if (threadIdx.x == 0) qn = 0;
        if (in_smem && have != S.cell) {
            for (int q = threadIdx.x; q < L.ngrains * TS; q += blockDim.x) {
                const int g = q / TS, c = q - g * TS;
                if (c < NC) ts[q] = tabfield<R>(L)[g * NC + c];
                else if (c < NC + 3) ts[q] = itabfield<R>(L)[3 * g + c - NC];
                else if (c < NC + 3 + RowN<M>::value) ts[q] = L.rows64[g * RowN<M>::value + c - NC - 3];
            }
            have = S.cell;
        }
        __syncthreads();
        const CellVec<R>& V = vec_of<R>(S, 0);
        const R *u, *b;
        R* out;
        if constexpr (OP == CELL_RESID) {
            u = S.x;
            b = S.b;
            out = S.r;
        } else {
            u = OP == CELL_SMOOTH && flag ? V.cor2 : V.cor;
            b = V.res;
            out = OP == CELL_SMOOTH ? (flag ? V.cor : V.cor2) : flag ? V.res : V.rescor;
        }
        const SCoef<R>& K = kfield<R>(L);
        const R sc = row_factor(K), omega = omega_of<R>(A);
        const auto body = [&](auto smem) {
            constexpr bool SM = decltype(smem)::value;
            const auto slot = [&](int g, int q) { return SM ? ts[g * TS + q] : __ldg(tabfield<R>(L) + g * NC + q); };
            const auto finish = [&](int t, int g, const R (&f)[3]) {
                R v[3];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    v[p] = row_residual(b[p * nn + t], sc, f[p]);
                    if (OP == CELL_SMOOTH) {
                        const R id = SM ? ts[g * TS + NC + p] : __ldg(itabfield<R>(L) + 3 * g + p);
                        v[p] = jacobi_update<R>(u[p * nn + t], v[p], id, omega);
                    }
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) out[p * nn + t] = v[p];
            };
            const int t = w.start + (int)threadIdx.x;
            bool wide = false;  // has a grad C column
            R f[3];
            if (t < nn) {
                int i, j, k;
                cell_ijk(L.n, t, i, j, k);
                const POff o = cell_offsets(L.n, i, j, k);
                const unsigned short* gid = L.gid + t;
                const int g = __ldg(gid);
                if (!A.uniform)
                    wide = __ldg(gid + o.xp) != __ldg(gid + o.xm) || __ldg(gid + o.yp) != __ldg(gid + o.ym) ||
                           __ldg(gid + o.zp) != __ldg(gid + o.zm);
                R gu[3][3];
                const CellAt<R> at{u + t, nn, o};
                R D[3][6];
                row_diffs<R>(K, at, D, gu);
                row_scale(K, D);
                row_sum<M>([&](int n) { return SM ? ts[g * TS + NC + 3 + n] : __ldg(L.rows64 + g * RowN<M>::value + n); }, D, f);
                if (!wide) finish(t, g, f);
            }
            const unsigned ball = __ballot_sync(0xffffffffu, wide);
            if (ball) {
                const int lane = threadIdx.x & 31, lead = __ffs(ball) - 1;
                int at = 0;
                if (lane == lead) at = atomicAdd(&qn, __popc(ball));
                at = __shfl_sync(0xffffffffu, at, lead) + __popc(ball & ((1u << lane) - 1u));
                if (wide) {
                    qt[at] = (unsigned char)threadIdx.x;
#pragma unroll
                    for (int p = 0; p < 3; ++p) qf[p][at] = f[p];
                }
            }
            __syncthreads();
            if ((int)threadIdx.x < qn) {
                const int tq = w.start + (int)qt[threadIdx.x];
                int i, j, k;
                cell_ijk(L.n, tq, i, j, k);
                const POff o = cell_offsets(L.n, i, j, k);
                const unsigned short* gid = L.gid + tq;
                const int off[3][2] = {{o.xp, o.xm}, {o.yp, o.ym}, {o.zp, o.zm}};
                R gu[3][3], col[3][3];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    f[p] = qf[p][threadIdx.x];
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        gu[p][d] = node_diff(K, d, u[p * nn + tq + off[d][0]], u[p * nn + tq + off[d][1]]);
                }
                grad_scale(K, gu);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int gp = __ldg(gid + off[d][0]), gm = __ldg(gid + off[d][1]);
                    if (gp == gm) {
                        col[d][0] = col[d][1] = col[d][2] = R(0);
                    } else {
                        gradC_col_f<M, R>([&](int q) { return slot(gp, q) - slot(gm, q); }, gu, d, col[d]);
                    }
                }
#pragma unroll
                for (int r = 0; r < 3; ++r) f[r] = row_gradc(K, f[r], col[0][r], col[1][r], col[2][r]);
                finish(tq, __ldg(gid), f);
            }
        };
        if (in_smem) body(std::true_type());
        else body(std::false_type());
        if constexpr (OP == CELL_RESID) {
            __syncthreads();
            const int t = w.start + (int)threadIdx.x;
            double v[3] = {0.0, 0.0, 0.0};
            if (t < nn)
#pragma unroll
                for (int p = 0; p < 3; ++p) v[p] = out[p * nn + t];
            block_partials<3>(v, S.part + (size_t)(w.start / kRedChunk) * kPartStride);
        }
    }
}

// The FP32 sweeps of cells on a grain map that march (CellLevelDev::march): a block takes kMarchNodes
// consecutive nodes of a plane and marches up to kz planes in k.  A ring of four planes in shared memory holds the whole rows the
// block's nodes touch, wrapped in y and z as they are loaded (cp.async, one plane ahead), so that a
// displacement is read from global memory once a block and no address in the row is wrapped but along x;
// the walk over solve, cell and level descriptors is paid once per kz planes.  A plane's nodes with a grad C
// column go to a queue, and the block's first threads finish them from the ring.  Any n[0] up to X fills
// the lanes: the nodes of a plane are taken in linear order.  (X: the longest row.  Fixed cycles of 6 cells of
// 128^3 in 64 grains, X = 128, 87.7 ms against 91.3 in one pass; of 46 of 64^3, X = 64, 84.6 against 93.5.)
//
// Bound by latency and by the shared-memory data path together.  128 cells of 16 to 64 nodes an edge:
// smoother sweep 0.415 -> 0.314 ms, residual of the correction 0.417 -> 0.300.  A queue per warp over several
// planes, its neighbours read from global memory, took 0.333; two planes a thread, 96 registers and five
// blocks of 128 threads, 0.356; five blocks of this form (spills) 0.367.
constexpr int kMarchRing = 4;  // planes k - 1, k, k + 1 and the next
template <int X>
constexpr int kMarchW = kMarchNodes - 1 + 4 * X;  // words a component's rows of up to X nodes take at most
template <int M, int X>
constexpr size_t march_smem() {
    return sizeof(float) * (kMarchRing * 3 * kMarchW<X> + kMarchGrains * grain_words<M, float>() + 4 * kMarchNodes + 2);
}
template <int M, int OP, int X>
__global__ void __launch_bounds__(kMarchNodes, kMarchBlocks)
    kb_grain_march(CellArgs A, const Work* __restrict__ tab, int ntab, int kz, int flag) {
    using R = float;
    constexpr int NC = NCoef<M>::value, TS = grain_words<M, R>(), W = kMarchW<X>;
    extern __shared__ __align__(16) unsigned char march_mem[];
    R* const ring = reinterpret_cast<R*>(march_mem);  // [kMarchRing][3][W]
    R* const ts = ring + kMarchRing * 3 * W;
    const int lane = threadIdx.x & 31;
    R* const qf = ts + kMarchGrains * TS;  // [3][kMarchNodes]: a queued node's row so far
    int* const qt = reinterpret_cast<int*>(qf + 3 * kMarchNodes);  // its thread
    int* const qn = qt + kMarchNodes;                                // entries, of even and odd planes
    int have = -1;  // the cell whose numbers are in ts
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        if ((OP == CELL_SMOOTH || !flag) && S.nlev <= 1) continue;
        if (!S.st->active) continue;
        const CellLevelDev& L = A.cells[S.cell].lv[0];
        const int n0 = L.n[0], n1 = L.n[1], n2 = L.n[2], nn = L.nn, sz = n0 * n1;
        const CellVec<R>& V = S.v32[0];
        const R* const u = OP == CELL_SMOOTH && flag ? V.cor2 : V.cor;
        const R* const b = V.res;
        R* const out = OP == CELL_SMOOTH ? (flag ? V.cor : V.cor2) : flag ? V.res : V.rescor;
        const unsigned short* const gids = L.gid;
        const SCoef<R>& K = L.K32;
        const R sc = row_factor(K), omega = omega_of<R>(A);
        const int z0 = w.start / sz, c0 = w.start - z0 * sz, z1 = min(z0 + kz, n2);  // planes z0 .. z1 - 1
        const int cm = min(c0 + (int)threadIdx.x, sz - 1);
        const bool act = c0 + (int)threadIdx.x < sz;
        const int j = cm / n0, i = cm - j * n0;
        // the rows j0 - 1 .. j1 + 1 of a plane, one after another
        const int j0 = c0 / n0, j1 = min(c0 + kMarchNodes - 1, sz - 1) / n0;
        const int words = (j1 - j0 + 3) * n0;
        const int at = (j - j0 + 1) * n0 + i, xp = i == n0 - 1 ? 1 - n0 : 1, xm = i == 0 ? n0 - 1 : -1;
        __syncthreads();  // the block is done with the ring and the numbers
        constexpr int kLoads = (W + kMarchNodes - 1) / kMarchNodes;
        int from[kLoads];  // the thread's words of a plane: their place in the cell's plane, or none
#pragma unroll
        for (int l = 0; l < kLoads; ++l) {
            const int q = threadIdx.x + l * kMarchNodes, r = q / n0;
            int jj = j0 - 1 + r;
            jj = jj < 0 ? jj + n1 : jj >= n1 ? jj - n1 : jj;
            from[l] = q < words ? jj * n0 + (q - r * n0) : -1;
        }
        const auto load = [&](int k) {  // plane k, z0 - 1 <= k <= z1
            const R* src = u + (k < 0 ? k + n2 : k >= n2 ? k - n2 : k) * sz;
            R* dst = ring + (k & (kMarchRing - 1)) * (3 * W) + threadIdx.x;
#pragma unroll
            for (int l = 0; l < kLoads; ++l)
                if (from[l] >= 0)
#pragma unroll
                    for (int p = 0; p < 3; ++p) cp_async<4>(dst + p * W + l * kMarchNodes, src + from[l] + p * nn);
            cp_async_commit();
        };
        load(z0 - 1);
        load(z0);
        load(z0 + 1);
        if (threadIdx.x < 2) qn[threadIdx.x] = 0;
        if (have != S.cell) {
            for (int q = threadIdx.x; q < L.ngrains * TS; q += kMarchNodes) {
                const int g = q / TS, c = q - g * TS;
                if (c < NC) ts[q] = L.tab32[g * NC + c];
                else if (c < NC + 3) ts[q] = L.itab32[3 * g + c - NC];
            }
            have = S.cell;
        }
        const auto finish = [&](int t, int g, const R (&xc)[3], const R (&f)[3]) {
            R v[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                v[p] = row_residual(b[p * nn + t], sc, f[p]);
                if (OP == CELL_SMOOTH) v[p] = jacobi_update<R>(xc[p], v[p], ts[g * TS + NC + p], omega);
            }
#pragma unroll
            for (int p = 0; p < 3; ++p) out[p * nn + t] = v[p];
        };
        const int yo = j == n1 - 1 ? (1 - n1) * n0 : n0, ym = j == 0 ? (n1 - 1) * n0 : -n0;
        for (int k = z0; k < z1; ++k) {
            cp_async_wait<0>();
            __syncthreads();
            if (k + 1 < z1) load(k + 2);
            const auto slot = [&](int kk) { return ring + (kk & (kMarchRing - 1)) * (3 * W); };
            const R* pl[3] = {slot(k - 1) + at, slot(k) + at, slot(k + 1) + at};
            const int t = cm + k * sz;
            const int up = k == n2 - 1 ? (1 - n2) * sz : sz, down = k == 0 ? (n2 - 1) * sz : -sz;
            const unsigned short* gid = gids + t;
            const int g = __ldg(gid);
            bool wide = false;  // has a grad C column
            if (act && !A.uniform)
                wide = __ldg(gid + xp) != __ldg(gid + xm) || __ldg(gid + yo) != __ldg(gid + ym) ||
                       __ldg(gid + up) != __ldg(gid + down);
            R f[3], gu[3][3];
            row_interior<M, R>(
                K,
                [&](int p, int a, int bb, int c) {
                    return pl[c + 1][p * W + (a > 0 ? xp : a < 0 ? xm : 0) + (bb > 0 ? n0 : bb < 0 ? -n0 : 0)];
                },
                [&](int q) { return ts[g * TS + q]; }, gu, f);
            if (act && !wide) {
                const R xc[3] = {pl[1][0], pl[1][W], pl[1][2 * W]};
                finish(t, g, xc, f);
            }
            int* const n = qn + (k & 1);
            const unsigned ball = __ballot_sync(0xffffffffu, wide);
            if (ball) {
                const int lead = __ffs(ball) - 1;
                int q = 0;
                if (lane == lead) q = atomicAdd(n, __popc(ball));
                q = __shfl_sync(0xffffffffu, q, lead) + __popc(ball & ((1u << lane) - 1u));
                if (wide) {
                    qt[q] = threadIdx.x;
#pragma unroll
                    for (int p = 0; p < 3; ++p) qf[p * kMarchNodes + q] = f[p];
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) qn[(k + 1) & 1] = 0;  // read last before this plane's first barrier
            if ((int)threadIdx.x < *n) {
                const int c = c0 + qt[threadIdx.x], jj = c / n0, ii = c - jj * n0, tq = c + k * sz;
                const int aq = (jj - j0 + 1) * n0 + ii;
                const int qxp = ii == n0 - 1 ? 1 - n0 : 1, qxm = ii == 0 ? n0 - 1 : -1;
                const int goff[3][2] = {{qxp, qxm},
                                        {jj == n1 - 1 ? (1 - n1) * n0 : n0, jj == 0 ? (n1 - 1) * n0 : -n0}, {up, down}};
                const R *qm = slot(k - 1) + aq, *qc = slot(k) + aq, *qp = slot(k + 1) + aq;
                R gv[3][3], col[3][3], fq[3];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    fq[p] = qf[p * kMarchNodes + threadIdx.x];
                    gv[p][0] = node_diff(K, 0, qc[p * W + qxp], qc[p * W + qxm]);
                    gv[p][1] = node_diff(K, 1, qc[p * W + n0], qc[p * W - n0]);
                    gv[p][2] = node_diff(K, 2, qp[p * W], qm[p * W]);
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int gp = __ldg(gids + tq + goff[d][0]), gm = __ldg(gids + tq + goff[d][1]);
                    if (gp == gm) {
                        col[d][0] = col[d][1] = col[d][2] = R(0);
                    } else {
                        const R *cp = ts + gp * TS, *cq = ts + gm * TS;
                        gradC_col_f<M, R>([&](int u_) { return cp[u_] - cq[u_]; }, gv, d, col[d]);
                    }
                }
#pragma unroll
                for (int r = 0; r < 3; ++r) fq[r] = row_gradc(K, fq[r], col[0][r], col[1][r], col[2][r]);
                const R xc[3] = {qc[0], qc[W], qc[2 * W]};
                finish(tq, __ldg(gids + tq), xc, fq);
            }
        }
    }
}

// b = -sum_d (d_d C) : E e_d, with per-chunk sums
template <int M>
__global__ void __launch_bounds__(kCellThreads) kb_rhs(CellArgs A, const Work* __restrict__ tab, int ntab) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        const CellLevelDev& L = A.cells[S.cell].lv[0];
        const int t = w.start + threadIdx.x;
        const int nn = L.nn;
        double v[3] = {0.0, 0.0, 0.0};
        if (t < nn) {
            double g[3][3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int c = 0; c < 3; ++c) g[a][c] = S.E[3 * a + c];
            if (!A.uniform) {
                int i, j, k;
                cell_ijk(L.n, t, i, j, k);
                const POff o = cell_offsets(L.n, i, j, k);
                double gc[3];
                cell_gradC<M, double>(L.K64, L.C64, nn, t, o, g, gc);
#pragma unroll
                for (int p = 0; p < 3; ++p) v[p] = -gc[p];
            }
#pragma unroll
            for (int p = 0; p < 3; ++p) S.b[p * nn + t] = v[p];
        }
        block_partials<3>(v, S.part + (size_t)(w.start / kRedChunk) * kPartStride);
    }
}

// per-chunk sums of x
__global__ void __launch_bounds__(kCellThreads) kb_xpart(CellArgs A, const Work* __restrict__ tab, int ntab) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        const int nn = A.cells[S.cell].lv[0].nn;
        const int t = w.start + threadIdx.x;
        double v[3] = {0.0, 0.0, 0.0};
        if (t < nn)
#pragma unroll
            for (int p = 0; p < 3; ++p) v[p] = S.x[p * nn + t];
        block_partials<3>(v, S.part + (size_t)(w.start / kRedChunk) * kPartStride);
    }
}

// per-chunk sums of the stress C : (E + grad w)
template <int M>
__global__ void __launch_bounds__(kCellThreads) kb_stress(CellArgs A, const Work* __restrict__ tab, int ntab) {
    constexpr int NC = NCoef<M>::value;
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        const CellLevelDev& L = A.cells[S.cell].lv[0];
        const int nn = L.nn;
        const int t = w.start + threadIdx.x;
        double v[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) v[q] = 0.0;
        if (t < nn) {
            int i, j, k;
            cell_ijk(L.n, t, i, j, k);
            const POff o = cell_offsets(L.n, i, j, k);
            const int ox[3] = {o.xp, o.yp, o.zp}, om[3] = {o.xm, o.ym, o.zm};
            double g[3][3], a[NC], s[3][3];
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    g[p][d] = S.E[3 * p + d] + (S.x[p * nn + t + ox[d]] - S.x[p * nn + t + om[d]]) * L.K64.h[d];
#pragma unroll
            for (int q = 0; q < NC; ++q) a[q] = L.C64[q * nn + t];
            stress_of<M, double>(a, g, s);
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int d = 0; d < 3; ++d) v[3 * p + d] = s[p][d];
        }
        block_partials<9>(v, S.part + (size_t)(w.start / kRedChunk) * kPartStride);
    }
}

// per-solve mean over its partials (one block per solve, fixed order)
__global__ void __launch_bounds__(kBottomThreads) kb_mean(CellArgs A, const int* slots, int which, int all) {
    __shared__ BlkRed sh;
    const SolveDev& S = A.solves[slots ? slots[blockIdx.x] : blockIdx.x];
    if (!all && !S.st->active) return;
    const int nn = A.cells[S.cell].lv[0].nn;
    const int nch = (nn + kRedChunk - 1) / kRedChunk;
    const int nq = which == 2 ? 9 : 3;
    double* dst = which == 0 ? S.st->mean : which == 1 ? S.st->wmean : S.st->sig;
    for (int q = 0; q < nq; ++q) {
        double s = 0.0;
        for (int c = threadIdx.x; c < nch; c += blockDim.x) s += S.part[(size_t)c * kPartStride + q];
        s = blk_sum(s, sh);
        if (threadIdx.x == 0) dst[q] = s / (double)nn;
    }
}

__device__ __forceinline__ double nan_to_inf(double a) { return a != a ? INFINITY : a; }

__device__ __forceinline__ void block_max_to(double v, unsigned long long* dst) {
    __shared__ double red[kCellThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s = fmax(s, red[q]);
        atomicMax(dst, (unsigned long long)__double_as_longlong(s));
    }
    __syncthreads();
}

template <class R>
__global__ void __launch_bounds__(kCellThreads) kb_project(CellArgs A, const Work* __restrict__ tab, int ntab, int vec) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        if (vec == 0 && !S.st->active) continue;
        const int nn = A.cells[S.cell].lv[0].nn;
        const int t = w.start + threadIdx.x;
        double mx = 0.0;
        if (t < nn) {
            if (vec == 0) {
                const CellVec<R>& V = vec_of<R>(S, 0);
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const double v = S.r[p * nn + t] - S.st->mean[p];
                    S.r[p * nn + t] = v;
                    V.res[p * nn + t] = (R)v;
                    mx = fmax(mx, nan_to_inf(fabs(v)));
                }
            } else if (vec == 1) {
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const double v = S.b[p * nn + t] - S.st->mean[p];
                    S.b[p * nn + t] = v;
                    mx = fmax(mx, nan_to_inf(fabs(v)));
                }
            } else {
#pragma unroll
                for (int p = 0; p < 3; ++p) S.x[p * nn + t] -= S.st->wmean[p];
            }
        }
        if (vec != 2) block_max_to(mx, vec == 0 ? &S.st->norm_bits : &S.st->bnorm_bits);
    }
}

template <class R>
__global__ void __launch_bounds__(kCellThreads) kb_update(CellArgs A, const Work* __restrict__ tab, int ntab) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        if (!S.st->active) continue;
        const int nn = A.cells[S.cell].lv[0].nn;
        const int t = w.start + threadIdx.x;
        if (t >= nn) continue;
        const R* cor = vec_of<R>(S, 0).cor;
#pragma unroll
        for (int p = 0; p < 3; ++p) S.x[p * nn + t] += (double)cor[p * nn + t];
    }
}

__global__ void __launch_bounds__(kCellThreads) kb_zero_x(CellArgs A, const Work* __restrict__ tab, int ntab) {
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const SolveDev& S = A.solves[w.id];
        const int nn = A.cells[S.cell].lv[0].nn;
        const int t = w.start + threadIdx.x;
        if (t >= nn) continue;
#pragma unroll
        for (int p = 0; p < 3; ++p) S.x[p * nn + t] = 0.0;
    }
}

__global__ void kb_begin(CellArgs A, const int* slots, int nsolves) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nsolves; s += gridDim.x * blockDim.x) {
        CellStatus* st = A.solves[slots ? slots[s] : s].st;
        st->active = 1;
        st->iters = 0;
        st->conv = 0;
        st->bfail = 0;
        st->norm_bits = 0ull;
        st->bnorm_bits = 0ull;
    }
}

// convergence test of every active solve (MLMG: ||r|| <= max(tol_abs, tol_rel max(||b||, ||r0||)))
__global__ void __launch_bounds__(1024) kb_status(CellArgs A, const int* slots, int nsolves, int first,
                                                  double tol_rel, double tol_abs, int max_iter, int* count,
                                                  int* active_out) {
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    int mine = 0;
    for (int s = threadIdx.x; s < nsolves; s += blockDim.x) {
        CellStatus* st = A.solves[slots ? slots[s] : s].st;
        if (active_out) active_out[s] = 0;
        if (!st->active) continue;
        const double norm = __longlong_as_double((long long)st->norm_bits);
        st->norm_bits = 0ull;
        st->resn = norm;
        if (first) {
            const double bn = __longlong_as_double((long long)st->bnorm_bits);
            st->bnorm = bn;
            st->res0 = norm;
            const double maxn = bn >= norm ? bn : norm;
            st->target = fmax(tol_abs, fmax(tol_rel, 1.e-16) * maxn);
        }
        if (!isfinite(norm)) {
            st->active = 0;
            st->conv = 0;
        } else if (norm <= st->target) {
            st->active = 0;
            st->conv = 1;
        } else if (st->iters >= max_iter) {
            st->active = 0;
            st->conv = 0;
        } else {
            st->iters += 1;
            ++mine;
            if (active_out) active_out[s] = 1;
        }
    }
    atomicAdd(&total, mine);
    __syncthreads();
    if (threadIdx.x == 0) *count = total;
}

// Loop condition of the batch's device-side iteration (the body of a conditional WHILE graph
// node): continue while some solve is active and fewer than `limit` iterations have run.  The
// counter bounds the loop whatever the status says.
__global__ void kb_loop_cond(cudaGraphConditionalHandle h, const int* count, int* iter, int limit) {
    const int it = *iter + 1;
    *iter = it;
    cudaGraphSetConditional(h, (*count > 0 && it < limit) ? 1u : 0u);
}
// ------------------------------------------------------------------ cell set-up
template <int M>
__global__ void __launch_bounds__(kCellThreads) kb_coarsen_C(CellArgs A, const Work* __restrict__ tab, int ntab,
                                                             int m) {
    constexpr int NC = NCoef<M>::value;
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const CellDev& Cd = A.cells[w.id];
        const CellLevelDev& Lf = Cd.lv[m - 1];
        const CellLevelDev& Lc = Cd.lv[m];
        const int t = w.start + threadIdx.x;
        if (t >= Lc.nn) continue;
        int I, J, K;
        cell_ijk(Lc.n, t, I, J, K);
        for (int q = 0; q < NC; ++q) Lc.C64[q * Lc.nn + t] = cell_restrict<double>(Lf.C64 + q * Lf.nn, Lf.n, I, J, K);
    }
}

template <int M>
__global__ void __launch_bounds__(kCellThreads) kb_diag(CellArgs A, const Work* __restrict__ tab, int ntab, int m,
                                                        int* nan_flag) {
    constexpr int NC = NCoef<M>::value;
    for (int e = blockIdx.x; e < ntab; e += gridDim.x) {
        const Work w = tab[e];
        const CellLevelDev& L = A.cells[w.id].lv[m];
        const int t = w.start + threadIdx.x;
        const int nn = L.nn;
        if (t >= nn) continue;
        double d[3];
        cell_diag<M, double>(L.K64, L.C64, nn, t, d);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            if (!(d[p] == d[p]) || d[p] == 0.0) atomicExch(nan_flag, 1);
            L.D64[p * nn + t] = d[p];
            L.I64[p * nn + t] = 1.0 / d[p];
            L.I32[p * nn + t] = (float)(1.0 / d[p]);
        }
        for (int q = 0; q < NC; ++q) L.C32[q * nn + t] = (float)L.C64[q * nn + t];
    }
}

// Voronoi cell model: node stiffness = table row of the nearest seed (minimum-image distance in
// the periodic cell; ties go to the lower seed index), the semantics of IC::Voronoi
// (src/IC/Voronoi.H:47-101) on a periodic cell.
template <int M>
__global__ void __launch_bounds__(kCellThreads) kb_grains(CellLevelDev L, double lx, double ly, double lz,
                                                          const double* __restrict__ seeds, int ng,
                                                          const double* __restrict__ table) {
    constexpr int NC = NCoef<M>::value;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L.nn) return;
    int i, j, k;
    cell_ijk(L.n, t, i, j, k);
    const double x = i * (lx / L.n[0]), y = j * (ly / L.n[1]), z = k * (lz / L.n[2]);
    int best = 0;
    double bd = 0.0;
    for (int g = 0; g < ng; ++g) {
        double dx = x - seeds[3 * g], dy = y - seeds[3 * g + 1], dz = z - seeds[3 * g + 2];
        dx -= lx * rint(dx / lx);
        dy -= ly * rint(dy / ly);
        dz -= lz * rint(dz / lz);
        const double d = dx * dx + dy * dy + dz * dz;
        if (g == 0 || d < bd) { bd = d; best = g; }
    }
    if (L.gid) L.gid[t] = (unsigned short)best;
    for (int q = 0; q < NC; ++q) L.C64[q * L.nn + t] = table[best * NC + q];
}

// per-grain FP32 stiffness, FP64 row numbers and 1/diagonal (the values kb_diag gives the grain's nodes)
template <int M>
__global__ void kb_grain_tables(CellLevelDev L) {
    constexpr int NC = NCoef<M>::value;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= L.ngrains) return;
    double d[3];
    cell_diag<M, double>(L.K64, L.tab64 + g * NC, 1, 0, d);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        L.itab64[3 * g + p] = 1.0 / d[p];
        L.itab32[3 * g + p] = (float)(1.0 / d[p]);
    }
    for (int q = 0; q < NC; ++q) L.tab32[g * NC + q] = (float)L.tab64[g * NC + q];
#pragma unroll
    for (int n = 0; n < RowN<M>::value; ++n)
        L.rows64[g * RowN<M>::value + n] = row_number<M>([&](int q) { return L.tab64[g * NC + q]; }, n);
}

inline int grid_of(int ntab, Shape sh) { return ntab < sh.grid ? ntab : sh.grid; }

template <class F>
void by_prec(int prec, F&& f) {
    if (prec == 1) f(float());
    else f(double());
}

}  // namespace

// ------------------------------------------------------------------ launchers
// the variants of a stencil kernel that the cells present need: f(true) on grain maps, f(false) per node
template <class F>
void by_rep(int reps, F&& f) {
    if (reps & kRepNode) f(std::false_type());
    if (reps & (kRepGrains | kRepMarch)) f(std::true_type());
}
// grain maps, smoother and correction residual: two passes in FP64; in FP32 marching cells apart from the
// others, which take one pass
template <int M, class R, int OP>
void launch_grain_sweep(const CellArgs& A, const Work* tab, int ntab, Shape sh, int flag, int reps, const MarchTab& mt,
                        cudaStream_t st) {
    if (sizeof(R) == 8 && mt.two_pass) {
        if (reps & (kRepGrains | kRepMarch)) {
            kb_grain_sweep<M, OP><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, flag);
            launched();
        }
        return;
    }
    if (reps & (sizeof(R) == 8 ? kRepGrains | kRepMarch : kRepGrains)) {
        if constexpr (OP == CELL_SMOOTH)
            kb_smooth<M, R, false, true><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, 0, flag);
        else
            kb_rescor<M, R, true><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, 0, flag);
        launched();
    }
    if constexpr (sizeof(R) == 4) {
        if (reps & kRepMarch) {
            const auto go = [&](auto x) {
                constexpr int X = decltype(x)::value;
                constexpr size_t smem = march_smem<M, X>();
                static std::once_flag once;
                std::call_once(once, [] {
                    AE_CUDA_CHECK(cudaFuncSetAttribute(kb_grain_march<M, OP, X>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                });
                kb_grain_march<M, OP, X><<<std::min(mt.n, mt.grid), kMarchNodes, smem, st>>>(A, mt.tab, mt.n, mt.kz, flag);
                launched();
            };
            if (mt.rows <= kMarchXs) go(std::integral_constant<int, kMarchXs>());
            else go(std::integral_constant<int, kMarchX>());
        }
    }
}

void cells_launch_smooth(int model, int prec, bool zero, const CellArgs& A, const Work* tab, int ntab, Shape sh,
                         int m, int from2, int reps, const MarchTab& mt, cudaStream_t st) {
    if (ntab == 0) return;
    dispatch_model<double>(model, [&](auto mm) {
        constexpr int M = decltype(mm)::value;
        by_prec(prec, [&](auto r) {
            using R = decltype(r);
            if (zero) {
                by_rep(reps, [&](auto gr) {
                    kb_smooth<M, R, true, decltype(gr)::value><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, m, from2);
                    launched();
                });
                return;
            }
            if (reps & kRepNode) {
                kb_smooth<M, R, false, false><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, m, from2);
                launched();
            }
            launch_grain_sweep<M, R, CELL_SMOOTH>(A, tab, ntab, sh, from2, reps, mt, st);
        });
    });
}
void cells_launch_copy2(int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m, cudaStream_t st) {
    if (ntab == 0) return;
    by_prec(prec, [&](auto r) { kb_copy2<decltype(r)><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, m, 0); });
    launched();
}
void cells_launch_fill0(int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m, cudaStream_t st) {
    if (ntab == 0) return;
    by_prec(prec, [&](auto r) { kb_copy2<decltype(r)><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, m, 1); });
    launched();
}
void cells_launch_rescor(int model, int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m,
                         int inplace, int reps, const MarchTab& mt, cudaStream_t st) {
    if (ntab == 0) return;
    dispatch_model<double>(model, [&](auto mm) {
        constexpr int M = decltype(mm)::value;
        by_prec(prec, [&](auto r) {
            using R = decltype(r);
            if (reps & kRepNode) {
                kb_rescor<M, R, false><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, m, inplace);
                launched();
            }
            launch_grain_sweep<M, R, CELL_RESCOR>(A, tab, ntab, sh, inplace, reps, mt, st);
        });
    });
}
void cells_launch_restrict(int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m, cudaStream_t st) {
    if (ntab == 0) return;
    by_prec(prec, [&](auto r) { kb_restrict<decltype(r)><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, m); });
    launched();
}
void cells_launch_interp(int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m, cudaStream_t st) {
    if (ntab == 0) return;
    by_prec(prec, [&](auto r) { kb_interp<decltype(r)><<<grid_of(ntab, sh), sh.chunk, 0, st>>>(A, tab, ntab, m); });
    launched();
}
void cells_launch_bottom(int model, int prec, const CellArgs& A, int nsolves, const KrylovParams& kp,
                         cudaStream_t st) {
    if (nsolves == 0) return;
    dispatch_model<double>(model, [&](auto mm) {
        constexpr int M = decltype(mm)::value;
        by_prec(prec, [&](auto r) {
            kb_bottom<M, decltype(r)><<<nsolves, kBottomThreads, kBottomSmemBytes, st>>>(A, kp, (int)kBottomSmemBytes);
        });
    });
    launched();
}
void cells_launch_resid_top(int model, const CellArgs& A, const Work* tab, int ntab, int reps, bool two_pass,
                            cudaStream_t st) {
    if (ntab == 0) return;
    dispatch_model<double>(model, [&](auto mm) {
        by_rep(reps, [&](auto gr) {
            constexpr int M = decltype(mm)::value;
            constexpr bool GR = decltype(gr)::value;
            if (GR && two_pass) kb_grain_sweep<M, CELL_RESID><<<ntab, kRedChunk, 0, st>>>(A, tab, ntab, 0);
            else kb_resid_top<M, GR><<<ntab, kRedChunk, 0, st>>>(A, tab, ntab);
            launched();
        });
    });
}
void cells_launch_rhs(int model, const CellArgs& A, const Work* tab, int ntab, cudaStream_t st) {
    if (ntab == 0) return;
    dispatch_model<double>(model, [&](auto mm) { kb_rhs<decltype(mm)::value><<<ntab, kRedChunk, 0, st>>>(A, tab, ntab); });
    launched();
}
void cells_launch_mean(const CellArgs& A, const int* slots, int nsolves, int which, int all, cudaStream_t st) {
    if (nsolves == 0) return;
    kb_mean<<<nsolves, kBottomThreads, 0, st>>>(A, slots, which, all);
    launched();
}
void cells_launch_project(int prec, int vec, const CellArgs& A, const Work* tab, int ntab, cudaStream_t st) {
    if (ntab == 0) return;
    by_prec(prec, [&](auto r) { kb_project<decltype(r)><<<ntab, kRedChunk, 0, st>>>(A, tab, ntab, vec); });
    launched();
}
void cells_launch_update(int prec, const CellArgs& A, const Work* tab, int ntab, cudaStream_t st) {
    if (ntab == 0) return;
    by_prec(prec, [&](auto r) { kb_update<decltype(r)><<<ntab, kRedChunk, 0, st>>>(A, tab, ntab); });
    launched();
}
void cells_launch_xpart(const CellArgs& A, const Work* tab, int ntab, cudaStream_t st) {
    if (ntab == 0) return;
    kb_xpart<<<ntab, kRedChunk, 0, st>>>(A, tab, ntab);
    launched();
}
void cells_launch_stress(int model, const CellArgs& A, const Work* tab, int ntab, cudaStream_t st) {
    if (ntab == 0) return;
    dispatch_model<double>(model, [&](auto mm) {
        kb_stress<decltype(mm)::value><<<ntab, kRedChunk, 0, st>>>(A, tab, ntab);
    });
    launched();
}
void cells_launch_status(const CellArgs& A, const int* slots, int nsolves, int first, double tol_rel, double tol_abs,
                         int max_iter, int* count, int* active_out, cudaStream_t st) {
    kb_status<<<1, 1024, 0, st>>>(A, slots, nsolves, first, tol_rel, tol_abs, max_iter, count, active_out);
    launched();
}
void cells_launch_begin(const CellArgs& A, const int* slots, int nsolves, cudaStream_t st) {
    if (nsolves == 0) return;
    kb_begin<<<(nsolves + 255) / 256, 256, 0, st>>>(A, slots, nsolves);
    launched();
}
void cells_launch_zero_x(const CellArgs& A, const Work* tab, int ntab, cudaStream_t st) {
    if (ntab == 0) return;
    kb_zero_x<<<ntab, kRedChunk, 0, st>>>(A, tab, ntab);
    launched();
}
void cells_launch_coarsen_C(int model, const CellArgs& A, const Work* tab, int ntab, int m, cudaStream_t st) {
    if (ntab == 0) return;
    dispatch_model<double>(model, [&](auto mm) {
        kb_coarsen_C<decltype(mm)::value><<<ntab, kRedChunk, 0, st>>>(A, tab, ntab, m);
    });
    launched();
}
void cells_launch_grains(int model, const CellLevelDev& L, const double len[3], const double* seeds, int ng,
                         const double* table, cudaStream_t st) {
    if (L.nn == 0) return;
    dispatch_model<double>(model, [&](auto mm) {
        kb_grains<decltype(mm)::value><<<(L.nn + kCellThreads - 1) / kCellThreads, kCellThreads, 0, st>>>(
            L, len[0], len[1], len[2], seeds, ng, table);
    });
    launched();
    if (L.gid && L.ngrains > 0) {
        dispatch_model<double>(model, [&](auto mm) {
            kb_grain_tables<decltype(mm)::value><<<(L.ngrains + 127) / 128, 128, 0, st>>>(L);
        });
        launched();
    }
}
void cells_launch_diag(int model, const CellArgs& A, const Work* tab, int ntab, int m, int* nan_flag,
                       cudaStream_t st) {
    if (ntab == 0) return;
    dispatch_model<double>(model, [&](auto mm) {
        kb_diag<decltype(mm)::value><<<ntab, kRedChunk, 0, st>>>(A, tab, ntab, m, nan_flag);
    });
    launched();
}

void cells_launch_loop_cond(cudaGraphConditionalHandle h, const int* count, int* iter, int limit, cudaStream_t st) {
    kb_loop_cond<<<1, 1, 0, st>>>(h, count, iter, limit);
    launched();
}

}  // namespace ae
