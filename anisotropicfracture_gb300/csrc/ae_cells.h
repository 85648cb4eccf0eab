// Batched periodic cells: device descriptors shared by the kernels (ae_cells_kernels.cu) and the
// host engine (ae_cells.cu).
//
// A cell is one periodic RVE with its own multigrid hierarchy (stiffness, diagonal, FP32 copies
// per level); a solve is one macroscopic displacement gradient E on a cell, with its own vectors.
// Kernels run over work tables whose entries name a solve (or a cell) and a run of consecutive
// nodes of one level, so one launch covers every live solve whatever its size.  Every per-solve
// reduction uses a chunking and tree fixed by the solve's own size, so a solve's arithmetic does
// not depend on which other solves share the launch.
#pragma once
#include <cuda_runtime.h>

#include "ae_device.cuh"
#include "ae_krylov.cuh"

namespace ae {

constexpr int kMaxCellLevels = 8;
constexpr int kRedChunk = 256;  // nodes per reduction partial (fixed: results must not depend on tuning)
constexpr int kPartStride = 9;  // doubles per partial slot

struct CellLevelDev {
    int n[3];
    int nn;
    double* C64;
    double* D64;
    double* I64;  // 1 / D
    float* C32;
    float* I32;
    SCoef<double> K64;
    SCoef<float> K32;
    // Voronoi cells, finest level only: grain id per node and per-grain tables of the stiffness
    // (ncoef), the FP64 row's numbers (cell_row_numbers) and 1/diagonal (3).  gid == nullptr: per-node arrays only.  The kernels of
    // the finest level read these instead of the per-node arrays (same values, far fewer bytes).
    unsigned short* gid;
    int ngrains;
    int march;  // in the engine's descriptors: whether the FP32 finest-level sweeps march
    double* tab64;
    float* tab32;
    double* rows64;
    double* itab64;
    float* itab32;
};
// numbers of an FP64 row for a model of ncoef slots (RowN)
inline int cell_row_numbers(int ncoef) { return ncoef == 21 ? 36 : ncoef; }
struct CellDev {
    int nlev;
    int pad_;
    CellLevelDev lv[kMaxCellLevels];
};

template <class R>
struct CellVec {
    R* cor;
    R* cor2;    // second Jacobi buffer
    R* res;
    R* rescor;
};

// device-resident status of one solve
struct CellStatus {
    int active;
    int iters;
    int conv;
    int bfail;
    unsigned long long norm_bits;  // max |r| of the current residual (bit pattern, atomicMax)
    unsigned long long bnorm_bits;
    double res0, target, resn, bnorm;
    double mean[3];   // mean of the last residual: the body force
    double wmean[3];
    double sig[9];    // cell-averaged stress
};

struct SolveDev {
    int cell;       // slot of its cell in the live cell table
    int nlev;
    double* x;      // w, level 0, FP64
    double* b;
    double* r;
    double* part;   // ceil(nn0 / kRedChunk) * kPartStride doubles
    double* bwork;  // bottom: 10 vectors of 3 nn_bottom doubles (8 work, b, x)
    CellStatus* st;
    double E[9];
    CellVec<float> v32[kMaxCellLevels];
    CellVec<double> v64[kMaxCellLevels];
};

struct Work {
    int id;     // solve (or cell) slot
    int start;  // first node of the run
};

struct CellArgs {
    const CellDev* cells;
    const SolveDev* solves;
    int uniform;
    int sweeps;
    double omega;
    float omega32;
};

// launch shape of one table: nodes per entry (= threads per block) and grid size
struct Shape {
    int chunk;
    int grid;
};

// How the finest-level sweeps of cells on a grain map run (CellEngine::rebuild); every way computes the same
// bits.  "nodes" below are those of all solves together.
//
// FP32: marching (kb_grain_march) or one pass (kb_smooth, kb_rescor).  A cell can march when its rows and its
// grains' numbers fit the kernel's shared memory: rows of up to 128 nodes in the wider of two forms (51 KB a
// block, still four an SM), up to 64 in the other (38 KB).  Marching wins once its blocks, which take several
// planes each, fill the chip a few times: for 21 or 2 slots from 1.5 million nodes on, for 9 slots, which leave
// less to save, from 3 million, with rows over 64 nodes from 5 million.  Time of a fixed number of cycles, ms,
// one pass / marching:
//   21 slots   24 cells of 24^3 (0.33 M nodes) 7.2 / 8.0   6 of 64^3 (1.6 M) 14.0 / 13.6   46 (12 M) 89 / 80
//    9 slots    6 cells of 64^3 8.9 / 9.3                 11 (2.9 M) 15.3 / 15.3           46 60 / 54
//   rows of 96  3 cells (2.7 M) 21.2 / 22.0                7 (6.2 M) 46.0 / 44.2           14 (12 M) 88 / 84
constexpr int kMarchX = 128, kMarchXs = 64, kMarchGrains = 96;
constexpr long long kMarchMinNodes = 1500000, kMarchMinNodesD = 3000000, kMarchMinNodesX = 5000000;
constexpr int kMarchNodes = 256, kMarchBlocks = 4;  // nodes of a plane a block takes, resident blocks per SM
inline bool cell_can_march(const CellLevelDev& L, int rows) {
    return L.gid != nullptr && L.n[0] <= rows && L.ngrains <= kMarchGrains;
}
// FP64: two passes (kb_grain_sweep) or one.  Two passes pack the nodes at grain boundaries, but run one after
// the other and start by loading the grains' numbers: one pass wins on little work, the more so the more of
// the nodes lie at a boundary.  FP64 cycles, ms, two passes / one: one cell of 16^3 in 32 grains 1.80 / 1.59,
// 48 of them (0.2 M nodes) 5.22 / 5.04, one of 48^3 3.16 / 3.27, 24 of 16^3 in 8 grains 2.29 / 2.37, 24 of
// 24^3 in 32 (0.33 M) 6.69 / 6.95, 24 of 32^3 (0.8 M) 12.9 / 14.2.
constexpr long long kTwoPassMinNodes = 300000, kTwoPassMinNodesWide = 90000;
constexpr int kTwoPassGrainNodes = 512;  // nodes per grain from which the lower of the two limits holds
// the marching cells' work: entry start = first node of a run of nodes in plane z, kz planes from there on
struct MarchTab {
    const Work* tab;
    int n, kz, grid;
    int rows;       // the longest row among the cells
    bool two_pass;  // the FP64 sweeps of all cells on a grain map: kb_grain_sweep, or one pass
};

// ---- launchers (ae_cells_kernels.cu); model 0 ISO, 1 MM, 2 DIAG
// reps (stencil launchers): the finest-level representations present; each entry is served by the
// variant that matches its cell, coarser levels always take the per-node variant.
constexpr int kRepNode = 1, kRepGrains = 2, kRepMarch = 4;
void cells_launch_smooth(int model, int prec, bool zero, const CellArgs& A, const Work* tab, int ntab, Shape sh,
                         int m, int from2, int reps, const MarchTab& mt, cudaStream_t st);
void cells_launch_copy2(int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m, cudaStream_t st);
void cells_launch_fill0(int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m, cudaStream_t st);
// rescor_m = res_m - A cor_m (inplace: res_m -= A cor_m)
void cells_launch_rescor(int model, int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m,
                         int inplace, int reps, const MarchTab& mt, cudaStream_t st);
// res_{m+1} = R rescor_m, tab over level m+1 nodes
void cells_launch_restrict(int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m, cudaStream_t st);
// cor_m += I cor_{m+1}, tab over level m nodes
void cells_launch_interp(int prec, const CellArgs& A, const Work* tab, int ntab, Shape sh, int m, cudaStream_t st);
void cells_launch_bottom(int model, int prec, const CellArgs& A, int nsolves, const KrylovParams& kp,
                         cudaStream_t st);
// FP64 top level (tab: level-0 runs of kRedChunk nodes, one block each)
void cells_launch_resid_top(int model, const CellArgs& A, const Work* tab, int ntab, int reps, bool two_pass,
                            cudaStream_t st);
void cells_launch_rhs(int model, const CellArgs& A, const Work* tab, int ntab, cudaStream_t st);
// per-solve mean of the partials: which 0 residual/rhs -> mean, 1 w -> wmean, 2 stress -> sig
// (slots: the solve slots to visit, nullptr = 0 .. nsolves-1)
void cells_launch_mean(const CellArgs& A, const int* slots, int nsolves, int which, int all, cudaStream_t st);
// vec 0: r (active solves): r -= mean, norm, res_0 = r in the cycle precision
// vec 1: b (setup, every solve): b -= mean, bnorm
// vec 2: x (final, every solve): x -= wmean
void cells_launch_project(int prec, int vec, const CellArgs& A, const Work* tab, int ntab, cudaStream_t st);
void cells_launch_update(int prec, const CellArgs& A, const Work* tab, int ntab, cudaStream_t st);
void cells_launch_xpart(const CellArgs& A, const Work* tab, int ntab, cudaStream_t st);
void cells_launch_stress(int model, const CellArgs& A, const Work* tab, int ntab, cudaStream_t st);
// status: first = 1 for the initial residual; count receives the number of solves still active,
// active_out (optional, one int per visited solve) their flags
void cells_launch_status(const CellArgs& A, const int* slots, int nsolves, int first, double tol_rel, double tol_abs,
                         int max_iter, int* count, int* active_out, cudaStream_t st);
// *iter += 1; the WHILE node's condition = (*count > 0 && *iter < limit)
void cells_launch_loop_cond(cudaGraphConditionalHandle h, const int* count, int* iter, int limit, cudaStream_t st);
void cells_launch_begin(const CellArgs& A, const int* slots, int nsolves, cudaStream_t st);
void cells_launch_zero_x(const CellArgs& A, const Work* tab, int ntab, cudaStream_t st);
// cell set-up (tab over cell ids): C_{m} = R C_{m-1}; D, 1/D, FP32 copies; NaN flag
void cells_launch_coarsen_C(int model, const CellArgs& A, const Work* tab, int ntab, int m, cudaStream_t st);
// level-0 stiffness of a Voronoi cell from seeds (ng x 3, in the cell's length units) and a
// per-grain coefficient table (ng x ncoef); device pointers.  When L.gid is set, also the grain
// ids and L's grain tables (L.tab64 must hold the table, L.ngrains = ng).
void cells_launch_grains(int model, const CellLevelDev& L, const double len[3], const double* seeds, int ng,
                         const double* table, cudaStream_t st);
void cells_launch_diag(int model, const CellArgs& A, const Work* tab, int ntab, int m, int* nan_flag, cudaStream_t st);

}  // namespace ae
