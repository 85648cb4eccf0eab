// Split sweeps on Voronoi (grain-map) levels, FP32 and FP64: a tiled kernel over the interior box plus
// the per-node code over a list of the nodes that need it (see ae_split.cu).
#pragma once
#include <cuda_runtime.h>

#include "ae_launch.h"
#include "ae_split_rules.h"

namespace ae {

struct SplitList {
    unsigned long long* list = nullptr;  // nodes outside the interior box: packed offsets from the
                                         // storage box's low corner
    long long n = 0;
    unsigned long long* list_r = nullptr;  // the same for the residual's region grow(valid,1) ∩ domain
    long long n_r = 0;
    unsigned* gidm = nullptr;            // per stored node: grain id | grad C directions << 16
    double* rows64 = nullptr;            // per grain: the numbers of its interior row (FP64 sweeps)
    int kz = 0;                          // planes per block of the tiled kernel (0: chosen by its rule)
};
// grain ids the split sweep can carry next to its 3-bit direction mask
constexpr int kSplitMaxGrains = 1 << 16;

// whether a level's layout allows the split sweep (row pitch a multiple of 4 nodes)
bool split_supported(const Geo& g);
// whether the split sweep can write a view
template <class R>
bool split_out(const View<R>& v) {
    return split_range(v.sz, v.sc);
}
// Build the node list and the id/mask array of a grain-map level (gid laid out like the level's
// storage, at most kSplitMaxGrains grains) and the grains' row numbers; allocates sl's arrays with
// cudaMalloc and returns the list's length.  scratch_count: one device counter.  Synchronises the
// stream.
long long split_build(const Geo& g, int model, View<const unsigned short> gid, int ngrains, const double* tab,
                      SplitList& sl, cudaStream_t st, unsigned long long* scratch_count);
void split_free(SplitList& sl);
// One damped-Jacobi sweep (FP32 or FP64) of a grain-map level: the tiled interior kernel, then the
// list.  *err is set (device) when a TMA load of the tiled kernel did not complete.  Inputs are the
// level's arrays; the result goes to any view over the storage box (split_out).
template <class R>
void launch_jacobi_split(const OpParams& P, const SplitList& sl, View<const R> C, View<const R> invD, View<const R> xi,
                         View<const R> b, View<R> xo, R omega, cudaStream_t st, Grains<R> G,
                         int ngrains, int* err);
// f = A x on the apply region of a grain-map level, the same split (f other than x, any view over the region).
template <class R>
void launch_fapply_split(const OpParams& P, const SplitList& sl, View<const R> C, View<const R> x, View<R> f,
                         cudaStream_t st, Grains<R> G, int ngrains, int* err);
// r = b - A x on the apply region of a grain-map level, the same split; r may alias b.
template <class R>
void launch_residual_split(const OpParams& P, const SplitList& sl, View<const R> C, View<const R> x, View<const R> b,
                           View<R> r, cudaStream_t st, Grains<R> G, int ngrains, int* err);

}  // namespace ae
