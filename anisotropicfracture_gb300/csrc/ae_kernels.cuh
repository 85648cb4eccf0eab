// Kernel templates of the nodal elastic operator.  Included by ae_kernels_f64.cu and
// ae_kernels_f32.cu, each of which instantiates the launchers for one precision.
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <stdexcept>
#include <string>
#include <type_traits>

#include "ae_device.cuh"
#include "ae_launch.h"

namespace ae {

#define AE_CUDA_CHECK(x)                                                                         \
    do {                                                                                         \
        cudaError_t e_ = (x);                                                                    \
        if (e_ != cudaSuccess)                                                                   \
            throw std::runtime_error(std::string("CUDA error: ") + cudaGetErrorString(e_) + " at " \
                                     + __FILE__ + ":" + std::to_string(__LINE__));               \
    } while (0)

constexpr int kBlock = 256;

// Flattened iteration over a box: thread t -> (i, j, k), i fastest.
struct Reg {
    int lo[3];
    unsigned nx, nxy;
    unsigned n;
};
inline Reg make_reg(const Box3& b) {
    Reg r;
    for (int d = 0; d < 3; ++d) r.lo[d] = b.lo[d];
    if (box_empty(b)) { r.nx = r.nxy = 1; r.n = 0; return r; }
    r.nx = (unsigned)(b.hi[0] - b.lo[0] + 1);
    r.nxy = r.nx * (unsigned)(b.hi[1] - b.lo[1] + 1);
    r.n = r.nxy * (unsigned)(b.hi[2] - b.lo[2] + 1);
    return r;
}
__device__ __forceinline__ void reg_ijk(const Reg& r, unsigned t, int& i, int& j, int& k) {
    const unsigned kk = t / r.nxy;
    const unsigned rem = t - kk * r.nxy;
    const unsigned jj = rem / r.nx;
    i = r.lo[0] + (int)(rem - jj * r.nx);
    j = r.lo[1] + (int)jj;
    k = r.lo[2] + (int)kk;
}
// A region as the part inside a box, and the slabs around that part.  Per-node sweeps run the slabs in a
// launch's first blocks (they take longer, and last they were its tail) and the inside in the rest: a warp
// that mixes a boundary row's one-sided gradient and stress with interior rows pays for both, and with rows of
// 65 nodes nearly every warp did (in FP64 about 70 operations on top of 100).  65^3 isotropic solve, all
// levels: Jacobi 28.6 -> 21.1 us a sweep, residual 27.8 -> 20.3; 97 x 81 x 113 cubic Jacobi 470 -> 407.  Slabs first:
// 129^3 cubic stress and energy 503 -> 489, set-up 1381 -> 1340, FP32 Fapply call 104.8 -> 102.0.  In FP32 the
// operations do not bound: 129^3 cubic Fapply 97.7 -> 94.9, but the coarse levels' Jacobi 25.7 -> 27.5 us, so
// that keeps all its nodes in one part; the residual and the 45-slot Fapply take the plain region (Region below):
// as Parts, 129^3 cubic residual 112.9 us, now 108.5, isotropic 59.4, now 56.9 (five blocks; of the compiler's
// own accord four, 68.0); 45 slots at 129^3 211 us and at 33^3 12.3, now 187 and 8.2.
struct Parts {
    Reg in;               // n == 0: none
    Reg slab[6];
    unsigned end[6];      // nodes of slabs 0 .. q
    unsigned out_blocks;  // blocks of the slabs, before those of the inside
};
inline Parts make_parts(const Box3& r, Box3 inside) {
    Parts P;
    inside = box_isect(inside, r);
    Box3 rest = r;
    Box3 s[6];
    for (Box3& b : s) {
        b = r;
        b.hi[0] = b.lo[0] - 1;  // empty
    }
    if (box_empty(inside)) {
        s[0] = r;
        inside = s[5];
    } else {
        for (int d = 2, q = 0; d >= 0; --d, q += 2) {
            s[q] = s[q + 1] = rest;
            s[q].hi[d] = inside.lo[d] - 1;
            s[q + 1].lo[d] = inside.hi[d] + 1;
            rest.lo[d] = inside.lo[d];
            rest.hi[d] = inside.hi[d];
        }
    }
    P.in = make_reg(inside);
    unsigned n = 0;
    for (int q = 0; q < 6; ++q) {
        P.slab[q] = make_reg(s[q]);
        n += P.slab[q].n;
        P.end[q] = n;
    }
    P.out_blocks = (P.end[5] + kBlock - 1) / kBlock;
    return P;
}
// the inside for the FP64 Jacobi sweep; empty in FP32
template <class R>
inline Box3 parts_inside(const Geo& g) {
    if (sizeof(R) == 8) return geo_interior(g);
    return Box3{{1, 1, 1}, {0, 0, 0}};
}
inline unsigned parts_blocks(const Parts& P) { return P.out_blocks + (P.in.n + kBlock - 1) / kBlock; }
// this thread's node; false: none.  The whole block is inside or outside.
__device__ __forceinline__ bool parts_ijk(const Parts& P, bool inside, int& i, int& j, int& k) {
    if (inside) {
        const unsigned t = (blockIdx.x - P.out_blocks) * blockDim.x + threadIdx.x;
        if (t >= P.in.n) return false;
        reg_ijk(P.in, t, i, j, k);
        return true;
    }
    unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= P.end[5]) return false;
    int q = 0;
    unsigned before = 0;
    while (t >= P.end[q]) before = P.end[q++];
    reg_ijk(P.slab[q], t - before, i, j, k);
    return true;
}
inline unsigned nblocks(unsigned n) { return (n + kBlock - 1) / kBlock; }

// What a sweep runs over: Parts (APART) or, where the interior is not taken apart, the plain region, whose
// kernels are shorter and take fewer registers.
template <bool APART>
using Region = std::conditional_t<APART, Parts, Reg>;
template <bool APART>
inline Region<APART> make_region(const Box3& r, const Geo& g) {
    if constexpr (APART) return make_parts(r, geo_interior(g));
    else return make_reg(r);
}
inline unsigned region_blocks(const Parts& P) { return parts_blocks(P); }
inline unsigned region_blocks(const Reg& r) { return nblocks(r.n); }
__device__ __forceinline__ bool region_inside(const Parts& P) { return blockIdx.x >= P.out_blocks; }
__device__ __forceinline__ bool region_inside(const Reg&) { return false; }
__device__ __forceinline__ bool region_ijk(const Parts& P, bool inside, int& i, int& j, int& k) {
    return parts_ijk(P, inside, i, j, k);
}
__device__ __forceinline__ bool region_ijk(const Reg& r, bool, int& i, int& j, int& k) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= r.n) return false;
    reg_ijk(r, t, i, j, k);
    return true;
}

// after every kernel launch: surface launch errors and count the launch
inline void launched() {
    AE_CUDA_CHECK(cudaGetLastError());
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

__device__ __forceinline__ bool in_box(const int lo[3], const int hi[3], int i, int j, int k) {
    return i >= lo[0] && i <= hi[0] && j >= lo[1] && j <= hi[1] && k >= lo[2] && k <= hi[2];
}

// warp + block max of a non-negative double, then one atomicMax on its bit pattern
__device__ __forceinline__ void block_max_atomic(double v, unsigned long long* out) {
    __shared__ double sm[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sm[w] = v;
    __syncthreads();
    if (w == 0) {
        v = (lane < (int)(blockDim.x >> 5)) ? sm[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0 && v > 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(v));
    }
}

// f = A u at one node: through the grain tables when the level has them (G.gid laid out like C),
// otherwise through the per-node stiffness C
// (GR: compiled for the grain tables, so each variant keeps its own register budget)
template <int M, class R, bool GR, bool IN>
__device__ __forceinline__ R apply_any(const OpParams& P, const SCoef<R>& K, const View<const R>& C,
                                          const Grains<R>& G, const View<const R>& u, int i, int j, int k, R v[3]) {
    if constexpr (GR)
        return apply_node_grains<M, R, IN>(P.g, K, P.bc, P.uniform, G.gid, C.at(i, j, k), C.sy, C.sz, G.tab, u.p, u.sc,
                                u.at(i, j, k), u.sy, u.sz, i, j, k, v);
    else
        return apply_node<M, R, true, IN>(P.g, K, P.bc, P.uniform, C.p, C.sc, C.at(i, j, k), C.sy, C.sz, u.p, u.sc, u.at(i, j, k),
                         u.sy, u.sz, i, j, k, v);
}

// The same with the node's offsets given: oc into C (and the grain ids), ou into u
template <int M, class R, bool GR, bool IN = false>
__device__ __forceinline__ R apply_at(const OpParams& P, const SCoef<R>& K, const View<const R>& C,
                                         const Grains<R>& G, const View<const R>& u, int i, int j, int k,
                                         long long oc, long long ou, R v[3]) {
    if constexpr (GR)
        return apply_node_grains<M, R, IN>(P.g, K, P.bc, P.uniform, G.gid, oc, C.sy, C.sz, G.tab, u.p, u.sc, ou, u.sy, u.sz, i,
                                j, k, v);
    else
        return apply_node<M, R, true, IN>(P.g, K, P.bc, P.uniform, C.p, C.sc, oc, C.sy, C.sz, u.p, u.sc, ou, u.sy, u.sz, i, j, k, v);
}

// true when two views index the same storage layout (same box origin and strides): the
// solver's level arrays all do, so one offset serves every array of a sweep
template <class A, class B>
inline bool same_layout(const View<A>& a, const View<B>& b) {
    return a.lo[0] == b.lo[0] && a.lo[1] == b.lo[1] && a.lo[2] == b.lo[2] && a.sy == b.sy && a.sz == b.sz &&
           a.sc == b.sc;
}

// Resident blocks per SM requested for the per-node sweeps.  The FP32 grain-map sweeps are
// bound by load latency: 5 blocks of 256 threads (48 registers) hide more of it than the 4
// (64 registers) the compiler picks by itself (257^3 Jacobi sweep 0.53 ms against 0.59 ms).
// 0: no request (the compiler's choice).
#ifndef AE_GRAIN_SWEEP_BLOCKS
#define AE_GRAIN_SWEEP_BLOCKS 5
#endif
#ifndef AE_PERNODE_SWEEP_BLOCKS
#define AE_PERNODE_SWEEP_BLOCKS 0
#endif
template <class R, bool GR, int M = MM>
constexpr int sweep_min_blocks() {
    // 45 slots in FP32: two blocks need 128 registers; without the request the compiler took 130 to 140 for
    // some variants, one block: 97^3 Jacobi sweep 147 us, residual 161, against 89.5 and 92.1
    if (M == MAJOR && sizeof(R) == 4) return 2;
    return sizeof(R) != 4 ? 0 : GR ? AE_GRAIN_SWEEP_BLOCKS : AE_PERNODE_SWEEP_BLOCKS;
}

// ------------------------------------------------------------------ Fapply
// (45 slots in FP32: one row and two requested blocks; 129^3 nodes 211 us with both rows, 198 with one row and
// the compiler's 102 registers, 187 with the 128 of two blocks)
template <int M, class R>
constexpr bool kFapplyApart = sizeof(R) == 8 || M != MAJOR;
template <int M, class R, bool GR>
__global__ void __launch_bounds__(kBlock, M == MAJOR && sizeof(R) == 4 ? 2 : 0)
    k_fapply(OpParams P, SCoef<R> K, Region<kFapplyApart<M, R>> region, View<const R> C, Grains<R> G, View<const R> u,
             View<R> f) {
    const bool inside = region_inside(region);
    int i, j, k;
    if (!region_ijk(region, inside, i, j, k)) return;
    R v[3];
    const R sc = inside ? apply_any<M, R, GR, true>(P, K, C, G, u, i, j, k, v)
                        : apply_any<M, R, GR, false>(P, K, C, G, u, i, j, k, v);
    const long long o = f.at(i, j, k);
#pragma unroll
    for (int n = 0; n < 3; ++n) f.p[o + n * f.sc] = mul_rn(sc, v[n]);
}

// ------------------------------------------------------------------ residual (+ norm, + FP32 copy)
template <class R>
constexpr bool kResidualApart = sizeof(R) == 8;
template <int M, class R, bool GR>
constexpr int residual_min_blocks() {
    return M == ISO && sizeof(R) == 4 && !GR ? 5 : sweep_min_blocks<R, GR, M>();
}
template <int M, class R, bool NORM, bool R32, bool GR, bool SAME>
__global__ void __launch_bounds__(kBlock, residual_min_blocks<M, R, GR>()) k_residual(OpParams P, SCoef<R> K, Region<kResidualApart<R>> region,
                                                                                 View<const R> C, Grains<R> G,
                                                                                 View<const R> x, View<const R> b,
                                                                                 View<R> r, unsigned long long* norm,
                                                                                 View<float> r32) {
    const bool inside = region_inside(region);
    double mx = 0.0;
    int i, j, k;
    if (region_ijk(region, inside, i, j, k)) {
        R v[3];
        // SAME: every view has the layout of x (checked by the launcher)
        const long long ox = x.at(i, j, k);
        const long long oc = SAME ? ox : C.at(i, j, k);
        const R sc = inside ? apply_at<M, R, GR, true>(P, K, C, G, x, i, j, k, oc, ox, v)
                            : apply_at<M, R, GR, false>(P, K, C, G, x, i, j, k, oc, ox, v);
        const long long ob = SAME ? ox : b.at(i, j, k), orr = SAME ? ox : r.at(i, j, k);
        const long long o32 = SAME ? ox : (R32 ? r32.at(i, j, k) : 0);
        const long long bsc = SAME ? x.sc : b.sc, rsc = SAME ? x.sc : r.sc, r32sc = SAME ? x.sc : r32.sc;
        const bool inv = in_box(P.g.vlo, P.g.vhi, i, j, k);
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            const R rv = row_residual(b.p[ob + n * bsc], sc, v[n]);
            r.p[orr + n * rsc] = rv;
            if (R32) r32.p[o32 + n * r32sc] = (float)rv;
            // a NaN residual reports an infinite norm (fmax alone would drop it)
            if (NORM && inv) mx = (rv != rv) ? (double)INFINITY : fmax(mx, (double)fabs(rv));
        }
    }
    if (NORM) block_max_atomic(mx, norm);
}

// ------------------------------------------------------------------ damped Jacobi sweep
// src/Operator/Operator.cpp:109-157 with the per-node Fapply fused in: one node (i, j, k).
// The damped-Jacobi update of one component from r = b - A x: x + w r / D, which is the reference's
// (1 - w) x + w (b - (A x - D x)) / D (Operator.cpp:154) without its D, in one fixed rounding order.
template <class R>
__device__ __forceinline__ R jacobi_update(R xv, R r, R invd, R omega) {
    return fma_rn(mul_rn(omega, r), invd, xv);
}

template <int M, class R, bool GR, bool SAME, bool IN = false>
__device__ __forceinline__ void jacobi_node(const OpParams& P, const SCoef<R>& K, const View<const R>& C,
                                            const Grains<R>& G, const View<const R>& invD,
                                            const View<const R>& xi, const View<const R>& b, const View<R>& xo,
                                            R omega, int i, int j, int k) {
    const Geo& g = P.g;
    // SAME: every view has the layout of xi (checked by the launcher)
    const long long ox = xi.at(i, j, k), oo = SAME ? ox : xo.at(i, j, k);
    const long long xsc = xi.sc, osc = SAME ? xsc : xo.sc;
    // outside the domain: untouched
    if (!IN && !in_box(g.dlo, g.dhi, i, j, k)) {
#pragma unroll
        for (int n = 0; n < 3; ++n) xo.p[oo + n * osc] = xi.p[ox + n * xsc];
        return;
    }
    // outermost ring of grow(valid, 2): zero
    if (!IN && g.ng >= 2 && (i == g.vlo[0] - 2 || i == g.vhi[0] + 2 || j == g.vlo[1] - 2 || j == g.vhi[1] + 2 ||
                             k == g.vlo[2] - 2 || k == g.vhi[2] + 2)) {
#pragma unroll
        for (int n = 0; n < 3; ++n) xo.p[oo + n * osc] = R(0);
        return;
    }
    R v[3];
    const R sc = apply_at<M, R, GR, IN>(P, K, C, G, xi, i, j, k, SAME ? ox : C.at(i, j, k), ox, v);
    const long long od = SAME ? ox : invD.at(i, j, k), ob = SAME ? ox : b.at(i, j, k);
    const long long isc = SAME ? xsc : invD.sc, bsc = SAME ? xsc : b.sc;
#pragma unroll
    for (int n = 0; n < 3; ++n)
        v[n] = jacobi_update<R>(xi.p[ox + n * xsc], row_residual(b.p[ob + n * bsc], sc, v[n]), invD.p[od + n * isc], omega);
#pragma unroll
    for (int n = 0; n < 3; ++n) xo.p[oo + n * osc] = v[n];
}

// The first sweep of a smoother call whose correction starts at zero (the pre-smoothing of a
// V-cycle level, a patch's mini-cycle): A 0 = 0 on every row, interior and boundary, so the
// sweep needs no stencil.  Every node gets what jacobi_node gives it for x = 0 and A x = 0,
// through the same update with the zeros passed in at run time (zero == 0), so the arithmetic
// and its rounding are the full sweep's.
template <class R>
__global__ void __launch_bounds__(kBlock) k_jacobi_zero(Geo g, Reg reg, View<const R> invD, View<const R> b,
                                                        View<R> xo, R omega, R zero) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    const long long oo = xo.at(i, j, k);
    const bool ring = g.ng >= 2 && (i == g.vlo[0] - 2 || i == g.vhi[0] + 2 || j == g.vlo[1] - 2 || j == g.vhi[1] + 2 ||
                                    k == g.vlo[2] - 2 || k == g.vhi[2] + 2);
    if (!in_box(g.dlo, g.dhi, i, j, k) || ring) {
#pragma unroll
        for (int n = 0; n < 3; ++n) xo.p[oo + n * xo.sc] = zero;
        return;
    }
    const long long od = invD.at(i, j, k), ob = b.at(i, j, k);
    R v[3];
#pragma unroll
    for (int n = 0; n < 3; ++n)
        v[n] = jacobi_update<R>(zero, row_residual(b.p[ob + n * b.sc], R(1), zero), invD.p[od + n * invD.sc], omega);
#pragma unroll
    for (int n = 0; n < 3; ++n) xo.p[oo + n * xo.sc] = v[n];
}

template <int M, class R, bool GR, bool SAME>
__global__ void __launch_bounds__(kBlock, sweep_min_blocks<R, GR, M>()) k_jacobi(OpParams P, SCoef<R> K, Parts parts,
                                                                               View<const R> C, Grains<R> G,
                                                                               View<const R> invD,
                                                                               View<const R> xi, View<const R> b,
                                                                               View<R> xo, R omega) {
    const bool inside = sizeof(R) == 8 && blockIdx.x >= parts.out_blocks;
    int i, j, k;
    if (!parts_ijk(parts, inside, i, j, k)) return;
    if (inside) jacobi_node<M, R, GR, SAME, true>(P, K, C, G, invD, xi, b, xo, omega, i, j, k);
    else jacobi_node<M, R, GR, SAME, false>(P, K, C, G, invD, xi, b, xo, omega, i, j, k);
}

// ------------------------------------------------------------------ z-marching tiled stencil sweeps
// A block owns a TX x TY column of nodes and marches KZ planes in z.  Displacement planes and
// stiffness planes sit in shared-memory rings with a one-node halo in x and y, filled by
// asynchronous global->shared copies (cp.async) one plane ahead of the plane being computed,
// so HBM streams while the block computes.  The stiffness slots the z column of the grad C
// term needs at k-1 are kept in registers.  Every array element is read from global memory
// once per block (plus the halo), all reads coalesced along i.  Domain-boundary nodes (a thin
// shell) take the per-node path.  The views must be the level's internal storage views (halo
// copies are guarded by the storage box).
enum SweepOp { OP_FAPPLY = 0, OP_JACOBI = 1, OP_RESIDUAL = 2 };
constexpr int TX = 32, TY = 8, KZ = 32;
constexpr int HX = TX + 2, HY = TY + 2, HP = HX * HY;
constexpr int NU_SLOTS = 4, NC_SLOTS = 3;  // displacement planes k-1..k+2, stiffness planes k..k+2

template <int M, class R>
constexpr size_t tiled_smem_bytes() {
    return sizeof(R) * (size_t)(NU_SLOTS * 3 + NC_SLOTS * NCoef<M>::value) * HP;
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem_dst, const void* gsrc) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gsrc), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

template <int M, class R, int OP>
__global__ void __launch_bounds__(TX* TY, 2) k_tiled(OpParams P, SCoef<R> K, Box3 box, View<const R> C,
                                                     View<const R> x, View<const R> b, View<const R> invD,
                                                     View<R> out, R omega) {
    constexpr int NC = NCoef<M>::value;
    constexpr int NZ = ZSlots<M>::n;
    constexpr int NT = TX * TY;
    static_assert(NT < HP && HP <= 2 * NT, "each thread stages two halo positions per plane");
    extern __shared__ __align__(16) unsigned char smraw[];
    R* su = reinterpret_cast<R*>(smraw);  // [NU_SLOTS][3 comps][HP]
    R* sC = su + NU_SLOTS * 3 * HP;        // [NC_SLOTS][NC][HP]
    const Geo& g = P.g;
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int i0 = box.lo[0] + blockIdx.x * TX, j0 = box.lo[1] + blockIdx.y * TY;
    const int kbeg = box.lo[2] + blockIdx.z * KZ;
    const int kend = min(kbeg + KZ, box.hi[2] + 1);
    const int i = i0 + tx, j = j0 + ty;
    const bool active = i <= box.hi[0] && j <= box.hi[1];
    int slo[3], shi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) { slo[d] = g.vlo[d] - g.ng; shi[d] = g.vhi[d] + g.ng; }

    // the two halo positions this thread stages in every plane, their in-plane offsets and validity
    const int r0 = threadIdx.x, r1 = threadIdx.x + NT;
    const bool has1 = r1 < HP;
    auto xy_of = [&](int r, long long& ou, long long& oc, bool& ok) {
        const int hy = r / HX, hx = r - hy * HX;
        const int gi = i0 - 1 + hx, gj = j0 - 1 + hy;
        ok = gi >= slo[0] && gi <= shi[0] && gj >= slo[1] && gj <= shi[1];
        ou = (long long)(gi - x.lo[0]) + (long long)(gj - x.lo[1]) * x.sy;
        oc = (long long)(gi - C.lo[0]) + (long long)(gj - C.lo[1]) * C.sy;
    };
    long long ou0, oc0, ou1 = 0, oc1 = 0;
    bool ok0, ok1 = false;
    xy_of(r0, ou0, oc0, ok0);
    if (has1) xy_of(r1, ou1, oc1, ok1);
    // asynchronous copy of plane kk of a field into a ring slot (zeros where the halo leaves storage)
    auto stage = [&](const View<const R>& v, long long o0, long long o1, int ncomp, int kk, R* dst) {
        const bool kok = kk >= slo[2] && kk <= shi[2];
        const R* base = v.p + (long long)(kk - v.lo[2]) * v.sz;
        for (int c = 0; c < ncomp; ++c) {
            const R* src = base + (long long)c * v.sc;
            if (kok && ok0) cp_async<sizeof(R)>(dst + c * HP + r0, src + o0);
            else dst[c * HP + r0] = R(0);
            if (has1) {
                if (kok && ok1) cp_async<sizeof(R)>(dst + c * HP + r1, src + o1);
                else dst[c * HP + r1] = R(0);
            }
        }
    };
    auto uslot = [&](int kk) { return su + ((kk - kbeg + 1) & 3) * 3 * HP; };
    auto cslot = [&](int kk) { return sC + ((kk - kbeg) % NC_SLOTS) * NC * HP; };

    // prologue: planes k-1..k+1 (displacement) and k, k+1 (stiffness); then the lookahead plane
    stage(x, ou0, ou1, 3, kbeg - 1, uslot(kbeg - 1));
    stage(x, ou0, ou1, 3, kbeg, uslot(kbeg));
    stage(x, ou0, ou1, 3, kbeg + 1, uslot(kbeg + 1));
    stage(C, oc0, oc1, NC, kbeg, cslot(kbeg));
    stage(C, oc0, oc1, NC, kbeg + 1, cslot(kbeg + 1));
    cp_async_commit();
    stage(x, ou0, ou1, 3, kbeg + 2, uslot(kbeg + 2));
    stage(C, oc0, oc1, NC, kbeg + 2, cslot(kbeg + 2));
    cp_async_commit();
    R Cm[NZ];
    const bool km_ok = active && kbeg - 1 >= slo[2];
#pragma unroll
    for (int s = 0; s < NZ; ++s)
        Cm[s] = km_ok ? __ldg(C.p + C.at(i, j, kbeg - 1) + ZSlots<M>::at(s) * C.sc) : R(0);
    cp_async_wait<1>();
    __syncthreads();

    const int idx = (ty + 1) * HX + (tx + 1);
    for (int k = kbeg; k < kend; ++k) {
        const R* Uc = uslot(k);
        const R* Um = uslot(k - 1);
        const R* Up = uslot(k + 1);
        const R* Cc = cslot(k);
        const R* Cn = cslot(k + 1);
        if (active) {
            const long long oo = out.at(i, j, k);
            bool done = false;
            if (OP == OP_JACOBI) {
                if (!in_box(g.dlo, g.dhi, i, j, k)) {
#pragma unroll
                    for (int n = 0; n < 3; ++n) out.p[oo + n * out.sc] = Uc[n * HP + idx];
                    done = true;
                } else if (g.ng >= 2 && (i == g.vlo[0] - 2 || i == g.vhi[0] + 2 || j == g.vlo[1] - 2 ||
                                         j == g.vhi[1] + 2 || k == g.vlo[2] - 2 || k == g.vhi[2] + 2)) {
#pragma unroll
                    for (int n = 0; n < 3; ++n) out.p[oo + n * out.sc] = R(0);
                    done = true;
                }
            }
            if (!done) {
                R f[3];
                const bool interior = i > g.dlo[0] && i < g.dhi[0] && j > g.dlo[1] && j < g.dhi[1] &&
                                      k > g.dlo[2] && k < g.dhi[2];
                if (!interior) {
                    apply_node<M, R>(g, K, P.bc, P.uniform, C.p, C.sc, C.at(i, j, k), C.sy, C.sz, x.p, x.sc,
                                     x.at(i, j, k), x.sy, x.sz, i, j, k, f);  // a boundary row: factor 1
                } else {
                    R gu[3][3], bb[3][3][3];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const R* u0 = Uc + p * HP + idx;
                        const R* um = Um + p * HP + idx;
                        const R* up = Up + p * HP + idx;
                        const R c0 = u0[0];
                        const R xm = u0[-1], xp = u0[1], ym = u0[-HX], yp = u0[HX], zm = um[0], zp = up[0];
                        gu[p][0] = (xp - xm) * K.h[0];
                        gu[p][1] = (yp - ym) * K.h[1];
                        gu[p][2] = (zp - zm) * K.h[2];
                        bb[p][0][0] = (xp - R(2) * c0 + xm) * K.i2[0];
                        bb[p][1][1] = (yp - R(2) * c0 + ym) * K.i2[1];
                        bb[p][2][2] = (zp - R(2) * c0 + zm) * K.i2[2];
                        bb[p][0][1] = (u0[1 + HX] + u0[-1 - HX] - u0[1 - HX] - u0[-1 + HX]) * K.m01;
                        bb[p][0][2] = (up[1] + um[-1] - um[1] - up[-1]) * K.m02;
                        bb[p][1][2] = (up[HX] + um[-HX] - um[HX] - up[-HX]) * K.m12;
                        bb[p][1][0] = bb[p][0][1];
                        bb[p][2][0] = bb[p][0][2];
                        bb[p][2][1] = bb[p][1][2];
                    }
                    R a[NC];
#pragma unroll
                    for (int q = 0; q < NC; ++q) a[q] = Cc[q * HP + idx];
                    div_of<M, R>(a, bb, f);
                    if (!P.uniform) {
                        R c0v[3], c1v[3], c2v[3];
                        gradC_col_f<M, R>([&](int q) { return Cc[q * HP + idx + 1] - Cc[q * HP + idx - 1]; }, gu, 0,
                                          c0v);
                        gradC_col_f<M, R>([&](int q) { return Cc[q * HP + idx + HX] - Cc[q * HP + idx - HX]; }, gu, 1,
                                          c1v);
                        gradC_col_f<M, R>([&](int q) { return Cn[q * HP + idx] - Cm[zslot_index<M>(q)]; }, gu, 2,
                                          c2v);
#pragma unroll
                        for (int r = 0; r < 3; ++r) f[r] = gradc_add(f[r], c0v[r], c1v[r], c2v[r], K.h);
                    }
                }
                if (OP == OP_FAPPLY) {
#pragma unroll
                    for (int n = 0; n < 3; ++n) out.p[oo + n * out.sc] = f[n];
                } else if (OP == OP_RESIDUAL) {
                    const long long ob = b.at(i, j, k);
#pragma unroll
                    for (int n = 0; n < 3; ++n) out.p[oo + n * out.sc] = b.p[ob + n * b.sc] - f[n];
                } else {
                    const long long ob = b.at(i, j, k), od = invD.at(i, j, k);
#pragma unroll
                    for (int n = 0; n < 3; ++n)
                        out.p[oo + n * out.sc] = jacobi_update<R>(Uc[n * HP + idx], b.p[ob + n * b.sc] - f[n],
                                                                  invD.p[od + n * invD.sc], omega);
                }
            }
        }
        // the stiffness of plane k becomes the k-1 plane of the next step
#pragma unroll
        for (int s = 0; s < NZ; ++s) Cm[s] = Cc[ZSlots<M>::at(s) * HP + idx];
        __syncthreads();  // every thread is done with the slots of planes k-1 (displacement) and k (stiffness)
        if (k + 1 < kend) {
            if (k + 3 <= kend) {  // the next lookahead plane reuses those slots
                stage(x, ou0, ou1, 3, k + 3, uslot(k + 3));
                stage(C, oc0, oc1, NC, k + 3, cslot(k + 3));
            }
            cp_async_commit();
            cp_async_wait<1>();  // plane k+2 has landed
            __syncthreads();
        }
    }
    cp_async_wait<0>();
}

// ------------------------------------------------------------------ Diagonal
// src/Operator/Elastic.cpp:285-350: the operator applied to a unit spike, component by component.  On
// interior rows the spike leaves three products a component (sum over d of C_pdpd (-2 / dx_d^2)); the
// zeros it meets the other slots with only matter when a slot is not finite, which is tested on its bits.
// 129^3 cubic nodes and the coarser levels, FP64:
// 1.58 -> 0.40 ms (0.08 at the HBM rate).
__device__ __forceinline__ bool finite_bits(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool finite_bits(float v) { return (__float_as_int(v) & 0x7f800000) != 0x7f800000; }
template <int M, class R>
__global__ void __launch_bounds__(kBlock) k_diagonal(OpParams P, SCoef<R> K, Parts parts, View<const R> C, View<R> D,
                                                     View<R> invD, int* nan_flag) {
    constexpr int NC = NCoef<M>::value;
    const bool inside = blockIdx.x >= parts.out_blocks;
    int i, j, k;
    if (!parts_ijk(parts, inside, i, j, k)) return;
    const Geo& g = P.g;
    const long long cc = C.at(i, j, k), od = D.at(i, j, k), oi = invD.at(i, j, k);
    R a[NC], val[3];
#pragma unroll
    for (int q = 0; q < NC; ++q) a[q] = C.p[cc + q * C.sc];
    if (inside) {
        bool ok = true;
#pragma unroll
        for (int q = 0; q < NC; ++q) ok = ok && finite_bits(a[q]);
        if constexpr (M == ISO) {
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                R bb[3][3][3], f[3];
#pragma unroll
                for (int q = 0; q < 3; ++q)
#pragma unroll
                    for (int l = 0; l < 3; ++l)
#pragma unroll
                        for (int jj = 0; jj < 3; ++jj) bb[q][l][jj] = (q == p && l == jj) ? K.bb[l] : R(0);
                div_of<M, R>(a, bb, f);
                val[p] = f[p];
            }
        } else {
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const auto c = [&](int d) { return a[M == DIAG ? 3 * p + d : slot_of<M == DIAG ? MM : M>(p, d, p, d)]; };
                val[p] = fx_sop(c(0), K.bb[0], c(1), K.bb[1], c(2), K.bb[2]);
            }
        }
        if (!ok) val[0] = val[1] = val[2] = R(NAN);
    } else {
        const int ci[3] = {i, j, k};
        bool mn[3], mx[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) { mn[d] = ci[d] == g.dlo[d]; mx[d] = ci[d] == g.dhi[d]; }
        R nrm[3];
        const int face = classify<R>(g, i, j, k, nrm);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            R gu[3][3], bb[3][3][3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const R hi = (mx[d] && p == q) ? R(1) : R(0);
                    const R lo = (mn[d] && p == q) ? R(1) : R(0);
                    gu[q][d] = (hi - lo) / ((mn[d] || mx[d] ? R(1) : R(2)) * (R)g.dx[d]);
                }
#pragma unroll
                for (int l = 0; l < 3; ++l)
#pragma unroll
                    for (int jj = 0; jj < 3; ++jj) bb[q][l][jj] = R(0);
#pragma unroll
                for (int d = 0; d < 3; ++d) bb[q][d][d] = (p == q) ? K.bb[d] : R(0);
            }
            if (face >= 0) {
                const unsigned char tp = P.bc.t[face][p];
                if (tp == DISP) val[p] = R(1);
                else if (tp == TRAC) {
                    R s[3][3];
                    stress_of<M, R>(a, gu, s);
                    val[p] = s[p][0] * nrm[0] + s[p][1] * nrm[1] + s[p][2] * nrm[2];
                } else if (tp == NEUMANN) val[p] = gu[p][0] * nrm[0] + gu[p][1] * nrm[1] + gu[p][2] * nrm[2];
                else val[p] = R(0);
            } else {
                R f[3];
                div_of<M, R>(a, bb, f);
                val[p] = f[p];  // the grad C term multiplies grad u = 0 at interior nodes
            }
        }
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        D.p[od + p * D.sc] = val[p];
        invD.p[oi + p * invD.sc] = R(1) / val[p];
        if (!(fabs((double)val[p]) <= 1.0e300) || val[p] == R(0)) atomicExch(nan_flag, 1);
    }
}

// ------------------------------------------------------------------ restriction / interpolation
// src/Operator/Operator.cpp:486-543 (coarse node I, fine node 2I).  A component per blockIdx.y, the
// coarse domain's interior and its boundary in separate blocks: with the components in a loop and both
// kinds of node in a warp the 21 slots of 129^3 -> 65^3 and the coarser levels took 0.82 ms, now 0.34 (the
// 30 FP64 operations a value need 0.30).
template <class R>
__global__ void __launch_bounds__(kBlock) k_restrict(Geo gc, Parts parts, View<R> crse, View<const R> fine) {
    const bool inside = blockIdx.x >= parts.out_blocks;
    int I, J, Kc;
    if (!parts_ijk(parts, inside, I, J, Kc)) return;
    const bool xe = !inside && (I == gc.dlo[0] || I == gc.dhi[0]);
    const bool ye = !inside && (J == gc.dlo[1] || J == gc.dhi[1]);
    const bool ze = !inside && (Kc == gc.dlo[2] || Kc == gc.dhi[2]);
    const long long sy = fine.sy, sz = fine.sz;
    {
        const int n = blockIdx.y;
        const R* f = fine.p + fine.at(2 * I, 2 * J, 2 * Kc) + n * fine.sc;
        R v;
        if (xe && ye && ze) v = f[0];
        else if (ye && ze) v = R(0.25) * f[-1] + R(0.5) * f[0] + R(0.25) * f[1];
        else if (ze && xe) v = R(0.25) * f[-sy] + R(0.5) * f[0] + R(0.25) * f[sy];
        else if (xe && ye) v = R(0.25) * f[-sz] + R(0.5) * f[0] + R(0.25) * f[sz];
        else if (xe)
            v = (f[-sy - sz] + R(2) * f[-sz] + f[sy - sz] + R(2) * f[-sy] + R(4) * f[0] + R(2) * f[sy] + f[-sy + sz] +
                 R(2) * f[sz] + f[sy + sz]) * R(1.0 / 16.0);
        else if (ye)
            v = (f[-1 - sz] + R(2) * f[-1] + f[-1 + sz] + R(2) * f[-sz] + R(4) * f[0] + R(2) * f[sz] + f[1 - sz] +
                 R(2) * f[1] + f[1 + sz]) * R(1.0 / 16.0);
        else if (ze)
            v = (f[-1 - sy] + R(2) * f[-sy] + f[1 - sy] + R(2) * f[-1] + R(4) * f[0] + R(2) * f[1] + f[-1 + sy] +
                 R(2) * f[sy] + f[1 + sy]) * R(1.0 / 16.0);
        else
            v = (f[-1 - sy - sz] + f[-1 - sy + sz] + f[-1 + sy - sz] + f[-1 + sy + sz] + f[1 - sy - sz] +
                 f[1 - sy + sz] + f[1 + sy - sz] + f[1 + sy + sz]) * R(1.0 / 64.0) +
                (f[-sy - sz] + f[-sy + sz] + f[sy - sz] + f[sy + sz] + f[-1 - sz] + f[1 - sz] + f[-1 + sz] +
                 f[1 + sz] + f[-1 - sy] + f[-1 + sy] + f[1 - sy] + f[1 + sy]) * R(1.0 / 32.0) +
                (f[-1] + f[-sy] + f[-sz] + f[1] + f[sy] + f[sz]) * R(1.0 / 16.0) + f[0] * R(1.0 / 8.0);
        crse.p[crse.at(I, J, Kc) + n * crse.sc] = v;
    }
}

// src/Operator/Operator.cpp:589-618 (fine node (i,j,k), coarse node (i/2, j/2, k/2)): the
// coarse field interpolated to fine node (i, j, k), component n, in the arithmetic type T
template <class T, class R>
__device__ __forceinline__ T interp_at(const View<const R>& crse, int i, int j, int k, int n) {
    const int I = i >> 1, J = j >> 1, Kc = k >> 1;  // non-negative indices
    const bool ie = !(i & 1), je = !(j & 1), ke = !(k & 1);
    const long long sy = crse.sy, sz = crse.sz;
    const R* c = crse.p + crse.at(I, J, Kc) + n * crse.sc;
    const auto C = [&](long long o) { return (T)c[o]; };
    if (ie && je && ke) return C(0);
    if (je && ke) return T(0.5) * (C(0) + C(1));
    if (ke && ie) return T(0.5) * (C(0) + C(sy));
    if (ie && je) return T(0.5) * (C(0) + C(sz));
    if (ie) return T(0.25) * (C(0) + C(sy) + C(sz) + C(sy + sz));
    if (je) return T(0.25) * (C(0) + C(sz) + C(1) + C(1 + sz));
    if (ke) return T(0.25) * (C(0) + C(1) + C(sy) + C(1 + sy));
    return T(0.125) * (C(0) + C(1) + C(sy) + C(sz) + C(sy + sz) + C(1 + sz) + C(1 + sy) + C(1 + sy + sz));
}

// Interpolation added into the fine level (the same weights), one thread per coarse node
// (I, J, K) of the coarse box cb: it adds into the up to 8 fine nodes (2I + a, 2J + b, 2K + c),
// a, b, c in {0, 1}, that lie in the fine region fr.  The parity of each of those nodes is known
// at compile time, so a warp runs no divergent branches and the coarse values are loaded once
// for the 8 nodes.  Each node's value is the expression of interp_at for its parity.
// Bound by the fine level's traffic: all 16 values are loaded before any is stored, a component per
// blockIdx.y.  FP32 F-cycles of 257^3 nodes, all levels: 57 -> 26 us a call.
template <class T>
struct alignas(2 * sizeof(T)) Vec2 {
    T v[2];
};
template <class R, bool VEC>
__global__ void __launch_bounds__(kBlock) k_interp_add8(Reg cb, Box3 fr, View<R> fine, View<const R> crse) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= cb.n) return;
    int I, J, Kc;
    reg_ijk(cb, t, I, J, Kc);
    const long long sy = crse.sy, sz = crse.sz;
    const bool x1 = 2 * I + 1 <= fr.hi[0], y1 = 2 * J + 1 <= fr.hi[1], z1 = 2 * Kc + 1 <= fr.hi[2];
    const bool x0 = 2 * I >= fr.lo[0], y0 = 2 * J >= fr.lo[1], z0 = 2 * Kc >= fr.lo[2];
    const int n = blockIdx.y;
    const R* __restrict__ c = crse.p + crse.at(I, J, Kc) + n * crse.sc;
    R* __restrict__ f = fine.p + fine.at(2 * I, 2 * J, 2 * Kc) + n * fine.sc;
    // coarse corner and fine node (a, b, c), when that fine node is in the region (a corner is one of a
    // node that needs it); VEC: the fine pair along x is one aligned access when both are
    R cv[8], fv[8];
    const bool pair = VEC && x0 && x1;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int a = q & 1, bq = (q >> 1) & 1, d = q >> 2;
        const bool need = (!a || x1) && (!bq || y1) && (!d || z1);
        cv[q] = need ? c[a + bq * sy + d * sz] : R(0);
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const int bq = h & 1, d = h >> 1;
        const bool row = (bq ? y1 : y0) && (d ? z1 : z0);
        R* fr_ = f + bq * fine.sy + d * fine.sz;
        fv[2 * h] = fv[2 * h + 1] = R(0);
        if (row) {
            if (pair) {
                const Vec2<R> w = *reinterpret_cast<const Vec2<R>*>(fr_);
                fv[2 * h] = w.v[0];
                fv[2 * h + 1] = w.v[1];
            } else {
                if (x0) fv[2 * h] = fr_[0];
                if (x1) fv[2 * h + 1] = fr_[1];
            }
        }
    }
    fv[0] += cv[0];
    fv[1] += R(0.5) * (cv[0] + cv[1]);
    fv[2] += R(0.5) * (cv[0] + cv[2]);
    fv[4] += R(0.5) * (cv[0] + cv[4]);
    fv[6] += R(0.25) * (cv[0] + cv[2] + cv[4] + cv[6]);
    fv[5] += R(0.25) * (cv[0] + cv[4] + cv[1] + cv[5]);
    fv[3] += R(0.25) * (cv[0] + cv[1] + cv[2] + cv[3]);
    fv[7] += R(0.125) * (cv[0] + cv[1] + cv[2] + cv[4] + cv[6] + cv[5] + cv[3] + cv[7]);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const int bq = h & 1, d = h >> 1;
        const bool row = (bq ? y1 : y0) && (d ? z1 : z0);
        R* fr_ = f + bq * fine.sy + d * fine.sz;
        if (row) {
            if (pair) {
                Vec2<R> w;
                w.v[0] = fv[2 * h];
                w.v[1] = fv[2 * h + 1];
                *reinterpret_cast<Vec2<R>*>(fr_) = w;
            } else {
                if (x0) fr_[0] = fv[2 * h];
                if (x1) fr_[1] = fv[2 * h + 1];
            }
        }
    }
}

// nodal average_down (src/Operator/Operator.cpp:631): coarse node I takes fine node 2I
template <class R>
__global__ void __launch_bounds__(kBlock) k_inject(Reg reg, int ncomp, View<R> crse, View<const R> fine) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int I, J, Kc;
    reg_ijk(reg, t, I, J, Kc);
    const long long oc = crse.at(I, J, Kc), of = fine.at(2 * I, 2 * J, 2 * Kc);
    for (int n = 0; n < ncomp; ++n) crse.p[oc + n * crse.sc] = fine.p[of + n * fine.sc];
}

// ------------------------------------------------------------------ elementwise
// Copies and updates are bound by bytes in flight: a thread takes U nodes and loads them all before it
// stores any (the compiler may not, since the views could overlap).  193 x 161 x 225 nodes of three
// FP32 components between a field and a level array: 55 -> 31 us.
template <class Ro, class Ri, int U>
__global__ void __launch_bounds__(kBlock) k_copy(Reg reg, int ncomp, View<Ro> dst, View<const Ri> src) {
    const unsigned t0 = blockIdx.x * (blockDim.x * U) + threadIdx.x;
    long long od[U], os[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
        const unsigned t = t0 + q * blockDim.x;
        if (t >= reg.n) break;
        int i, j, k;
        reg_ijk(reg, t, i, j, k);
        od[q] = dst.at(i, j, k);
        os[q] = src.at(i, j, k);
    }
    int n = 0;
    for (; n + 3 <= ncomp; n += 3) {
        Ri v[U][3];
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (t0 + q * blockDim.x < reg.n)
#pragma unroll
                for (int c = 0; c < 3; ++c) v[q][c] = src.p[os[q] + (n + c) * src.sc];
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (t0 + q * blockDim.x < reg.n)
#pragma unroll
                for (int c = 0; c < 3; ++c) dst.p[od[q] + (n + c) * dst.sc] = (Ro)v[q][c];
    }
    for (; n < ncomp; ++n)
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (t0 + q * blockDim.x < reg.n) dst.p[od[q] + n * dst.sc] = (Ro)src.p[os[q] + n * src.sc];
}
// nodes a thread of k_copy takes: four once that still gives every SM of 152 its eight blocks
template <class F>
inline void dispatch_copy(unsigned n, F&& f) {
    if (n >= 152u * 8u * kBlock * 4u) f(std::integral_constant<int, 4>());
    else f(std::integral_constant<int, 1>());
}
template <class Ro, class Ri>
__global__ void __launch_bounds__(kBlock) k_axpy(Reg reg, int ncomp, View<Ro> dst, double alpha, View<const Ri> src) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    const long long od = dst.at(i, j, k), os = src.at(i, j, k);
    for (int n = 0; n < ncomp; ++n) dst.p[od + n * dst.sc] += (Ro)(alpha * (double)src.p[os + n * src.sc]);
}
template <class R>
__global__ void __launch_bounds__(kBlock) k_fill(Reg reg, int ncomp, View<R> dst, R value) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    const long long od = dst.at(i, j, k);
    for (int n = 0; n < ncomp; ++n) dst.p[od + n * dst.sc] = value;
}
// Flat forms of copy / fill / axpy for a region that is the whole storage of its views (the
// common case: level-wide vectors): the components are one contiguous run of n values, so a
// grid-stride loop streams it with no index arithmetic.  ADD: alpha == 1, where the general form
// dst + (Ro)(1.0 * (double)src) is exactly dst + (Ro)src (no FP64 multiply).
// Four elements a thread and turn, as 16-byte accesses (the launcher checks that both runs begin on a
// 16-byte boundary; the remainder of the run, or a run that does not, goes element by element).
template <class T>
struct alignas(16) Vec4 {
    T v[4];
};
template <class Ro, class Ri>
__global__ void __launch_bounds__(kBlock) k_flat_copy(long long n, bool vec, Ro* __restrict__ dst, const Ri* __restrict__ src) {
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
    const long long n4 = vec ? n / 4 : 0;
    for (long long t = t0; t < n4; t += nt) {
        const Vec4<Ri> s = reinterpret_cast<const Vec4<Ri>*>(src)[t];
        Vec4<Ro> d;
#pragma unroll
        for (int q = 0; q < 4; ++q) d.v[q] = (Ro)s.v[q];
        reinterpret_cast<Vec4<Ro>*>(dst)[t] = d;
    }
    for (long long t = 4 * n4 + t0; t < n; t += nt) dst[t] = (Ro)src[t];
}
template <class R>
__global__ void __launch_bounds__(kBlock) k_flat_fill(long long n, R* __restrict__ dst, R value) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        dst[t] = value;
}
template <class Ro, class Ri, bool ADD>
__global__ void __launch_bounds__(kBlock) k_flat_axpy(long long n, bool vec, Ro* __restrict__ dst, double alpha,
                                                      const Ri* __restrict__ src) {
    const auto sum = [&](Ro d, Ri s) { return d + (ADD ? (Ro)s : (Ro)(alpha * (double)s)); };
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
    const long long n4 = vec ? n / 4 : 0;
    for (long long t = t0; t < n4; t += nt) {
        const Vec4<Ri> s = reinterpret_cast<const Vec4<Ri>*>(src)[t];
        Vec4<Ro> d = reinterpret_cast<const Vec4<Ro>*>(dst)[t];
#pragma unroll
        for (int q = 0; q < 4; ++q) d.v[q] = sum(d.v[q], s.v[q]);
        reinterpret_cast<Vec4<Ro>*>(dst)[t] = d;
    }
    for (long long t = 4 * n4 + t0; t < n; t += nt) dst[t] = sum(dst[t], src[t]);
}
inline bool vec4_aligned(const void* a, const void* b) { return (((uintptr_t)a | (uintptr_t)b) & 15) == 0; }
// true when region, taken over ncomp components, covers whole rows and planes of v's storage
// from its first node, so that the elements from there on form one contiguous run (row padding
// included: padding is never read by the stencil kernels, and the level arrays hold it)
template <class T>
inline bool flat_view(const Reg& reg, int ncomp, const View<T>& v) {
    const long long w = v.wx > 0 ? v.wx : v.sy;
    const long long ny = reg.nxy / reg.nx, nz = reg.n / reg.nxy;
    return reg.n > 0 && reg.lo[0] == v.lo[0] && reg.lo[1] == v.lo[1] && reg.lo[2] == v.lo[2] &&
           (long long)reg.nx == w && ny * v.sy == v.sz && (ncomp == 1 || nz * v.sz == v.sc);
}
// elements of that contiguous run
template <class T>
inline long long flat_count(const Reg& reg, int ncomp, const View<T>& v) {
    const long long nz = reg.n / reg.nxy;
    return ncomp == 1 ? nz * v.sz : v.sc * ncomp;
}
// the same run in two views: same pitches
template <class A, class B>
inline bool same_pitch(const View<A>& a, const View<B>& b) {
    return a.sy == b.sy && a.sz == b.sz && a.sc == b.sc;
}
// grid of a flat loop: enough blocks to cover n, capped at 8 resident blocks per SM of 152
inline unsigned flat_blocks(long long n) {
    const long long b = (n + kBlock - 1) / kBlock;
    return (unsigned)(b < 152 * 8 ? b : 152 * 8);
}

// max-norm of a region: grid-stride over the nodes with a capped grid (kNormBlocks), so that a
// few thousand blocks, not one per 256 nodes, end in a barrier and an atomic
constexpr unsigned kNormBlocks = 152 * 8;
template <class R>
__global__ void __launch_bounds__(kBlock) k_norminf(Reg reg, int ncomp, View<const R> v, unsigned long long* out) {
    double mx = 0.0;
    for (unsigned long long t = blockIdx.x * blockDim.x + threadIdx.x; t < reg.n; t += gridDim.x * blockDim.x) {
        int i, j, k;
        reg_ijk(reg, (unsigned)t, i, j, k);
        const long long o = v.at(i, j, k);
        for (int n = 0; n < ncomp; ++n) {
            const R a = v.p[o + n * v.sc];
            mx = (a != a) ? (double)INFINITY : fmax(mx, (double)fabs(a));
        }
    }
    block_max_atomic(mx, out);
}

// ------------------------------------------------------------------ launcher bodies
template <class R, class F>
inline void dispatch_model(int model, F&& f) {
    if (model == ISO) f(std::integral_constant<int, ISO>());
    else if (model == MM) f(std::integral_constant<int, MM>());
    else f(std::integral_constant<int, DIAG>());
}
// the box operator's kinds: the three above and the 45-slot Sym::Major tangent of a
// finite-kinematics model
template <class R, class F>
inline void dispatch_model4(int model, F&& f) {
    if (model == MAJOR) f(std::integral_constant<int, MAJOR>());
    else dispatch_model<R>(model, f);
}

}  // namespace ae
