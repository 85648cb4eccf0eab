// Split sweeps on Voronoi (grain-map) levels, FP32 and FP64.
//
// On a grain-map level the per-node sweep spends most of its issue slots on work that few nodes
// need -- the domain-boundary classification, six neighbour grain ids, the grad C branch that
// only the nodes whose stencil straddles a grain boundary take -- and waits on scattered loads.
// A sweep there is split by node:
//
//   k_sweep_tile64/32  every node of the interior box I (not on the domain boundary, inside
//                  grow(valid, 1)).  A block owns a 32 x 8 column of (i, j) and marches in k, its
//                  planes of x, b, 1/D and the ids loaded by TMA (cp.async.bulk.tensor) ahead of
//                  the plane being computed, the grain tables in shared memory.  The grad C term
//                  is computed only where the node's mask says a direction's two neighbours lie in
//                  different grains.
//   k_*_list       every node of the sweep region outside I (domain-boundary rows, the ghost
//                  ring, nodes outside the domain), through the per-node code.
//
// Three operations are split this way: the damped-Jacobi smoother, the residual r = b - A x and
// Fapply.
//
// Every node is computed by the per-node sweep's own arithmetic: where a direction's neighbours
// share a grain the grad C column is exactly zero, and the interior and grad C expressions are
// those of ae_device.cuh in their explicitly rounded order, so the split sweep equals the one-pass
// sweep bit for bit.  The list and the id/mask array are built once per level (k_split_mark), when the
// operator is prepared.  TMA needs 16-byte aligned rows: the level arrays' row pitch is a
// multiple of 4 nodes (Geo::px).
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <atomic>
#include <mutex>
#include <type_traits>

#include "ae_kernels.cuh"
#include "ae_split.h"

namespace ae {

namespace {

constexpr int STX = 32, STY = 8;   // nodes of a tile per plane: a warp per row
constexpr int SXR = STY + 2;       // x tile rows (one-node halo in j)
constexpr int kWaitLimit = 1 << 20;  // try_wait polls before a wait is declared failed
constexpr int kTileThreads = 32 * (STY + 1);  // the rows' warps and a producer
#ifndef AE_RING
#define AE_RING 4
#endif
constexpr int SRING = AE_RING;     // planes in flight or in use
__host__ __device__ constexpr int up128(int b) { return (b + 127) / 128 * 128; }

// Nodes with a grad C column are put off: a warp keeps what the column needs -- the in-plane
// differences, the two neighbours in k, the interior sum and the node's offset -- in a queue of its own
// and computes 32 of them at a time, because a warp-wide FP64 instruction costs the same whatever lanes
// are active.
constexpr int QCAP = 64;  // entries per warp: at most 31 left over and 32 new ones
constexpr int QN = 15;    // numbers per entry

// Shared memory of the tiled kernel, in bytes, for elements R: per ring slot the x halo tile, the b and
// 1/D tiles and the ids (TMA destinations on a 128-byte boundary); then the barriers, the warps' queues
// (FP64) and the grain tables.
template <class R>
struct TL {
    static constexpr int E = (int)sizeof(R);
    static constexpr int AL = 16 / E;              // columns per 16 bytes: TMA boxes start on such a column
    static constexpr int BW = STX + 2 * AL;        // x box width: the tile and AL columns to each side
    static constexpr int XP = BW * SXR;            // elements per x component plane tile
    static constexpr int VP = STX * STY;           // elements per b / 1/D / id component plane tile
    static constexpr int oB = up128(3 * XP * E);
    static constexpr int oI = oB + 3 * VP * E;
    static constexpr int oG = oI + 3 * VP * E;
    static constexpr int kSlot = oG + VP * 4;
    static constexpr int oBar = SRING * kSlot;
    static constexpr int oQ = up128(oBar + 16 * SRING + 8);  // the ring's barriers and the table's
    static constexpr int kQ = QCAP * (QN * E + 8);  // bytes per warp queue
    static constexpr int oT = up128(oQ + STY * kQ);
    static constexpr unsigned kX = 3 * XP * E, kV = 3 * VP * E, kG = VP * 4;
    static_assert(oB % 128 == 0 && oI % 128 == 0 && oG % 128 == 0 && kSlot % 128 == 0, "TMA destinations");
};
// bytes of grain tables kept in shared memory: the rows' numbers up to kRowSmemMax, and the stiffness
// table beside them up to kTabSmemMax in all (three FP32 blocks an SM up to 110 cubic grains)
constexpr int kRowSmemMax = 40 * 1024, kTabSmemMax = 44 * 1024;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait for a phase of the barrier: false when it did not complete within kWaitLimit polls
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
    for (int it = 0; it < kWaitLimit; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// 4-D tiled TMA load (x, y, z, component) into shared memory, completing on an mbarrier
__device__ __forceinline__ void tma_load4(unsigned dst, const CUtensorMap* map, int x, int y, int z, int c,
                                          unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];\n" ::"r"(dst),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(c), "r"(bar)
        : "memory");
}

// global -> shared memory, addresses and size multiples of 16 bytes, completing on an mbarrier
__device__ __forceinline__ void bulk_copy(unsigned dst, const void* src, int bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// packed node of a list: offsets from the storage box's low corner, 21 bits each
__device__ __forceinline__ unsigned long long pack_node(int di, int dj, int dk) {
    return (unsigned long long)di | ((unsigned long long)dj << 21) | ((unsigned long long)dk << 42);
}
__device__ __forceinline__ void unpack_node(unsigned long long c, const int lo[3], int& i, int& j, int& k) {
    i = lo[0] + (int)(c & 0x1fffffull);
    j = lo[1] + (int)((c >> 21) & 0x1fffffull);
    k = lo[2] + (int)((c >> 42) & 0x1fffffull);
}

// Mark the nodes of region R (inside the storage box) outside the interior box I, which a list
// kernel computes, and compact them (FILL = false: count only; order within a block follows the
// node order).  With FILL and gidm, also write gidm = gid | mask << 16 for every stored node, mask
// bit d set (nodes of I only) when the two neighbours in direction d lie in different grains: a
// non-zero grad C column.
template <bool FILL>
__global__ void __launch_bounds__(kBlock) k_split_mark(Reg reg, Box3 R, Box3 I, View<const unsigned short> gid,
                                                       unsigned* gidm, unsigned long long* list,
                                                       unsigned long long* count) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    bool f = false;
    unsigned long long code = 0;
    if (t < reg.n) {
        int i, j, k;
        reg_ijk(reg, t, i, j, k);
        const long long o = gid.at(i, j, k);
        if (!in_box(I.lo, I.hi, i, j, k)) {
            f = in_box(R.lo, R.hi, i, j, k);
            if (FILL && gidm) gidm[o] = gid.p[o];
        } else if (FILL && gidm) {
            const long long off[3] = {1, gid.sy, gid.sz};
            unsigned mask = 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) mask |= (gid.p[o + off[d]] != gid.p[o - off[d]]) ? (1u << d) : 0u;
            gidm[o] = (unsigned)gid.p[o] | (mask << 16);
        }
        code = pack_node(i - reg.lo[0], j - reg.lo[1], k - reg.lo[2]);
    }
    __shared__ unsigned wcnt[kBlock / 32];
    __shared__ unsigned long long base;
    const unsigned ball = __ballot_sync(0xffffffffu, f);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) wcnt[w] = __popc(ball);
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned tot = 0;
        for (int q = 0; q < kBlock / 32; ++q) {
            const unsigned c = wcnt[q];
            wcnt[q] = tot;
            tot += c;
        }
        base = tot ? atomicAdd(count, (unsigned long long)tot) : 0ull;
    }
    __syncthreads();
    if (FILL && f) list[base + wcnt[w] + __popc(ball & ((1u << lane) - 1u))] = code;
}

// Row numbers of every grain (RowN), in rows of whole pairs: what row_sum takes for a node of the grain.
template <int M>
__host__ __device__ constexpr int row_stride() { return (RowN<M>::value + 1) / 2 * 2; }
template <int M>
__global__ void __launch_bounds__(kBlock) k_row_table(const double* __restrict__ tab, int ngr, double* __restrict__ rows) {
    constexpr int NC = NCoef<M>::value, NR = RowN<M>::value;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ngr) return;
#pragma unroll
    for (int n = 0; n < NR; ++n) {
        rows[(long long)g * row_stride<M>() + n] = row_number<M>([&](int q) { return __ldg(tab + (long long)g * NC + q); }, n);
    }
}

// Tile geometry shared by the host and the kernel: tensor coordinates are offsets from the
// storage box's low corner.  Tiles start on columns that are multiples of 32 there, so a warp's rows
// of b, 1/D, the ids and the output are aligned; the x box starts AL columns before.
struct TileGeo {
    Box3 I;        // interior box (absolute node indices)
    int slo[3];    // storage box low corner
    int tiles_x;   // tiles per row of the storage box
    int kz;        // planes per block
};

// One sweep over the interior box I of a grain-map level, A the interior row of
// Elastic<T>::Fapply: OP = SPLIT_JACOBI, the damped-Jacobi update (Operator.cpp:109-157);
// OP = SPLIT_RESIDUAL, out = b - A x (out may alias b: every node reads only its own b);
// OP = SPLIT_FAPPLY, out = A x.
//
// A block owns a 32 x 8 column of (i, j) and marches in k.  One producer warp keeps up to SRING planes
// in flight by TMA (cp.async.bulk.tensor onto a full barrier per slot): the x halo tile (three
// components) of a plane and the b, 1/D and id tiles of the plane before, which is the one that becomes
// computable.  The other warps hold a row (FP32: two rows) each.  An x plane is read from shared memory
// once: each node takes from it the centre value, the two in-plane central differences and the three
// in-plane second differences; the differences across planes come from those of the planes before, in
// registers (9 values a component).  Warps run up to a ring apart, and no block barrier is in the loop.
//
// The row's numbers sit in shared memory per grain (TABS: the table of k_row_table, one bulk copy) or are
// formed from the slots in global memory.  err: set when
// a wait ran out.
//
// Bound by the FP64 pipe (89 % busy): 99 operations a node on a cubic level and about 6 for the queue.
// Fapply at 257^3 3.45 ms, with the boundary list 3.52, against 4.34 and 4.42 with the scaled rows (154
// operations) and a queue per plane that one warp worked off behind two block barriers; residual 3.52
// against 4.54, Jacobi 3.73 against 4.98.  A queue per block instead of per warp: 3.66.
enum SplitOp { SPLIT_JACOBI = 0, SPLIT_RESIDUAL = 1, SPLIT_FAPPLY = 2 };
// what a thread keeps of a plane, per component: centre, in-plane central differences
template <class R>
struct PlaneRegs {
    R c[3], dx[3], dy[3];
};
template <int M, bool TABS, int OP>
__global__ void __launch_bounds__(kTileThreads, 1)
    k_sweep_tile64(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_b,
                 const __grid_constant__ CUtensorMap tm_i, const __grid_constant__ CUtensorMap tm_g, SCoef<double> K, TileGeo T,
                 int uniform, int sy, int sz, long long sc, const unsigned* __restrict__ gidm,
                 const double* __restrict__ tab, const double* __restrict__ rows, int rows_bytes, int tab_bytes,
                 const double* __restrict__ x, const double* b, const double* __restrict__ invD, double* out, int osy, int osz,
                 long long osc, double omega, int* err) {
    using R = double;
    using L = TL<R>;
    constexpr int NC = NCoef<M>::value, TS = row_stride<M>();
    extern __shared__ __align__(128) unsigned char smem[];
    const unsigned sb = smem_u32(smem);
    const auto full = [&](int s) { return sb + (unsigned)L::oBar + 16u * (unsigned)s; };
    const auto empty = [&](int s) { return sb + (unsigned)L::oBar + 16u * (unsigned)s + 8u; };
    const R* ts = reinterpret_cast<const R*>(smem + L::oT);
    const unsigned tbar = sb + (unsigned)L::oBar + 16u * SRING;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = (int)(blockIdx.x % T.tiles_x) * STX;  // the tile's first column, from slo
    const int j0 = T.I.lo[1] + (int)(blockIdx.x / T.tiles_x) * STY;
    const int k0 = T.I.lo[2] + (int)blockIdx.y * T.kz;
    const int k1 = min(k0 + T.kz - 1, T.I.hi[2]);
    if (threadIdx.x == 0) {
        for (int s = 0; s < SRING; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), STY);
        }
        mbar_init(tbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    const int planes = k1 - k0 + 3;  // x planes k0 - 1 .. k1 + 1; with plane k0 - 1 + t come the tiles of plane k0 - 2 + t
    if (warp == STY) {               // producer
        if (lane == 0) {
            int t = 0;
            bool ok = true;
            if (TABS) {
                mbar_expect_tx(tbar, (unsigned)(rows_bytes + tab_bytes));
                bulk_copy(sb + (unsigned)L::oT, rows, rows_bytes, tbar);
                if (tab_bytes) bulk_copy(sb + (unsigned)(L::oT + rows_bytes), tab, tab_bytes, tbar);
            }
            for (; t < planes; ++t) {
                const int s = t % SRING;
                if (t >= SRING && !mbar_wait(empty(s), (unsigned)((t / SRING - 1) & 1))) {
                    ok = false;
                    break;
                }
                constexpr unsigned kTiles = (OP == SPLIT_JACOBI ? 2 : OP == SPLIT_RESIDUAL ? 1 : 0) * L::kV + L::kG;
                const unsigned dst = sb + (unsigned)(s * L::kSlot);
                const int y = j0 - T.slo[1], z = k0 - 1 + t - T.slo[2];
                mbar_expect_tx(full(s), L::kX + (t >= 2 ? kTiles : 0u));
                tma_load4(dst, &tm_x, c0 - L::AL, y - 1, z, 0, full(s));
                if (t >= 2) {
                    tma_load4(dst + L::oG, &tm_g, c0, y, z - 1, 0, full(s));
                    if (OP != SPLIT_FAPPLY) tma_load4(dst + L::oB, &tm_b, c0, y, z - 1, 0, full(s));
                    if (OP == SPLIT_JACOBI) tma_load4(dst + L::oI, &tm_i, c0, y, z - 1, 0, full(s));
                }
            }
            if (!ok) atomicExch(err, 1);
            // let the loads in flight land (bounded) before the block's memory goes
            for (int q = max(t - SRING, 0); q < t; ++q) mbar_wait(full(q % SRING), (unsigned)((q / SRING) & 1));
            if (TABS) mbar_wait(tbar, 0);
        }
        return;
    }
    const int i = T.slo[0] + c0 + lane, j = j0 + warp;
    const bool act = i >= T.I.lo[0] && i <= T.I.hi[0] && j <= T.I.hi[1];
    int o = c0 + lane + (j - T.slo[1]) * sy + (k0 - T.slo[2] - 2) * sz;  // node (i, j) of the plane computed
    int oo = c0 + lane + (j - T.slo[1]) * osy + (k0 - T.slo[2] - 2) * osz;  // ... in the output
    // the grains' stiffness: beside the rows in shared memory, or global
    const R* gt = TABS && tab_bytes ? reinterpret_cast<const R*>(smem + L::oT + rows_bytes) : tab;
    // F plus the grad C term of a node at offset on: gu its central differences, gp and gm the grains of
    // its neighbours, mask the directions
    const auto with_gradc = [&](unsigned mask, const unsigned (&gp)[3], const unsigned (&gm)[3], R (&gu)[3][3], R (&F)[3]) {
        grad_scale(K, gu);
        R col[3][3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (mask & (1u << d)) {
                const R* cp = gt + (int)(gp[d] & 0xffffu) * NC;
                const R* cm = gt + (int)(gm[d] & 0xffffu) * NC;
                gradC_col_f<M, R>([&](int q) { return cp[q] - cm[q]; }, gu, d, col[d]);
            } else {
                col[d][0] = col[d][1] = col[d][2] = R(0);
            }
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) F[r] = row_gradc(K, F[r], col[0][r], col[1][r], col[2][r]);
    };
    const auto value = [&](R xc, R bc, R ic, R F) {
        if (OP == SPLIT_JACOBI) return jacobi_update<R>(xc, row_residual(bc, K.i2[0], F), ic, omega);
        if (OP == SPLIT_RESIDUAL) return row_residual(bc, K.i2[0], F);
        return mul_rn(K.i2[0], F);
    };
    R* qv = reinterpret_cast<R*>(smem + L::oQ + warp * L::kQ);  // [QN][QCAP]
    int* qo = reinterpret_cast<int*>(qv + QN * QCAP);  // the node, and its place in the output
    int qhead = 0, qcnt = 0;
    // the first cnt (at most 32) nodes of the queue
    const auto work_off = [&](int cnt) {
        __syncwarp();
        if (lane < cnt) {
            const int e = (qhead + lane) & (QCAP - 1);
            const int on = qo[e], ow = qo[QCAP + e];
            const int step[3] = {1, sy, sz};
            unsigned gp[3], gm[3];
            R xc[3], bc[3], ic[3], gu[3][3], F[3];
            const unsigned mask = __ldg(gidm + on) >> 16;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                gp[d] = __ldg(gidm + on + step[d]);
                gm[d] = __ldg(gidm + on - step[d]);
            }
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                xc[r] = OP == SPLIT_JACOBI ? __ldg(x + on + r * sc) : R(0);
                bc[r] = OP != SPLIT_FAPPLY ? b[on + r * sc] : R(0);
                ic[r] = OP == SPLIT_JACOBI ? __ldg(invD + on + r * sc) : R(0);
                F[r] = qv[(12 + r) * QCAP + e];
                gu[r][0] = qv[r * QCAP + e];
                gu[r][1] = qv[(3 + r) * QCAP + e];
                gu[r][2] = sub_rn(qv[(6 + r) * QCAP + e], qv[(9 + r) * QCAP + e]);
            }
            with_gradc(mask, gp, gm, gu, F);
#pragma unroll
            for (int r = 0; r < 3; ++r) out[ow + r * osc] = value(xc[r], bc[r], ic[r], F[r]);
        }
        __syncwarp();
        qhead = (qhead + cnt) & (QCAP - 1);
        qcnt -= cnt;
    };

    PlaneRegs<R> even, odd;
    R xx[3], yy[3], xy[3];                               // in-plane second differences of the middle plane
    const int at = (warp + 1) * L::BW + L::AL + lane;    // node (i, j) inside an x component tile
    const int av = warp * STX + lane;                    // ... inside a b / 1/D / id component tile
    // One plane: x plane k + 1 has arrived in the slot at base.  lo holds plane k - 1 and receives plane
    // k + 1, mid holds plane k, whose row is formed (for the block's first two planes from nothing, and
    // not stored).
    const auto plane = [&](PlaneRegs<R>& lo, PlaneRegs<R>& mid, const unsigned char* base, bool store) {
        const R* xs = reinterpret_cast<const R*>(base) + at;
        const R* vb = reinterpret_cast<const R*>(base + L::oB) + av;
        const R* vi = reinterpret_cast<const R*>(base + L::oI) + av;
        const unsigned gw = store ? reinterpret_cast<const unsigned*>(base + L::oG)[av] : 0u;
        const bool wide = !uniform && (gw >> 16) != 0;  // has a grad C column
        const unsigned ball = __ballot_sync(0xffffffffu, wide);
        int e = -1;  // queue entry
        if (wide) {
            e = (qhead + qcnt + __popc(ball & ((1u << lane) - 1u))) & (QCAP - 1);
            qo[e] = o;
            qo[QCAP + e] = oo;
        }
        qcnt += __popc(ball);
        const R* tr = TABS ? ts + (int)(gw & 0xffffu) * TS : tab;
        R D[3][6], F[3];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const R* u = xs + p * L::XP;
            const R c = u[0], xm = u[-1], xp = u[1], ym = u[-L::BW], yp = u[L::BW];
            const R dx = sub_rn(xp, xm), dy = sub_rn(yp, ym);
            D[p][kXX] = xx[p];
            D[p][kYY] = yy[p];
            D[p][kXY] = xy[p];
            D[p][kZZ] = add_rn(fma_rn(R(-2), mid.c[p], c), lo.c[p]);
            D[p][kXZ] = sub_rn(dx, lo.dx[p]);
            D[p][kYZ] = sub_rn(dy, lo.dy[p]);
            if (e >= 0) {
                qv[p * QCAP + e] = mid.dx[p];
                qv[(3 + p) * QCAP + e] = mid.dy[p];
                qv[(6 + p) * QCAP + e] = c;
                qv[(9 + p) * QCAP + e] = lo.c[p];
            }
            lo.c[p] = c;
            lo.dx[p] = dx;
            lo.dy[p] = dy;
            xx[p] = add_rn(fma_rn(R(-2), c, xp), xm);
            yy[p] = add_rn(fma_rn(R(-2), c, yp), ym);
            xy[p] = sub_rn(sub_rn(u[1 + L::BW], u[1 - L::BW]), sub_rn(u[-1 + L::BW], u[-1 - L::BW]));
        }
        {
            row_scale(K, D);
            if constexpr (TABS) {
                row_sum<M>([&](int q) { return tr[q]; }, D, F);
            } else {
                R a[NC];
                const R* ag = tab + (int)(gw & 0xffffu) * NC;
#pragma unroll
                for (int q = 0; q < NC; ++q) a[q] = __ldg(ag + q);
                row_sum<M>([&](int q) { return row_number<M>([&](int u) { return a[u]; }, q); }, D, F);
            }
        }
        if (e >= 0) {
#pragma unroll
            for (int r = 0; r < 3; ++r) qv[(12 + r) * QCAP + e] = F[r];
        }
        if (store && e < 0) {
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const R bc = OP != SPLIT_FAPPLY ? vb[r * L::VP] : R(0), ic = OP == SPLIT_JACOBI ? vi[r * L::VP] : R(0);
                out[oo + r * osc] = value(mid.c[r], bc, ic, F[r]);
            }
        }
    };
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        even.c[p] = even.dx[p] = even.dy[p] = odd.c[p] = odd.dx[p] = odd.dy[p] = R(0);
        xx[p] = yy[p] = xy[p] = R(0);
    }
    bool failed = TABS && !__all_sync(0xffffffffu, mbar_wait(tbar, 0));
    int s = 0;
    unsigned phase = 0;
    for (int t = 0; !failed && t < planes; ++t, o += sz, oo += osz) {  // x plane k0 - 1 + t
        failed = !__all_sync(0xffffffffu, mbar_wait(full(s), phase));
        if (failed) break;
        const unsigned char* base = smem + s * L::kSlot;
        if (t & 1) plane(odd, even, base, act && t >= 2);
        else plane(even, odd, base, act && t >= 2);
        // the slot has been read by every lane: hand it back
        __syncwarp();
        if (lane == 0) mbar_arrive(empty(s));
        if (qcnt >= 32 || (t + 1 == planes && qcnt > 0)) work_off(min(qcnt, 32));
        if (t + 1 == planes && qcnt > 0) work_off(qcnt);
        if (++s == SRING) {
            s = 0;
            phase ^= 1u;
        }
    }
    if (failed && lane == 0) atomicExch(err, 1);
}

// ------------------------------------------------------------------ FP32
// The same sweep in FP32.  It is bound by issue and by the shared-memory data path (a word per lane and
// cycle), no unit saturated: a block of 128 threads owns a 32 x 8 column and marches 8 planes, two rows
// per thread, which share the loads of the rows between them in every plane (28 instead of 38 loads per
// component).  One thread issues, per plane, the TMA loads of the x halo tile, b, 1/D and the ids one
// stage ahead.  The rows are div_mm's 21 coefficients a node: the 36 sums of the FP64 rows would be 12
// more words of that path.  Nodes with a grad C column (a mask in the id word) go to a queue and are
// finished after a block barrier by the first threads.
//
// Jacobi at 257^3, tile and list kernels: 0.264 ms.  Slower: packed FMAs over the 36 sums, 0.290 (1/D
// past the tiles, five blocks) and 0.296 (four); the register-marching form of the FP64 kernel, 0.315
// at 112 registers and two blocks, 0.355 at 72 and three, two rows a thread 0.42-0.48.
constexpr int SNT = STX * STY;
constexpr int T32B = 36;                      // box width: 32 nodes + halo + alignment shift (<= 2)
constexpr int T32X = T32B * SXR;              // elements per x component plane tile
constexpr int T32V = T32B * STY;              // elements per b / 1/D / id component tile (no halo)
#ifndef AE_SPLIT_PAIR_BLOCKS
#define AE_SPLIT_PAIR_BLOCKS 5
#endif
struct TL32 {
    static constexpr int XS = up128(3 * T32X * 4);  // bytes per x ring slot (planes k - 1, k, k + 1, one in flight)
    static constexpr int VS = 3 * T32V * 4;         // bytes per b / 1/D ring slot (two)
    static constexpr int GS = T32V * 4;             // bytes per id ring slot (two)
    static constexpr int oB = 4 * XS, oI = oB + 2 * VS, oG = oI + 2 * VS, oBar = oG + 2 * GS;
    static constexpr int oQ = oBar + 16, oQt = oQ + 16, oQf = oQt + 4 * SNT;  // queue: count, places, sums
    static constexpr int oT = oQf + 3 * SNT * 4;
    static constexpr unsigned kX = 3 * T32X * 4, kV = 3 * T32V * 4, kG = T32V * 4;
    static_assert(VS % 128 == 0 && GS % 128 == 0 && oB % 128 == 0 && oT % 16 == 0, "TMA slots, table");
};
constexpr int kTab32SmemMax = 24 * 1024;  // bytes of grain table kept in shared memory
template <int M, bool TABS, int OP>
__global__ void __launch_bounds__(SNT / 2, AE_SPLIT_PAIR_BLOCKS)
    k_sweep_tile32(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_b,
                 const __grid_constant__ CUtensorMap tm_i, const __grid_constant__ CUtensorMap tm_g,
                   SCoef<float> K, TileGeo T, int sh, int uniform, long long sy, long long sz, long long sc,
                   const unsigned* __restrict__ gidm_g, const float* __restrict__ tab, int tab_n, float* __restrict__ xo,
                   long long osy, long long osz, long long osc, float omega, int* err) {
    using R = float;
    constexpr int NPT = 2, NT = SNT / NPT;  // rows per thread, threads per block
    using L = TL32;
    constexpr int NC = NCoef<M>::value;
    // grain rows in shared memory padded to whole 16-byte vectors (four coefficients)
    constexpr int NCP = (NC + 3) / 4 * 4;
    constexpr int TS = TABS ? NCP : NC;  // row stride of the table the kernel reads
    extern __shared__ __align__(128) unsigned char smem[];
    auto xslot = [&](int k) { return reinterpret_cast<const R*>(smem + (k & 3) * L::XS); };
    const unsigned* gring = reinterpret_cast<const unsigned*>(smem + L::oG);
    int* qn = reinterpret_cast<int*>(smem + L::oQ);
    int* qtid = reinterpret_cast<int*>(smem + L::oQt);
    R* qf = reinterpret_cast<R*>(smem + L::oQf);
    const R* tb = tab;
    if (TABS) {
        R* ts = reinterpret_cast<R*>(smem + L::oT);
        const int rows = tab_n / NC;
        for (int q = threadIdx.x; q < rows * NCP; q += NT) {
            const int g = q / NCP, c = q - g * NCP;
            ts[q] = c < NC ? __ldg(tab + g * NC + c) : R(0);
        }
        tb = ts;
    }
    const int tx = threadIdx.x % STX, ty = NPT * (threadIdx.x / STX);  // the thread's first row
    const int i0 = T.I.lo[0] + (int)(blockIdx.x % T.tiles_x) * STX, j0 = T.I.lo[1] + (int)(blockIdx.x / T.tiles_x) * STY;
    const int k0 = T.I.lo[2] + (int)blockIdx.y * T.kz;
    const int k1 = min(k0 + T.kz - 1, T.I.hi[2]);
    const int i = i0 + tx, j = j0 + ty;
    const bool act = i <= T.I.hi[0] && j <= T.I.hi[1];
    auto act_n = [&](int n) { return i <= T.I.hi[0] && j + n <= T.I.hi[1]; };  // node n of the thread
    // tensor coordinates of the boxes
    const int xa = i0 - 1 - T.slo[0] - sh;
    const int yx = j0 - 1 - T.slo[1], yv = j0 - T.slo[1];
    const unsigned sb = smem_u32(smem);
    const unsigned bar0 = sb + (unsigned)L::oBar;
    const bool leader = threadIdx.x == 0;
    if (leader) {
        *qn = 0;
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    auto load_x = [&](int k, unsigned bar) {
        tma_load4(sb + (unsigned)((k & 3) * L::XS), &tm_x, xa, yx, k - T.slo[2], 0, bar);
    };
    auto load_v = [&](int k, unsigned bar) {
        const unsigned s = (unsigned)(k & 1);
        if (OP != SPLIT_FAPPLY) tma_load4(sb + (unsigned)L::oB + s * L::VS, &tm_b, xa, yv, k - T.slo[2], 0, bar);
        if (OP == SPLIT_JACOBI) tma_load4(sb + (unsigned)L::oI + s * L::VS, &tm_i, xa, yv, k - T.slo[2], 0, bar);
        tma_load4(sb + (unsigned)L::oG + s * L::GS, &tm_g, xa, yv, k - T.slo[2], 0, bar);
    };
    constexpr unsigned kVTile = (OP == SPLIT_JACOBI ? 2 : OP == SPLIT_RESIDUAL ? 1 : 0) * L::kV + L::kG;
    // stage 0: planes k0-1, k0, k0+1 of x and the b, 1/D, id tiles of plane k0
    if (leader) {
        mbar_expect_tx(bar0, 3 * L::kX + kVTile);
        load_x(k0 - 1, bar0);
        load_x(k0, bar0);
        load_x(k0 + 1, bar0);
        load_v(k0, bar0);
    }
    const int col = sh + 1 + tx;
    const int cx = (ty + 1) * T32B + col;  // this node inside an x component tile
    const int cv = ty * T32B + col;        // ... inside a b / 1/D / id component tile
    // node (i, j, k) in the output
    long long o = (long long)(i - T.slo[0]) + (long long)(j - T.slo[1]) * osy + (long long)(k0 - T.slo[2]) * osz;
    bool failed = false;
    int last = 0;  // last stage issued
    for (int k = k0; k <= k1; ++k, o += osz) {
        const int s = k - k0;
        // stage s + 1: plane k + 2 of x and the tiles of plane k + 1; their ring slots were last
        // read in iteration k - 1, which the barrier at its end closed
        if (k + 1 <= k1) {
            last = s + 1;
            if (leader) {
                const unsigned bn = bar0 + 8u * (unsigned)((s + 1) & 1);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                mbar_expect_tx(bn, L::kX + kVTile);
                load_x(k + 2, bn);
                load_v(k + 1, bn);
            }
        }
        const bool ok = mbar_wait(bar0 + 8u * (unsigned)(s & 1), (unsigned)((s >> 1) & 1));
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
        const unsigned vs = (unsigned)(k & 1);
        const R* pm = xslot(k - 1) + cx;
        const R* pc = xslot(k) + cx;
        const R* pp = xslot(k + 1) + cx;
        const R* bv = reinterpret_cast<const R*>(smem + L::oB + vs * L::VS) + cv;
        const R* iv = reinterpret_cast<const R*>(smem + L::oI + vs * L::VS) + cv;
        bool queued[NPT];
        R f[NPT][3], xv[NPT][3];
        // the 21 (9, 2, 45) coefficients of a node's grain, then its interior term div(C : grad grad x)
        auto interior = [&](unsigned gw, const R (&bb)[3][3][3], R (&fo)[3]) {
            R a[NCP];
            const R* a0 = tb + (int)(gw & 0xffffu) * TS;
            if (TABS) {
#pragma unroll
                for (int q = 0; q < NCP; q += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(a0 + q);
                    a[q] = v.x;
                    a[q + 1] = v.y;
                    a[q + 2] = v.z;
                    a[q + 3] = v.w;
                }
            } else {
#pragma unroll
                for (int q = 0; q < NC; ++q) a[q] = a0[q];
            }
            div_of<M, R>(a, bb, fo);
        };
        {
#pragma unroll
            for (int n = 0; n < NPT; ++n) queued[n] = false;
            if (act) {
                // per component: plane k at rows j - 1 .. j + NPT and columns i - 1 .. i + 1;
                // planes k -+ 1 at rows j .. j + NPT - 1 (three columns) and rows j - 1, j + NPT
                // (column i).  Row r of these arrays is row j - 1 + r.
                constexpr int NR = NPT + 2;
                R h[NPT][3][6];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const R* um = pm + p * T32X;
                    const R* uc = pc + p * T32X;
                    const R* up = pp + p * T32X;
                    R ac[NR][3], am[NR][3], ap[NR][3];
#pragma unroll
                    for (int r = 0; r < NR; ++r)
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            ac[r][c] = uc[(r - 1) * T32B + c - 1];
                            const bool need = (r >= 1 && r <= NPT) || c == 1;
                            am[r][c] = need ? um[(r - 1) * T32B + c - 1] : R(0);
                            ap[r][c] = need ? up[(r - 1) * T32B + c - 1] : R(0);
                        }
#pragma unroll
                    for (int n = 0; n < NPT; ++n) {
                        const R c0 = ac[n + 1][1];
                        xv[n][p] = c0;
                        const R xm = ac[n + 1][0], xp = ac[n + 1][2], ym = ac[n][1], yp = ac[n + 2][1];
                        const R zm = am[n + 1][1], zp = ap[n + 1][1];
                        h[n][p][0] = (xp - R(2) * c0 + xm) * K.i2[0];
                        h[n][p][1] = (yp - R(2) * c0 + ym) * K.i2[1];
                        h[n][p][2] = (zp - R(2) * c0 + zm) * K.i2[2];
                        h[n][p][3] = (ac[n + 2][2] + ac[n][0] - ac[n][2] - ac[n + 2][0]) * K.m01;
                        h[n][p][4] = (ap[n + 1][2] + am[n + 1][0] - am[n + 1][2] - ap[n + 1][0]) * K.m02;
                        h[n][p][5] = (ap[n + 2][1] + am[n][1] - am[n + 2][1] - ap[n][1]) * K.m12;
                    }
                }
#pragma unroll
                for (int n = 0; n < NPT; ++n) {
                    if (n > 0 && !act_n(n)) break;
                    const unsigned gw = gring[vs * T32V + cv + n * T32B];
                    R bb[3][3][3];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        bb[p][0][0] = h[n][p][0];
                        bb[p][1][1] = h[n][p][1];
                        bb[p][2][2] = h[n][p][2];
                        bb[p][0][1] = bb[p][1][0] = h[n][p][3];
                        bb[p][0][2] = bb[p][2][0] = h[n][p][4];
                        bb[p][1][2] = bb[p][2][1] = h[n][p][5];
                    }
                    interior(gw, bb, f[n]);
                    queued[n] = !uniform && (gw >> 16) != 0;
                }
            }
        }
        // nodes with a grad C column go to the plane's queue (one shared-memory atomic per warp
        // and row); the others are finished here
#pragma unroll
        for (int n = 0; n < NPT; ++n) {
            const bool an = n == 0 ? act : act && act_n(n);
            const unsigned ball = __ballot_sync(0xffffffffu, queued[n]);
            if (ball) {
                const int lane = threadIdx.x & 31;
                int base = 0;
                if (lane == __ffs(ball) - 1) base = atomicAdd(qn, __popc(ball));
                base = __shfl_sync(0xffffffffu, base, __ffs(ball) - 1);
                if (queued[n]) {
                    const int e = base + __popc(ball & ((1u << lane) - 1u));
                    qtid[e] = (ty + n) * STX + tx;  // the node's place in the tile
                    qf[3 * e] = f[n][0];
                    qf[3 * e + 1] = f[n][1];
                    qf[3 * e + 2] = f[n][2];
                }
            }
            if (an && !queued[n]) {
                const long long on = o + n * osy;
                const int vn = n * T32B;
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    if (OP == SPLIT_JACOBI)
                        xo[on + r * osc] = jacobi_update<R>(xv[n][r], sub_rn(bv[vn + r * T32V], f[n][r]), iv[vn + r * T32V], omega);
                    else if (OP == SPLIT_RESIDUAL)
                        xo[on + r * osc] = bv[vn + r * T32V] - f[n][r];
                    else
                        xo[on + r * osc] = f[n][r];
                }
            }
        }
        __syncthreads();
        // the queued nodes, one per thread: grad C columns of the directions whose neighbours lie in
        // different grains, then the update
        for (int e = threadIdx.x; e < *qn; e += NT) {
            const int t = qtid[e];
            const int qx = t % STX, qy = t / STX;
            const int qcx = (qy + 1) * T32B + sh + 1 + qx, qcv = qy * T32B + sh + 1 + qx;
            const long long qo = (long long)(i0 + qx - T.slo[0]) + (long long)(j0 + qy - T.slo[1]) * sy + (long long)(k - T.slo[2]) * sz;
            const long long ow = o + (long long)(qx - tx) + (long long)(qy - ty) * osy;
            const R* qm = xslot(k - 1) + qcx;
            const R* qc = xslot(k) + qcx;
            const R* qp = xslot(k + 1) + qcx;
            R gu[3][3];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                gu[p][0] = (qc[p * T32X + 1] - qc[p * T32X - 1]) * K.h[0];
                gu[p][1] = (qc[p * T32X + T32B] - qc[p * T32X - T32B]) * K.h[1];
                gu[p][2] = (qp[p * T32X] - qm[p * T32X]) * K.h[2];
            }
            // neighbour ids: x from the tile, y from the tile inside it, the rest from global
            const unsigned* gv = gring + vs * T32V + qcv;
            const unsigned mask = gv[0] >> 16;
            const int gid_n[3][2] = {
                {(int)(gv[1] & 0xffffu), (int)(gv[-1] & 0xffffu)},
                {(int)((qy + 1 < STY ? gv[T32B] : __ldg(gidm_g + qo + sy)) & 0xffffu),
                 (int)((qy > 0 ? gv[-T32B] : __ldg(gidm_g + qo - sy)) & 0xffffu)},
                {(int)(__ldg(gidm_g + qo + sz) & 0xffffu), (int)(__ldg(gidm_g + qo - sz) & 0xffffu)}};
            R colv[3][3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (mask & (1u << d)) {
                    const R* cp = tb + gid_n[d][0] * TS;
                    const R* cm = tb + gid_n[d][1] * TS;
                    gradC_col_f<M, R>([&](int q) { return cp[q] - cm[q]; }, gu, d, colv[d]);
                } else {
                    colv[d][0] = colv[d][1] = colv[d][2] = R(0);
                }
            }
            const R* qb = reinterpret_cast<const R*>(smem + L::oB + vs * L::VS) + qcv;
            const R* qi = reinterpret_cast<const R*>(smem + L::oI + vs * L::VS) + qcv;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                R fr = qf[3 * e + r];
                fr = gradc_add(fr, colv[0][r], colv[1][r], colv[2][r], K.h);
                if (OP == SPLIT_JACOBI)
                    xo[ow + r * osc] = jacobi_update<R>(qc[r * T32X], sub_rn(qb[r * T32V], fr), qi[r * T32V], omega);
                else if (OP == SPLIT_RESIDUAL)
                    xo[ow + r * osc] = qb[r * T32V] - fr;
                else
                    xo[ow + r * osc] = fr;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) *qn = 0;
    }
    if (failed) {
        if (leader) atomicExch(err, 1);
        // loads still in flight may land: wait (bounded) for the stages issued before leaving
        for (int s = max(last - 1, 0); s <= last; ++s) mbar_wait(bar0 + 8u * (unsigned)(s & 1), (unsigned)((s >> 1) & 1));
    }
}

// FP32: 4 resident blocks (64 registers): at 48 the cubic variant spills
template <int M, class R, bool SAME>
__global__ void __launch_bounds__(kBlock, sizeof(R) == 4 ? 4 : 2)
    k_jacobi_list(OpParams P, SCoef<R> K, const unsigned long long* __restrict__ list, long long n, Box3 S,
                  View<const R> C, Grains<R> G, View<const R> invD, View<const R> xi, View<const R> b, View<R> xo,
                  R omega) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int i, j, k;
    unpack_node(list[t], S.lo, i, j, k);
    jacobi_node<M, R, true, SAME>(P, K, C, G, invD, xi, b, xo, omega, i, j, k);
}

// r = b - A x at the listed nodes (the per-node residual, k_residual's arithmetic); r may alias b
template <int M, class R>
__global__ void __launch_bounds__(kBlock, sizeof(R) == 4 ? 4 : 2)
    k_residual_list(OpParams P, SCoef<R> K, const unsigned long long* __restrict__ list, long long n, Box3 S,
                    View<const R> C, Grains<R> G, View<const R> x, View<const R> b, View<R> r) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int i, j, k;
    unpack_node(list[t], S.lo, i, j, k);
    R v[3];
    const long long ox = x.at(i, j, k);
    const R sc = apply_at<M, R, true>(P, K, C, G, x, i, j, k, ox, ox, v);
#pragma unroll
    for (int q = 0; q < 3; ++q) r.p[ox + q * x.sc] = row_residual(b.p[ox + q * x.sc], sc, v[q]);
}

// f = A x at the listed nodes (k_fapply's arithmetic)
template <int M, class R>
__global__ void __launch_bounds__(kBlock, sizeof(R) == 4 ? 4 : 2)
    k_fapply_list(OpParams P, SCoef<R> K, const unsigned long long* __restrict__ list, long long n, Box3 S,
                  View<const R> C, Grains<R> G, View<const R> x, View<R> f) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int i, j, k;
    unpack_node(list[t], S.lo, i, j, k);
    R v[3];
    const long long ox = x.at(i, j, k);
    const R sc = apply_at<M, R, true>(P, K, C, G, x, i, j, k, ox, ox, v);
    const long long of = f.at(i, j, k);
#pragma unroll
    for (int q = 0; q < 3; ++q) f.p[of + q * f.sc] = mul_rn(sc, v[q]);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda)
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    if (!fn) throw std::runtime_error("cuTensorMapEncodeTiled is not available");
    return fn;
}

// Tensor map over a level array [comp][k][j][i] (storage box, row pitch px), boxes of
// width x rows x 1 x ncomp elements of esize bytes.
CUtensorMap level_tmap(const void* base, const Geo& g, int ncomp, int width, int rows, CUtensorMapDataType type, int esize) {
    const Box3 s = geo_store(g);
    const cuuint64_t nx = (cuuint64_t)(s.hi[0] - s.lo[0] + 1), ny = (cuuint64_t)(s.hi[1] - s.lo[1] + 1),
                     nz = (cuuint64_t)(s.hi[2] - s.lo[2] + 1);
    const cuuint64_t px = (cuuint64_t)g.px;
    const cuuint64_t dims[4] = {nx, ny, nz, (cuuint64_t)ncomp};
    const cuuint64_t e = (cuuint64_t)esize;
    const cuuint64_t strides[3] = {px * e, px * ny * e, px * ny * nz * e};
    const cuuint32_t box[4] = {(cuuint32_t)width, (cuuint32_t)rows, 1, (cuuint32_t)ncomp};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUtensorMap m;
    const CUresult r = encode_fn()(&m, type, 4, const_cast<void*>(base), dims, strides, box, estr,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    return m;
}

template <int M, class R, bool TABS, int OP>
void tile_smem_attr() {
    static std::once_flag once;
    std::call_once(once, [] {
        const int tables = !TABS ? 0 : sizeof(R) == 4 ? kTab32SmemMax : kTabSmemMax;
        if constexpr (sizeof(R) == 4)
            AE_CUDA_CHECK(cudaFuncSetAttribute(k_sweep_tile32<M, TABS, OP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               TL32::oT + tables));
        else
            AE_CUDA_CHECK(cudaFuncSetAttribute(k_sweep_tile64<M, TABS, OP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               TL<double>::oT + tables));
    });
}

// the tiled kernel of one operation over I; b: the right-hand side, invD: 1/D (Jacobi only)
template <class R, int OP>
void launch_tile(const OpParams& P, const SplitList& sl, const Box3& I, const Box3& S, View<const R> x, const R* b,
                 const R* invD, View<R> out, R omega, cudaStream_t st, Grains<R> G, int ngrains, int* err) {
    constexpr int E = (int)sizeof(R);
    constexpr bool F32 = E == 4;
    const SCoef<R> K = make_scoef<R>(P.g);
    R* const po = out.p + out.at(S.lo[0], S.lo[1], S.lo[2]);
    const CUtensorMapDataType dt = F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
    dispatch_model<R>(P.model, [&](auto m) {
        constexpr int Mv = decltype(m)::value;
        TileGeo T;
        T.I = I;
        for (int q = 0; q < 3; ++q) T.slo[q] = S.lo[q];
        // FP32 tiles start at I's first column, FP64 tiles at the storage box's
        const int nx = I.hi[0] - (F32 ? I : S).lo[0] + 1, ny = I.hi[1] - I.lo[1] + 1, nz = I.hi[2] - I.lo[2] + 1;
        T.tiles_x = (nx + STX - 1) / STX;
        const int tiles = T.tiles_x * ((ny + STY - 1) / STY);
        T.kz = sl.kz > 0 ? sl.kz : F32 ? 8 : tile_kz(tiles, nz, 152);
        const int vw = F32 ? T32B : STX;
        const CUtensorMap tx = level_tmap(x.p, P.g, 3, F32 ? T32B : TL<double>::BW, SXR, dt, E);
        const CUtensorMap tb = level_tmap(b ? b : x.p, P.g, 3, vw, STY, dt, E);
        const CUtensorMap ti = level_tmap(invD ? invD : x.p, P.g, 3, vw, STY, dt, E);
        const CUtensorMap tg = level_tmap(sl.gidm, P.g, 1, vw, STY, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4);
        const dim3 grid((unsigned)tiles, (unsigned)((nz + T.kz - 1) / T.kz));
        const size_t rows_bytes = ((size_t)ngrains * row_stride<Mv>() * E + 15) / 16 * 16;
        size_t tab_bytes = ((size_t)ngrains * NCoef<Mv>::value * E + 15) / 16 * 16;
        if (rows_bytes + tab_bytes > kTabSmemMax) tab_bytes = 0;
        // FP32: the stiffness table alone, rows padded to 16 bytes
        const size_t pad_bytes = (size_t)ngrains * ((NCoef<Mv>::value + 3) / 4 * 4) * E;
        const auto go = [&](auto tabs) {
            constexpr bool TABS = decltype(tabs)::value;
            tile_smem_attr<Mv, R, TABS, OP>();
            if constexpr (F32) {
                // every tile starts 32 nodes after the previous one, so one shift serves all of them: the
                // boxes' first column is then a multiple of 4
                const int sh = (I.lo[0] - 1 - S.lo[0]) & 3;
                k_sweep_tile32<Mv, TABS, OP><<<grid, SNT / 2, TL32::oT + (TABS ? pad_bytes : 0), st>>>(
                    tx, tb, ti, tg, K, T, sh, P.uniform, x.sy, x.sz, x.sc, sl.gidm, G.tab, ngrains * NCoef<Mv>::value, po,
                    out.sy, out.sz, out.sc, omega, err);
            } else {
                k_sweep_tile64<Mv, TABS, OP><<<grid, kTileThreads, TL<double>::oT + (TABS ? rows_bytes + tab_bytes : 0), st>>>(
                    tx, tb, ti, tg, K, T, P.uniform, (int)x.sy, (int)x.sz, x.sc, sl.gidm, G.tab, sl.rows64,
                    TABS ? (int)rows_bytes : 0, TABS ? (int)tab_bytes : 0, x.p, b, invD, po, (int)out.sy,
                    (int)out.sz, out.sc, omega, err);
            }
            launched();
        };
        if (F32 ? pad_bytes <= kTab32SmemMax : rows_bytes <= kRowSmemMax) go(std::true_type());
        else go(std::false_type());
    });
}

}  // namespace

bool split_supported(const Geo& g) {
    if (g.px <= 0 || g.px % 4 != 0) return false;
    const Box3 S = geo_store(g);
    for (int q = 0; q < 3; ++q)
        if (S.hi[q] - S.lo[q] >= (1 << 21)) return false;
    // the FP32 tiles' column shift (sh in launch_tile) must leave the 34 columns of a tile inside the box:
    // 0 on level 0 and on refined patches with 2 ghost layers, 1 or 2 where one touches the domain's
    // low face
    const Box3 I = geo_interior(g);
    return ((I.lo[0] - 1 - S.lo[0]) & 3) <= T32B - 34 && split_range(geo_nn(g) / (S.hi[2] - S.lo[2] + 1), geo_nn(g));
}

// count and fill the list of region R \ I (and, with gidm, the id/mask array)
long long build_list(const Reg& reg, const Box3& R, const Box3& I, View<const unsigned short> gid, unsigned* gidm,
                     unsigned long long** list, cudaStream_t st, unsigned long long* scratch_count) {
    AE_CUDA_CHECK(cudaMemsetAsync(scratch_count, 0, sizeof(unsigned long long), st));
    k_split_mark<false><<<nblocks(reg.n), kBlock, 0, st>>>(reg, R, I, gid, nullptr, nullptr, scratch_count);
    launched();
    unsigned long long n = 0;
    AE_CUDA_CHECK(cudaMemcpyAsync(&n, scratch_count, sizeof(n), cudaMemcpyDeviceToHost, st));
    AE_CUDA_CHECK(cudaStreamSynchronize(st));
    *list = nullptr;
    if (n > 0) AE_CUDA_CHECK(cudaMalloc(list, sizeof(unsigned long long) * n));
    if (n > 0 || gidm) {
        AE_CUDA_CHECK(cudaMemsetAsync(scratch_count, 0, sizeof(unsigned long long), st));
        k_split_mark<true><<<nblocks(reg.n), kBlock, 0, st>>>(reg, R, I, gid, gidm, *list, scratch_count);
        launched();
        AE_CUDA_CHECK(cudaStreamSynchronize(st));
    }
    return (long long)n;
}

void split_free(SplitList& sl) {
    cudaFree(sl.list);
    cudaFree(sl.list_r);
    cudaFree(sl.gidm);
    cudaFree(sl.rows64);
    sl = SplitList{};
}

long long split_build(const Geo& g, int model, View<const unsigned short> gid, int ngrains, const double* tab,
                      SplitList& sl, cudaStream_t st, unsigned long long* scratch_count) {
    if (!split_supported(g)) throw std::runtime_error("split sweep: level layout not supported");
    const Box3 S = geo_store(g);
    const Reg reg = make_reg(S);
    const Box3 I = geo_interior(g);
    AE_CUDA_CHECK(cudaMalloc(&sl.gidm, sizeof(unsigned) * (size_t)geo_nn(g)));
    AE_CUDA_CHECK(cudaMemsetAsync(sl.gidm, 0, sizeof(unsigned) * (size_t)geo_nn(g), st));
    dispatch_model<double>(model, [&](auto m) {
        constexpr int M = decltype(m)::value;
        const size_t n = (size_t)ngrains * row_stride<M>() + 4;  // the bulk copy takes whole 16 bytes
        AE_CUDA_CHECK(cudaMalloc(&sl.rows64, n * sizeof(double)));
        k_row_table<M><<<nblocks((unsigned)ngrains), kBlock, 0, st>>>(tab, ngrains, sl.rows64);
        launched();
    });
    // the Jacobi sweep writes the whole storage box, the residual the apply region
    sl.n = build_list(reg, S, I, gid, sl.gidm, &sl.list, st, scratch_count);
    sl.n_r = build_list(reg, geo_apply_region(g), I, gid, nullptr, &sl.list_r, st, scratch_count);
    return sl.n;
}

template <class R>
void launch_jacobi_split(const OpParams& P, const SplitList& sl, View<const R> C, View<const R> invD, View<const R> xi,
                         View<const R> b, View<R> xo, R omega, cudaStream_t st, Grains<R> G,
                         int ngrains, int* err) {
    const Box3 S = geo_store(P.g);
    const Box3 I = geo_interior(P.g);
    const bool in = same_layout(xi, C) && same_layout(xi, invD) && same_layout(xi, b), same = in && same_layout(xi, xo);
    if (!in || !split_out(xo) || !split_supported(P.g)) throw std::runtime_error("split sweep needs the level's internal arrays");
    if (!box_empty(I))
        launch_tile<R, SPLIT_JACOBI>(P, sl, I, S, xi, b.p, invD.p, xo, omega, st, G, ngrains, err);
    if (sl.n > 0) {
        const SCoef<R> K = make_scoef<R>(P.g);
        dispatch_model<R>(P.model, [&](auto m) {
            constexpr int Mv = decltype(m)::value;
            const unsigned nb = (unsigned)((sl.n + kBlock - 1) / kBlock);
            if (same) k_jacobi_list<Mv, R, true><<<nb, kBlock, 0, st>>>(P, K, sl.list, sl.n, S, C, G, invD, xi, b, xo, omega);
            else k_jacobi_list<Mv, R, false><<<nb, kBlock, 0, st>>>(P, K, sl.list, sl.n, S, C, G, invD, xi, b, xo, omega);
        });
        launched();
    }
}

template <class R>
void launch_residual_split(const OpParams& P, const SplitList& sl, View<const R> C, View<const R> x, View<const R> b,
                           View<R> r, cudaStream_t st, Grains<R> G, int ngrains, int* err) {
    const Box3 S = geo_store(P.g);
    const Box3 I = geo_interior(P.g);
    const bool same = same_layout(x, C) && same_layout(x, b) && same_layout(x, r);
    if (!same || !split_supported(P.g)) throw std::runtime_error("split sweep needs the level's internal arrays");
    if (!box_empty(I))
        launch_tile<R, SPLIT_RESIDUAL>(P, sl, I, S, x, b.p, nullptr, r, R(0), st, G, ngrains, err);
    if (sl.n_r > 0) {
        const SCoef<R> K = make_scoef<R>(P.g);
        dispatch_model<R>(P.model, [&](auto m) {
            k_residual_list<decltype(m)::value, R><<<(unsigned)((sl.n_r + kBlock - 1) / kBlock), kBlock, 0, st>>>(
                P, K, sl.list_r, sl.n_r, S, C, G, x, b, r);
        });
        launched();
    }
}

template <class R>
void launch_fapply_split(const OpParams& P, const SplitList& sl, View<const R> C, View<const R> x, View<R> f,
                         cudaStream_t st, Grains<R> G, int ngrains, int* err) {
    const Box3 S = geo_store(P.g);
    const Box3 I = geo_interior(P.g);
    if (!same_layout(x, C) || !split_out(f) || !split_supported(P.g)) throw std::runtime_error("split sweep needs the level's internal arrays");
    if (!box_empty(I)) launch_tile<R, SPLIT_FAPPLY>(P, sl, I, S, x, (const R*)nullptr, nullptr, f, R(0), st, G, ngrains, err);
    if (sl.n_r > 0) {
        const SCoef<R> K = make_scoef<R>(P.g);
        dispatch_model<R>(P.model, [&](auto m) {
            k_fapply_list<decltype(m)::value, R><<<(unsigned)((sl.n_r + kBlock - 1) / kBlock), kBlock, 0, st>>>(
                P, K, sl.list_r, sl.n_r, S, C, G, x, f);
        });
        launched();
    }
}

template void launch_fapply_split<float>(const OpParams&, const SplitList&, View<const float>, View<const float>,
                                         View<float>, cudaStream_t, Grains<float>, int, int*);
template void launch_fapply_split<double>(const OpParams&, const SplitList&, View<const double>, View<const double>,
                                          View<double>, cudaStream_t, Grains<double>, int, int*);
template void launch_jacobi_split<float>(const OpParams&, const SplitList&, View<const float>, View<const float>,
                                         View<const float>, View<const float>, View<float>, float,
                                         cudaStream_t, Grains<float>, int, int*);
template void launch_jacobi_split<double>(const OpParams&, const SplitList&, View<const double>, View<const double>,
                                          View<const double>, View<const double>, View<double>, double,
                                          cudaStream_t, Grains<double>, int, int*);
template void launch_residual_split<float>(const OpParams&, const SplitList&, View<const float>, View<const float>,
                                           View<const float>, View<float>, cudaStream_t, Grains<float>, int, int*);
template void launch_residual_split<double>(const OpParams&, const SplitList&, View<const double>, View<const double>,
                                            View<const double>, View<double>, cudaStream_t, Grains<double>, int, int*);

}  // namespace ae
