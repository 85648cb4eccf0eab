// Device-side building blocks of the nodal elastic operator: geometry, field views,
// finite-difference stencils, stiffness contractions, boundary rows and the per-node
// operator.  Templated on the arithmetic type R (double or float) and on the stiffness
// kind M.
//
// Reference formulas restated here:
//   stencils          src/Numeric/Stencil.H:16-176
//   MajorMinor C:grad src/Set/Matrix4_MajorMinor.H:253-269, C:gradgrad :287-345
//   Isotropic         src/Set/Matrix4_Isotropic.H:60-91
//   Diagonal          src/Set/Matrix4_Diagonal.H:48-74
//   Major (45 slots)  src/Set/Matrix4_Major.H:198-300, 399-428
//   boundary rows     src/BC/Operator/Elastic.H:218-303
//   Fapply            src/Operator/Elastic.cpp:174-258
#pragma once
#include <cstdint>

namespace ae {

enum Model { ISO = 0, MM = 1, DIAG = 2, MAJOR = 3 };
template <int M> struct NCoef;
template <> struct NCoef<ISO> { static constexpr int value = 2; };
template <> struct NCoef<MM> { static constexpr int value = 21; };
template <> struct NCoef<DIAG> { static constexpr int value = 9; };
template <> struct NCoef<MAJOR> { static constexpr int value = 45; };

// Set::Matrix4<3, Sym::Major>: the 9 x 9 matrix A(3i+j, 3k+l) = C_ijkl is symmetric; its upper
// triangle is stored row by row in 45 slots.  Slot of entry (I, K).
__host__ __device__ constexpr int major_slot(int I, int K) {
    return I <= K ? I * 9 - I * (I - 1) / 2 + (K - I) : K * 9 - K * (K - 1) / 2 + (I - K);
}

// Rows in one fixed rounding order.  The compiler fuses a product into a neighbouring addition at its
// own discretion, and the choice can differ between kernels that inline the same expression in
// different surroundings.  The operator's interior rows therefore go through explicitly rounded
// operations, so that every kernel computes a node's row to the same bits.
__device__ __forceinline__ float mul_rn(float x, float y) { return __fmul_rn(x, y); }
__device__ __forceinline__ double mul_rn(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ float add_rn(float x, float y) { return __fadd_rn(x, y); }
__device__ __forceinline__ double add_rn(double x, double y) { return __dadd_rn(x, y); }
__device__ __forceinline__ float sub_rn(float x, float y) { return __fsub_rn(x, y); }
__device__ __forceinline__ double sub_rn(double x, double y) { return __dsub_rn(x, y); }
__device__ __forceinline__ float fma_rn(float x, float y, float z) { return __fmaf_rn(x, y, z); }
__device__ __forceinline__ double fma_rn(double x, double y, double z) { return __fma_rn(x, y, z); }
template <class R>
__device__ __forceinline__ R fx_sop_acc(R r) { return r; }
template <class R, class... T>
__device__ __forceinline__ R fx_sop_acc(R r, R a, R x, T... rest) {
    return fx_sop_acc(fma_rn(a, x, r), rest...);
}
// a0 x0 + a1 x1 + ... in that order: the first product rounded, each further one fused into the sum
template <class R, class... T>
__device__ __forceinline__ R fx_sop(R a, R x, T... rest) {
    return fx_sop_acc(mul_rn(a, x), rest...);
}
template <class R>
__device__ __forceinline__ R add2(R x, R y) { return add_rn(x, y); }
// a0 x0 + ... + a5 x5 (one row of a MajorMinor contraction)
template <class R>
__device__ __forceinline__ R sop6(R a0, R x0, R a1, R x1, R a2, R x2, R a3, R x3, R a4, R x4, R a5, R x5) {
    return fx_sop(a0, x0, a1, x1, a2, x2, a3, x3, a4, x4, a5, x5);
}
// (c0 h0 + c1 h1) + c2 h2: the grad C columns of a row scaled by the central-difference factors
template <class R>
__device__ __forceinline__ R gradc_sum(R c0, R c1, R c2, const R h[3]) { return fx_sop(c0, h[0], c1, h[1], c2, h[2]); }
// f + the grad C term of the row
template <class R>
__device__ __forceinline__ R gradc_add(R f, R c0, R c1, R c2, const R h[3]) { return add_rn(f, gradc_sum(c0, c1, c2, h)); }

enum BCType { DISP = 0, TRAC = 1, PERIODIC = 2, NEUMANN = 3 };

struct Box3 {
    int lo[3], hi[3];
};

// One level (one nodal patch): domain, valid box, ghost layers stored around it.
struct Geo {
    int dlo[3], dhi[3];  // nodal problem domain (inclusive)
    int vlo[3], vhi[3];  // nodal valid box
    int ng;              // ghost layers stored: storage box = grow(valid, ng)
    int px = 0;          // row pitch of the level's internal arrays in nodes (0: the storage box's
                         // x-extent); padded to a multiple of 4 so rows start on 16-byte boundaries
    double dx[3];
};

// Field view in AMReX Array4 order: p points at (lo, comp 0).
template <class T>
struct View {
    T* p;
    int lo[3];
    long long sy, sz, sc;
    int wx = 0;  // nodes per row when the row pitch sy is padded past them (0: sy)
    __host__ __device__ __forceinline__ long long at(int i, int j, int k) const {
        return (long long)(i - lo[0]) + (long long)(j - lo[1]) * sy + (long long)(k - lo[2]) * sz;
    }
};

// Stencil constants, computed on the host in double precision.
template <class R>
struct SCoef {
    R h[3];        // 0.5 / dx   (central first derivative)
    R id[3];       // 1 / dx     (one-sided first derivative)
    R i2[3];       // 1 / dx^2   (second derivative)
    R m01, m02, m12;  // 0.25 / (dx_a dx_b)  (mixed derivative)
    R bb[3];       // -2 / dx / dx  (diagonal of the second derivative)
    // the interior row as i2[0] times a row of unscaled differences (row_of below)
    R q[3];        // dx_0 / dx_d
    R sd[6];       // q factors of the differences xx, yy, zz, xy, xz, yz (1/4 of the mixed ones apart)
    int iso;       // equal spacing: every q is 1
};
// fills the members for the spacing dx (host)
template <class R>
inline SCoef<R> scoef_of(const double dx[3]) {
    SCoef<R> K;
    for (int d = 0; d < 3; ++d) {
        K.h[d] = (R)(0.5 / dx[d]);
        K.id[d] = (R)(1.0 / dx[d]);
        K.i2[d] = (R)(1.0 / (dx[d] * dx[d]));
        K.bb[d] = (R)(-2.0 / dx[d] / dx[d]);
        K.q[d] = (R)(dx[0] / dx[d]);
    }
    K.m01 = (R)(0.25 / (dx[0] * dx[1]));
    K.m02 = (R)(0.25 / (dx[0] * dx[2]));
    K.m12 = (R)(0.25 / (dx[1] * dx[2]));
    const int a[6] = {0, 1, 2, 0, 0, 1}, b[6] = {0, 1, 2, 1, 2, 2};
    for (int s = 0; s < 6; ++s) K.sd[s] = (R)((dx[0] / dx[a[s]]) * (dx[0] / dx[b[s]]));
    K.iso = dx[0] == dx[1] && dx[0] == dx[2];
    return K;
}

// BC types per face (26) and direction (3).
struct BCP {
    unsigned char t[26][3];
};

// Truncated normals of src/BC/Operator/Elastic.H:218-219
#define AE_SQRT3INV 0.57735026919
#define AE_SQRT2INV 0.70710678118

// Face index of a domain-boundary node, -1 for interior nodes; numbering and
// precedence (corner, edge, face) of src/BC/Operator/Elastic.H:236-278.
template <class R>
__device__ __forceinline__ int classify(const Geo& g, int i, int j, int k, R n[3]) {
    const int s0 = (i == g.dlo[0]) ? -1 : (i == g.dhi[0]) ? 1 : 0;
    const int s1 = (j == g.dlo[1]) ? -1 : (j == g.dhi[1]) ? 1 : 0;
    const int s2 = (k == g.dlo[2]) ? -1 : (k == g.dhi[2]) ? 1 : 0;
    const int cnt = (s0 != 0) + (s1 != 0) + (s2 != 0);
    if (cnt == 0) return -1;
    const R w = cnt == 3 ? R(AE_SQRT3INV) : cnt == 2 ? R(AE_SQRT2INV) : R(1.0);
    n[0] = s0 == 0 ? R(0) : (s0 > 0 ? w : -w);
    n[1] = s1 == 0 ? R(0) : (s1 > 0 ? w : -w);
    n[2] = s2 == 0 ? R(0) : (s2 > 0 ? w : -w);
    if (cnt == 3) return 18 + 4 * (s0 > 0) + 2 * (s1 > 0) + (s2 > 0);
    if (cnt == 2) {
        if (s0 == 0) return 6 + 2 * (s1 > 0) + (s2 > 0);
        if (s1 == 0) return 10 + 2 * (s2 > 0) + (s0 > 0);
        return 14 + 2 * (s0 > 0) + (s1 > 0);
    }
    if (s0) return s0 < 0 ? 0 : 3;
    if (s1) return s1 < 0 ? 1 : 4;
    return s2 < 0 ? 2 : 5;
}

// ------------------------------------------------------------------ contractions
template <class R>
__device__ __forceinline__ void stress_mm(const R* a, const R g[3][3], R s[3][3]) {
    const R e01 = g[0][1] + g[1][0], e02 = g[0][2] + g[2][0], e12 = g[1][2] + g[2][1];
    const R r00 = a[0] * g[0][0] + a[1] * e01 + a[2] * e02 + a[3] * g[1][1] + a[4] * e12 + a[5] * g[2][2];
    const R r11 = a[3] * g[0][0] + a[8] * e01 + a[12] * e02 + a[15] * g[1][1] + a[16] * e12 + a[17] * g[2][2];
    const R r22 = a[5] * g[0][0] + a[10] * e01 + a[14] * e02 + a[17] * g[1][1] + a[19] * e12 + a[20] * g[2][2];
    const R r12 = a[4] * g[0][0] + a[9] * e01 + a[13] * e02 + a[16] * g[1][1] + a[18] * e12 + a[19] * g[2][2];
    const R r20 = a[2] * g[0][0] + a[7] * e01 + a[11] * e02 + a[12] * g[1][1] + a[13] * e12 + a[14] * g[2][2];
    const R r01 = a[1] * g[0][0] + a[6] * e01 + a[7] * e02 + a[8] * g[1][1] + a[9] * e12 + a[10] * g[2][2];
    s[0][0] = r00; s[1][1] = r11; s[2][2] = r22;
    s[1][2] = r12; s[2][1] = r12;
    s[2][0] = r20; s[0][2] = r20;
    s[0][1] = r01; s[1][0] = r01;
}
template <class R>
__device__ __forceinline__ void stress_iso(const R* a, const R g[3][3], R s[3][3]) {
    const R lambda = a[0], mu = a[1];
    s[0][0] = (lambda + R(2) * mu) * g[0][0] + lambda * g[1][1] + lambda * g[2][2];
    s[1][1] = lambda * g[0][0] + (lambda + R(2) * mu) * g[1][1] + lambda * g[2][2];
    s[2][2] = lambda * g[0][0] + lambda * g[1][1] + (lambda + R(2) * mu) * g[2][2];
    s[1][2] = mu * (g[1][2] + g[2][1]); s[2][1] = s[1][2];
    s[2][0] = mu * (g[2][0] + g[0][2]); s[0][2] = s[2][0];
    s[0][1] = mu * (g[0][1] + g[1][0]); s[1][0] = s[0][1];
}
template <class R>
__device__ __forceinline__ void stress_diag(const R* a, const R g[3][3], R s[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) s[i][j] = a[3 * i + j] * g[i][j];
}
// Matrix4_Major.H:399-413: sigma_ij = sum_kl C_ijkl g_kl, summed in (k, l) order
template <class R>
__device__ __forceinline__ void stress_major(const R* a, const R g[3][3], R s[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            R r = R(0);
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int l = 0; l < 3; ++l) r += a[major_slot(3 * i + j, 3 * k + l)] * g[k][l];
            s[i][j] = r;
        }
}
template <int M, class R>
__device__ __forceinline__ void stress_of(const R* a, const R g[3][3], R s[3][3]) {
    if (M == ISO) stress_iso(a, g, s);
    else if (M == MM) stress_mm(a, g, s);
    else if (M == MAJOR) stress_major(a, g, s);
    else stress_diag(a, g, s);
}

// C_ijkl u_{k,lj} with b[k][l][j] = u_{k,lj}
template <class R>
__device__ __forceinline__ void div_mm(const R* a, const R b[3][3][3], R f[3]) {
#define B(p, q, r) b[p][q][r]
    if constexpr (sizeof(R) == 4) {
        // the same terms in the same order, explicitly rounded
#define S2(x, y) __fadd_rn(x, y)
#define S3(x, y, z) __fadd_rn(__fadd_rn(x, y), z)
#define S4(x, y, z, w) __fadd_rn(__fadd_rn(__fadd_rn(x, y), z), w)
        f[0] = fx_sop(a[0], B(0, 0, 0), a[1], S3(B(0, 1, 0), B(1, 0, 0), B(0, 0, 1)),
                      a[2], S3(B(0, 2, 0), B(2, 0, 0), B(0, 0, 2)), a[3], B(1, 1, 0), a[4], S2(B(1, 2, 0), B(2, 1, 0)),
                      a[5], B(2, 2, 0), a[6], S2(B(0, 1, 1), B(1, 0, 1)),
                      a[7], S4(B(0, 2, 1), B(2, 0, 1), B(0, 1, 2), B(1, 0, 2)), a[8], B(1, 1, 1),
                      a[9], S2(B(1, 2, 1), B(2, 1, 1)), a[10], B(2, 2, 1), a[11], S2(B(0, 2, 2), B(2, 0, 2)),
                      a[12], B(1, 1, 2), a[13], S2(B(1, 2, 2), B(2, 1, 2)), a[14], B(2, 2, 2));
        f[1] = fx_sop(a[1], B(0, 0, 0), a[4], B(0, 0, 2), a[3], B(0, 0, 1), a[6], S2(B(0, 1, 0), B(1, 0, 0)),
                      a[7], S2(B(0, 2, 0), B(2, 0, 0)), a[8], S3(B(1, 1, 0), B(0, 1, 1), B(1, 0, 1)),
                      a[9], S4(B(1, 2, 0), B(2, 1, 0), B(0, 1, 2), B(1, 0, 2)), a[10], B(2, 2, 0),
                      a[12], S2(B(0, 2, 1), B(2, 0, 1)), a[13], S2(B(0, 2, 2), B(2, 0, 2)), a[15], B(1, 1, 1),
                      a[16], S3(B(1, 2, 1), B(2, 1, 1), B(1, 1, 2)), a[17], B(2, 2, 1), a[18], S2(B(1, 2, 2), B(2, 1, 2)),
                      a[19], B(2, 2, 2));
        f[2] = fx_sop(a[2], B(0, 0, 0), a[4], B(0, 0, 1), a[5], B(0, 0, 2), a[7], S2(B(0, 1, 0), B(1, 0, 0)),
                      a[9], S2(B(0, 1, 1), B(1, 0, 1)), a[10], S2(B(0, 1, 2), B(1, 0, 2)),
                      a[11], S2(B(0, 2, 0), B(2, 0, 0)), a[12], B(1, 1, 0),
                      a[13], S4(B(1, 2, 0), B(2, 1, 0), B(0, 2, 1), B(2, 0, 1)),
                      a[14], S3(B(2, 2, 0), B(0, 2, 2), B(2, 0, 2)), a[16], B(1, 1, 1), a[17], B(1, 1, 2),
                      a[18], S2(B(1, 2, 1), B(2, 1, 1)), a[19], S3(B(2, 2, 1), B(1, 2, 2), B(2, 1, 2)), a[20], B(2, 2, 2));
#undef S2
#undef S3
#undef S4
        return;
    }
    f[0] = a[0] * B(0, 0, 0) + a[1] * (B(0, 1, 0) + B(1, 0, 0) + B(0, 0, 1)) +
           a[2] * (B(0, 2, 0) + B(2, 0, 0) + B(0, 0, 2)) + a[3] * B(1, 1, 0) + a[4] * (B(1, 2, 0) + B(2, 1, 0)) +
           a[5] * B(2, 2, 0) + a[6] * (B(0, 1, 1) + B(1, 0, 1)) +
           a[7] * (B(0, 2, 1) + B(2, 0, 1) + B(0, 1, 2) + B(1, 0, 2)) + a[8] * B(1, 1, 1) +
           a[9] * (B(1, 2, 1) + B(2, 1, 1)) + a[10] * B(2, 2, 1) + a[11] * (B(0, 2, 2) + B(2, 0, 2)) +
           a[12] * B(1, 1, 2) + a[13] * (B(1, 2, 2) + B(2, 1, 2)) + a[14] * B(2, 2, 2);
    f[1] = a[1] * B(0, 0, 0) + a[4] * B(0, 0, 2) + a[3] * B(0, 0, 1) + a[6] * (B(0, 1, 0) + B(1, 0, 0)) +
           a[7] * (B(0, 2, 0) + B(2, 0, 0)) + a[8] * (B(1, 1, 0) + B(0, 1, 1) + B(1, 0, 1)) +
           a[9] * (B(1, 2, 0) + B(2, 1, 0) + B(0, 1, 2) + B(1, 0, 2)) + a[10] * B(2, 2, 0) +
           a[12] * (B(0, 2, 1) + B(2, 0, 1)) + a[13] * (B(0, 2, 2) + B(2, 0, 2)) + a[15] * B(1, 1, 1) +
           a[16] * (B(1, 2, 1) + B(2, 1, 1) + B(1, 1, 2)) + a[17] * B(2, 2, 1) + a[18] * (B(1, 2, 2) + B(2, 1, 2)) +
           a[19] * B(2, 2, 2);
    f[2] = a[2] * B(0, 0, 0) + a[4] * B(0, 0, 1) + a[5] * B(0, 0, 2) + a[7] * (B(0, 1, 0) + B(1, 0, 0)) +
           a[9] * (B(0, 1, 1) + B(1, 0, 1)) + a[10] * (B(0, 1, 2) + B(1, 0, 2)) +
           a[11] * (B(0, 2, 0) + B(2, 0, 0)) + a[12] * B(1, 1, 0) +
           a[13] * (B(1, 2, 0) + B(2, 1, 0) + B(0, 2, 1) + B(2, 0, 1)) +
           a[14] * (B(2, 2, 0) + B(0, 2, 2) + B(2, 0, 2)) + a[16] * B(1, 1, 1) + a[17] * B(1, 1, 2) +
           a[18] * (B(1, 2, 1) + B(2, 1, 1)) + a[19] * (B(2, 2, 1) + B(1, 2, 2) + B(2, 1, 2)) + a[20] * B(2, 2, 2);
#undef B
}
template <class R>
__device__ __forceinline__ void div_iso(const R* a, const R b[3][3][3], R f[3]) {
    const R lambda = a[0], mu = a[1];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        R r = R(0);
#pragma unroll
        for (int j = 0; j < 3; ++j) r += mu * (b[i][j][j] + b[j][i][j]) + lambda * b[j][j][i];
        f[i] = r;
    }
}
template <class R>
__device__ __forceinline__ void div_diag(const R* a, const R b[3][3][3], R f[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        R r = R(0);
#pragma unroll
        for (int j = 0; j < 3; ++j) r += a[3 * i + j] * b[i][j][j];
        f[i] = r;
    }
}
// Matrix4_Major.H:415-428: f_i = sum_{j,k,l} C_ijkl b[k][l][j], b[k][l][j] = u_{k,lj}
template <class R>
__device__ __forceinline__ void div_major(const R* a, const R b[3][3][3], R f[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        R r = R(0);
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int l = 0; l < 3; ++l) r += a[major_slot(3 * i + j, 3 * k + l)] * b[k][l][j];
        f[i] = r;
    }
}
template <int M, class R>
__device__ __forceinline__ void div_of(const R* a, const R b[3][3][3], R f[3]) {
    if (M == ISO) div_iso(a, b, f);
    else if (M == MM) div_mm(a, b, f);
    else if (M == MAJOR) div_major(a, b, f);
    else div_diag(a, b, f);
}

// read-only load: through the non-coherent cache for global memory (LDG), plain otherwise
// (stiffness staged in shared memory)
// A Voronoi stiffness on one level: a grain id per node (laid out like the level's stiffness
// view) and a per-grain coefficient table tab[g * ncoef + q].  gid == nullptr: not used.
template <class R>
struct Grains {
    const unsigned short* gid = nullptr;
    const R* tab = nullptr;
};

template <bool LDG, class T>
__device__ __forceinline__ T ldv(const T* p) {
    if constexpr (LDG) return __ldg(p);
    else return *p;
}

// Column d of (dC : grad u), dC the (unscaled) central difference of the stiffness in
// direction d.  Only the slots that feed column d are read: 15 of 21 for MajorMinor.
template <int M, class R, bool LDG = true>
__device__ __forceinline__ void gradC_col(const R* __restrict__ C, long long cs, long long c, long long o,
                                          const R g[3][3], int d, R col[3]) {
#define DC(q) (ldv<LDG>(C + (q) * cs + c + o) - ldv<LDG>(C + (q) * cs + c - o))
    if (M == MM) {
        const R e00 = g[0][0], e11 = g[1][1], e22 = g[2][2];
        const R e01 = add2(g[0][1], g[1][0]), e02 = add2(g[0][2], g[2][0]), e12 = add2(g[1][2], g[2][1]);
        if (d == 0) {  // (s00, s01, s20)
            const R a0 = DC(0), a1 = DC(1), a2 = DC(2), a3 = DC(3), a4 = DC(4), a5 = DC(5), a6 = DC(6), a7 = DC(7);
            const R a8 = DC(8), a9 = DC(9), a10 = DC(10), a11 = DC(11), a12 = DC(12), a13 = DC(13), a14 = DC(14);
            col[0] = sop6(a0, e00, a1, e01, a2, e02, a3, e11, a4, e12, a5, e22);
            col[1] = sop6(a1, e00, a6, e01, a7, e02, a8, e11, a9, e12, a10, e22);
            col[2] = sop6(a2, e00, a7, e01, a11, e02, a12, e11, a13, e12, a14, e22);
        } else if (d == 1) {  // (s01, s11, s12)
            const R a1 = DC(1), a3 = DC(3), a4 = DC(4), a6 = DC(6), a7 = DC(7), a8 = DC(8), a9 = DC(9), a10 = DC(10);
            const R a12 = DC(12), a13 = DC(13), a15 = DC(15), a16 = DC(16), a17 = DC(17), a18 = DC(18), a19 = DC(19);
            col[0] = sop6(a1, e00, a6, e01, a7, e02, a8, e11, a9, e12, a10, e22);
            col[1] = sop6(a3, e00, a8, e01, a12, e02, a15, e11, a16, e12, a17, e22);
            col[2] = sop6(a4, e00, a9, e01, a13, e02, a16, e11, a18, e12, a19, e22);
        } else {  // (s20, s12, s22)
            const R a2 = DC(2), a4 = DC(4), a5 = DC(5), a7 = DC(7), a9 = DC(9), a10 = DC(10), a11 = DC(11), a12 = DC(12);
            const R a13 = DC(13), a14 = DC(14), a16 = DC(16), a17 = DC(17), a18 = DC(18), a19 = DC(19), a20 = DC(20);
            col[0] = sop6(a2, e00, a7, e01, a11, e02, a12, e11, a13, e12, a14, e22);
            col[1] = sop6(a4, e00, a9, e01, a13, e02, a16, e11, a18, e12, a19, e22);
            col[2] = sop6(a5, e00, a10, e01, a14, e02, a17, e11, a19, e12, a20, e22);
        }
    } else if (M == MAJOR) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            R v = R(0);
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int l = 0; l < 3; ++l) v = fma_rn(DC(major_slot(3 * r + d, 3 * k + l)), g[k][l], v);
            col[r] = v;
        }
    } else if (M == ISO) {
        const R dl = DC(0), dm = DC(1);
        const R tr = mul_rn(dl, add_rn(add_rn(g[0][0], g[1][1]), g[2][2])), dm2 = add_rn(dm, dm);
        const R s01 = mul_rn(dm, add_rn(g[0][1], g[1][0])), s02 = mul_rn(dm, add_rn(g[2][0], g[0][2]));
        const R s12 = mul_rn(dm, add_rn(g[1][2], g[2][1]));
        col[0] = d == 0 ? fma_rn(dm2, g[0][0], tr) : d == 1 ? s01 : s02;
        col[1] = d == 0 ? s01 : d == 1 ? fma_rn(dm2, g[1][1], tr) : s12;
        col[2] = d == 0 ? s02 : d == 1 ? s12 : fma_rn(dm2, g[2][2], tr);
    } else {
#pragma unroll
        for (int r = 0; r < 3; ++r) col[r] = mul_rn(DC(3 * r + d), g[r][d]);
    }
#undef DC
}

// Column d of (dC : grad u) with the slot differences supplied by a callable dC(q); the same
// 15-of-21 slot selection as gradC_col.
template <int M, class R, class F>
__device__ __forceinline__ void gradC_col_f(F&& dC, const R g[3][3], int d, R col[3]) {
    if (M == MM) {
        const R e00 = g[0][0], e11 = g[1][1], e22 = g[2][2];
        const R e01 = add2(g[0][1], g[1][0]), e02 = add2(g[0][2], g[2][0]), e12 = add2(g[1][2], g[2][1]);
        if (d == 0) {
            const R a0 = dC(0), a1 = dC(1), a2 = dC(2), a3 = dC(3), a4 = dC(4), a5 = dC(5), a6 = dC(6), a7 = dC(7);
            const R a8 = dC(8), a9 = dC(9), a10 = dC(10), a11 = dC(11), a12 = dC(12), a13 = dC(13), a14 = dC(14);
            col[0] = sop6(a0, e00, a1, e01, a2, e02, a3, e11, a4, e12, a5, e22);
            col[1] = sop6(a1, e00, a6, e01, a7, e02, a8, e11, a9, e12, a10, e22);
            col[2] = sop6(a2, e00, a7, e01, a11, e02, a12, e11, a13, e12, a14, e22);
        } else if (d == 1) {
            const R a1 = dC(1), a3 = dC(3), a4 = dC(4), a6 = dC(6), a7 = dC(7), a8 = dC(8), a9 = dC(9), a10 = dC(10);
            const R a12 = dC(12), a13 = dC(13), a15 = dC(15), a16 = dC(16), a17 = dC(17), a18 = dC(18), a19 = dC(19);
            col[0] = sop6(a1, e00, a6, e01, a7, e02, a8, e11, a9, e12, a10, e22);
            col[1] = sop6(a3, e00, a8, e01, a12, e02, a15, e11, a16, e12, a17, e22);
            col[2] = sop6(a4, e00, a9, e01, a13, e02, a16, e11, a18, e12, a19, e22);
        } else {
            const R a2 = dC(2), a4 = dC(4), a5 = dC(5), a7 = dC(7), a9 = dC(9), a10 = dC(10), a11 = dC(11), a12 = dC(12);
            const R a13 = dC(13), a14 = dC(14), a16 = dC(16), a17 = dC(17), a18 = dC(18), a19 = dC(19), a20 = dC(20);
            col[0] = sop6(a2, e00, a7, e01, a11, e02, a12, e11, a13, e12, a14, e22);
            col[1] = sop6(a4, e00, a9, e01, a13, e02, a16, e11, a18, e12, a19, e22);
            col[2] = sop6(a5, e00, a10, e01, a14, e02, a17, e11, a19, e12, a20, e22);
        }
    } else if (M == MAJOR) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            R v = R(0);
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int l = 0; l < 3; ++l) v = fma_rn(dC(major_slot(3 * r + d, 3 * k + l)), g[k][l], v);
            col[r] = v;
        }
    } else if (M == ISO) {
        const R dl = dC(0), dm = dC(1);
        const R tr = mul_rn(dl, add_rn(add_rn(g[0][0], g[1][1]), g[2][2])), dm2 = add_rn(dm, dm);
        const R s01 = mul_rn(dm, add_rn(g[0][1], g[1][0])), s02 = mul_rn(dm, add_rn(g[2][0], g[0][2]));
        const R s12 = mul_rn(dm, add_rn(g[1][2], g[2][1]));
        col[0] = d == 0 ? fma_rn(dm2, g[0][0], tr) : d == 1 ? s01 : s02;
        col[1] = d == 0 ? s01 : d == 1 ? fma_rn(dm2, g[1][1], tr) : s12;
        col[2] = d == 0 ? s02 : d == 1 ? s12 : fma_rn(dm2, g[2][2], tr);
    } else {
#pragma unroll
        for (int r = 0; r < 3; ++r) col[r] = mul_rn(dC(3 * r + d), g[r][d]);
    }
}

// Slots that the z column of the grad C term reads (gradC_col, d = 2), in order.
template <int M> struct ZSlots;
template <> struct ZSlots<MM> {
    static constexpr int n = 15;
    __device__ static constexpr int at(int s) {
        return s < 1 ? 2 : s < 2 ? 4 : s < 3 ? 5 : s < 4 ? 7 : s < 5 ? 9 : s < 6 ? 10 : s < 7 ? 11 : s < 8 ? 12
             : s < 9 ? 13 : s < 10 ? 14 : s < 11 ? 16 : s < 12 ? 17 : s < 13 ? 18 : s < 14 ? 19 : 20;
    }
};
template <> struct ZSlots<ISO> {
    static constexpr int n = 2;
    __device__ static constexpr int at(int s) { return s; }
};
template <> struct ZSlots<DIAG> {
    static constexpr int n = 3;
    __device__ static constexpr int at(int s) { return 3 * s + 2; }
};

// position of slot q in the ZSlots list (-1 if absent)
template <int M>
__device__ __forceinline__ constexpr int zslot_index(int q) {
    for (int s = 0; s < ZSlots<M>::n; ++s)
        if (ZSlots<M>::at(s) == q) return s;
    return -1;
}

// ------------------------------------------------------------------ the interior row
// C : grad grad u + sum_d (d_d C : grad u) e_d, written to take few operations (GB300 issues FP64 at
// 1/64 of its FP32 rate, so the FP64 sweeps are bound by their number):
//   - differences are not scaled one by one: a row is i2[0] times a sum over the unscaled differences
//     (with unequal spacing scaled by ratios of the spacings), the mixed ones times 1/4;
//   - the products run over the differences, not over the slots: row i is the sum over k and the six
//     (l, j) of A_ik,lj u_k,lj with A_ik,lj = C_ijkl + C_ilkj for l != j, C_ilkl for l = j, which is
//     symmetric in i and k (36 numbers, from a table for a grain map).
// MajorMinor: 45 + 60 FP64 operations a node on a grain map, against 154 before; the difference of a
// pair comes first, so a smooth field's differences are exact.  FP32 keeps div_of over scaled
// differences: it is not bound by operations, and reads 21 coefficients a node instead of 36.
enum { kXX = 0, kYY = 1, kZZ = 2, kXY = 3, kXZ = 4, kYZ = 5 };

// D: the six second differences of each component, g: its three central differences, from
// u(p, di, dj, dk)
template <class R, class U>
__device__ __forceinline__ void row_diffs(const SCoef<R>&, U&& u, R D[3][6], R g[3][3]) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const R c = u(p, 0, 0, 0);
        const R xm = u(p, -1, 0, 0), xp = u(p, 1, 0, 0), ym = u(p, 0, -1, 0), yp = u(p, 0, 1, 0), zm = u(p, 0, 0, -1),
                zp = u(p, 0, 0, 1);
        g[p][0] = sub_rn(xp, xm);
        g[p][1] = sub_rn(yp, ym);
        g[p][2] = sub_rn(zp, zm);
        D[p][kXX] = add_rn(fma_rn(R(-2), c, xp), xm);
        D[p][kYY] = add_rn(fma_rn(R(-2), c, yp), ym);
        D[p][kZZ] = add_rn(fma_rn(R(-2), c, zp), zm);
        D[p][kXY] = sub_rn(sub_rn(u(p, 1, 1, 0), u(p, 1, -1, 0)), sub_rn(u(p, -1, 1, 0), u(p, -1, -1, 0)));
        D[p][kXZ] = sub_rn(sub_rn(u(p, 1, 0, 1), u(p, -1, 0, 1)), sub_rn(u(p, 1, 0, -1), u(p, -1, 0, -1)));
        D[p][kYZ] = sub_rn(sub_rn(u(p, 0, 1, 1), u(p, 0, -1, 1)), sub_rn(u(p, 0, 1, -1), u(p, 0, -1, -1)));
    }
}
template <class R>
__device__ __forceinline__ void row_scale(const SCoef<R>& K, R D[3][6]) {
    if (K.iso) return;
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int s = 1; s < 6; ++s) D[p][s] = mul_rn(D[p][s], K.sd[s]);
}
// the central difference along d that row_interior hands on, from the two neighbours
template <class R>
__device__ __forceinline__ R node_diff(const SCoef<R>& K, int d, R p, R m) {
    if constexpr (sizeof(R) == 8) return sub_rn(p, m);
    else return (p - m) * K.h[d];
}
// (FP64: row_interior's FP32 differences are scaled already)
template <class R>
__device__ __forceinline__ void grad_scale(const SCoef<R>& K, R g[3][3]) {
    if (sizeof(R) == 4 || K.iso) return;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        g[p][1] = mul_rn(g[p][1], K.q[1]);
        g[p][2] = mul_rn(g[p][2], K.q[2]);
    }
}

// (written without recursion, so that unrolled loops see constants)
__host__ __device__ constexpr int pair_index(int i, int j) {
    return (i < j ? i : j) == 0 ? (i < j ? j : i) : i + j + 1;
}
__host__ __device__ constexpr int pair_slot(int p, int q) {
    return (p < q ? p : q) * 6 - (p < q ? p : q) * ((p < q ? p : q) - 1) / 2 + (p < q ? q : p) - (p < q ? p : q);
}
__host__ __device__ constexpr int mm_slot(int i, int j, int k, int l) {
    return pair_slot(pair_index(i, j), pair_index(k, l));
}
static_assert(pair_index(1, 1) == 3 && pair_index(2, 1) == 4 && pair_index(2, 2) == 5 && mm_slot(2, 2, 2, 2) == 20 &&
                  mm_slot(1, 0, 2, 1) == 9 && mm_slot(1, 2, 0, 0) == 4,
              "slot order of Matrix4<3, MajorMinor>");
template <int M>
__host__ __device__ constexpr int slot_of(int i, int j, int k, int l) {
    return M == MAJOR ? major_slot(3 * i + j, 3 * k + l) : mm_slot(i, j, k, l);
}
__host__ __device__ constexpr int ik_row(int n) { return n < 3 ? 0 : n < 5 ? 1 : 2; }
__host__ __device__ constexpr int ik_col(int n) { return n < 3 ? n : n < 5 ? n - 2 : 2; }
__host__ __device__ constexpr int diff_a(int s) { return s < 3 ? s : s < 5 ? 0 : 1; }
__host__ __device__ constexpr int diff_b(int s) { return s < 3 ? s : s == 3 ? 1 : 2; }
// coefficient 6 n + s of a row: n the pair (i, k) in the order 00 01 02 11 12 22, s the difference;
// a(q): slot q of the stiffness
template <int M, class A>
__device__ __forceinline__ auto row_coef(A&& a, int n, int s) {
    const int i = ik_row(n), k = ik_col(n), l = diff_a(s), j = diff_b(s);
    const auto c = a(slot_of<M>(i, j, k, l));
    return l == j ? c : add_rn(c, a(slot_of<M>(i, l, k, j)));
}

// numbers a row takes per node or grain: the 36 sums (MajorMinor, Major), or the slots themselves
template <int M> struct RowN { static constexpr int value = 36; };
template <> struct RowN<ISO> { static constexpr int value = 2; };
template <> struct RowN<DIAG> { static constexpr int value = 9; };

// F / i2[0] of the interior term from the differences; r(n): number n of the row
template <int M, class A>
__device__ __forceinline__ void row_sum(A&& r, const double D[3][6], double F[3]) {
    if constexpr (M == ISO) {
        const double lam = r(0), mu = r(1), lm = add_rn(lam, mu);
        const double g0 = fma_rn(0.25, add_rn(D[1][kXY], D[2][kXZ]), D[0][kXX]);
        const double g1 = fma_rn(0.25, add_rn(D[0][kXY], D[2][kYZ]), D[1][kYY]);
        const double g2 = fma_rn(0.25, add_rn(D[0][kXZ], D[1][kYZ]), D[2][kZZ]);
        const double g[3] = {g0, g1, g2};
#pragma unroll
        for (int i = 0; i < 3; ++i)
            F[i] = fma_rn(mu, add_rn(add_rn(D[i][kXX], D[i][kYY]), D[i][kZZ]), mul_rn(lm, g[i]));
    } else if constexpr (M == DIAG) {
#pragma unroll
        for (int i = 0; i < 3; ++i) F[i] = fx_sop(r(3 * i), D[i][kXX], r(3 * i + 1), D[i][kYY], r(3 * i + 2), D[i][kZZ]);
    } else {
        // the mixed differences in a sum of their own, which takes the 1/4
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            double fd, fm;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int n = 6 * pair_index(i, k);
                fd = k == 0 ? mul_rn(r(n), D[k][0]) : fma_rn(r(n), D[k][0], fd);
                fd = fma_rn(r(n + 1), D[k][1], fd);
                fd = fma_rn(r(n + 2), D[k][2], fd);
                fm = k == 0 ? mul_rn(r(n + 3), D[k][3]) : fma_rn(r(n + 3), D[k][3], fm);
                fm = fma_rn(r(n + 4), D[k][4], fm);
                fm = fma_rn(r(n + 5), D[k][5], fm);
            }
            F[i] = fma_rn(0.25, fm, fd);
        }
    }
}
// number n of the row from the slots a(q)
template <int M, class A>
__device__ __forceinline__ auto row_number(A&& a, int n) {
    if constexpr (M == ISO || M == DIAG) return a(n);
    else return row_coef<M>(a, n / 6, n % 6);
}
// b - scale f and scale f, for the f and the factor that apply_node returns
template <class R>
__device__ __forceinline__ R row_residual(R b, R scale, R f) { return fma_rn(-scale, f, b); }
// The interior term of a node and its central differences for the grad C term: FP64 as above (a row
// over i2[0]), FP32 from the scaled differences (factor 1).  u(p, di, dj, dk); slot(q) loads a
// coefficient (after the differences: loaded first, FP32 Fapply took 0.129 ms at 129^3, not 0.097).
template <int M, class R, class U, class A>
__device__ __forceinline__ void row_interior(const SCoef<R>& K, U&& u, A&& slot, R gu[3][3], R f[3]) {
    constexpr int NC = NCoef<M>::value;
    R a[NC];
    if constexpr (sizeof(R) == 8) {
        R D[3][6];
        row_diffs<R>(K, u, D, gu);
        row_scale(K, D);
#pragma unroll
        for (int q = 0; q < NC; ++q) a[q] = slot(q);
        row_sum<M>([&](int n) { return row_number<M>([&](int q) { return a[q]; }, n); }, D, f);
    } else {
        R b[3][3][3];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const R c0 = u(p, 0, 0, 0);
            const R xm = u(p, -1, 0, 0), xp = u(p, 1, 0, 0), ym = u(p, 0, -1, 0), yp = u(p, 0, 1, 0),
                    zm = u(p, 0, 0, -1), zp = u(p, 0, 0, 1);
            gu[p][0] = (xp - xm) * K.h[0];
            gu[p][1] = (yp - ym) * K.h[1];
            gu[p][2] = (zp - zm) * K.h[2];
            b[p][0][0] = (xp - R(2) * c0 + xm) * K.i2[0];
            b[p][1][1] = (yp - R(2) * c0 + ym) * K.i2[1];
            b[p][2][2] = (zp - R(2) * c0 + zm) * K.i2[2];
            b[p][0][1] = (u(p, 1, 1, 0) + u(p, -1, -1, 0) - u(p, 1, -1, 0) - u(p, -1, 1, 0)) * K.m01;
            b[p][0][2] = (u(p, 1, 0, 1) + u(p, -1, 0, -1) - u(p, 1, 0, -1) - u(p, -1, 0, 1)) * K.m02;
            b[p][1][2] = (u(p, 0, 1, 1) + u(p, 0, -1, -1) - u(p, 0, 1, -1) - u(p, 0, -1, 1)) * K.m12;
            b[p][1][0] = b[p][0][1];
            b[p][2][0] = b[p][0][2];
            b[p][2][1] = b[p][1][2];
        }
#pragma unroll
        for (int q = 0; q < NC; ++q) a[q] = slot(q);
        div_of<M, R>(a, b, f);
    }
}
// the factor of the interior rows of row_interior
template <class R>
__device__ __forceinline__ R row_factor(const SCoef<R>& K) {
    if constexpr (sizeof(R) == 8) return K.i2[0];
    else return R(1);
}
// f plus its grad C columns (from row_interior's central differences)
template <class R>
__device__ __forceinline__ R row_gradc(const SCoef<R>& K, R f, R c0, R c1, R c2) {
    if constexpr (sizeof(R) == 8) return fma_rn(0.25, fma_rn(c2, K.q[2], fma_rn(c1, K.q[1], c0)), f);
    else return gradc_add(f, c0, c1, c2, K.h);
}

// ------------------------------------------------------------------ the operator at one node
// f = A u at node (i,j,k): boundary rows through the BC table, interior rows
// C : grad grad u + sum_d (d_d C : grad u) e_d  (src/Operator/Elastic.cpp:174-258).
// u and C are read through views whose strides may differ.  LDG = false when C lives in
// shared memory.  Returns the factor that A u is f times: row_factor on interior rows, 1 on boundary
// rows (b - A u is then one fused operation a component, row_residual).  IN: the node is known to be
// inside the domain's boundary.
template <int M, class R, bool LDG = true, bool IN = false>
__device__ __forceinline__ R apply_node(const Geo& g, const SCoef<R>& K, const BCP& bc, bool uniform,
                                           const R* __restrict__ C, long long cs, long long cc,
                                           long long csy, long long csz, const R* __restrict__ U,
                                           long long usc, long long uc, long long usy, long long usz, int i, int j,
                                           int k, R f[3]) {
    constexpr int NC = NCoef<M>::value;
    R nrm[3];
    const int face = IN ? -1 : classify<R>(g, i, j, k, nrm);
    if (face >= 0) {
        // one-sided first derivatives: Hi stencil on the lo face, Lo on the hi face
        const int ci[3] = {i, j, k};
        const long long os[3] = {1, usy, usz};
        R gu[3][3], u[3];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const R* up = U + p * usc + uc;
            u[p] = up[0];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const long long o = os[d];
                if (ci[d] == g.dlo[d]) gu[p][d] = (up[o] - up[0]) * K.id[d];
                else if (ci[d] == g.dhi[d]) gu[p][d] = (up[0] - up[-o]) * K.id[d];
                else gu[p][d] = (up[o] - up[-o]) * K.h[d];
            }
        }
        const unsigned char* t = bc.t[face];
        R s[3][3];
        bool need_s = (t[0] == TRAC) || (t[1] == TRAC) || (t[2] == TRAC);
        if (need_s) {
            R a[NC];
#pragma unroll
            for (int q = 0; q < NC; ++q) a[q] = ldv<LDG>(C + q * cs + cc);
            stress_of<M, R>(a, gu, s);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            R v = R(0);
            if (t[r] == DISP) v = u[r];
            else if (t[r] == TRAC) v = s[r][0] * nrm[0] + s[r][1] * nrm[1] + s[r][2] * nrm[2];
            else if (t[r] == NEUMANN) v = gu[r][0] * nrm[0] + gu[r][1] * nrm[1] + gu[r][2] * nrm[2];
            f[r] = v;
        }
        return R(1);
    }
    R gu[3][3];
    row_interior<M, R>(K, [&](int p, int di, int dj, int dk) { return U[p * usc + uc + di + dj * usy + dk * usz]; },
                       [&](int q) { return ldv<LDG>(C + q * cs + cc); }, gu, f);
    if (!uniform) {
        R c0[3], c1[3], c2[3];
        grad_scale(K, gu);
        gradC_col<M, R, LDG>(C, cs, cc, 1, gu, 0, c0);
        gradC_col<M, R, LDG>(C, cs, cc, csy, gu, 1, c1);
        gradC_col<M, R, LDG>(C, cs, cc, csz, gu, 2, c2);
#pragma unroll
        for (int r = 0; r < 3; ++r) f[r] = row_gradc(K, f[r], c0[r], c1[r], c2[r]);
    }
    return row_factor(K);
}

// apply_node for a stiffness given as a grain id per node (gid, strides gsy, gsz, node index gc)
// and a per-grain coefficient table (tab[g * ncoef + q]): the same arithmetic on the same values.
// A direction whose two neighbours lie in one grain has an exactly zero stiffness difference; its
// grad C column is zero and its table reads are skipped.
template <int M, class R, bool IN = false>
__device__ __forceinline__ R apply_node_grains(const Geo& g, const SCoef<R>& K, const BCP& bc, bool uniform,
                                                  const unsigned short* __restrict__ gid, long long gc,
                                                  long long gsy, long long gsz, const R* __restrict__ tab,
                                                  const R* __restrict__ U, long long usc, long long uc, long long usy,
                                                  long long usz, int i, int j, int k, R f[3]) {
    constexpr int NC = NCoef<M>::value;
    const R* a0 = tab + (int)__ldg(gid + gc) * NC;
    R nrm[3];
    const int face = IN ? -1 : classify<R>(g, i, j, k, nrm);
    if (face >= 0) {
        const int ci[3] = {i, j, k};
        const long long os[3] = {1, usy, usz};
        R gu[3][3], u[3];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const R* up = U + p * usc + uc;
            u[p] = up[0];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const long long o = os[d];
                if (ci[d] == g.dlo[d]) gu[p][d] = (up[o] - up[0]) * K.id[d];
                else if (ci[d] == g.dhi[d]) gu[p][d] = (up[0] - up[-o]) * K.id[d];
                else gu[p][d] = (up[o] - up[-o]) * K.h[d];
            }
        }
        const unsigned char* t = bc.t[face];
        R s[3][3];
        bool need_s = (t[0] == TRAC) || (t[1] == TRAC) || (t[2] == TRAC);
        if (need_s) {
            R a[NC];
#pragma unroll
            for (int q = 0; q < NC; ++q) a[q] = __ldg(a0 + q);
            stress_of<M, R>(a, gu, s);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            R v = R(0);
            if (t[r] == DISP) v = u[r];
            else if (t[r] == TRAC) v = s[r][0] * nrm[0] + s[r][1] * nrm[1] + s[r][2] * nrm[2];
            else if (t[r] == NEUMANN) v = gu[r][0] * nrm[0] + gu[r][1] * nrm[1] + gu[r][2] * nrm[2];
            f[r] = v;
        }
        return R(1);
    }
    R gu[3][3];
    row_interior<M, R>(K, [&](int p, int di, int dj, int dk) { return U[p * usc + uc + di + dj * usy + dk * usz]; },
                       [&](int q) { return __ldg(a0 + q); }, gu, f);
    if (!uniform) {
        const long long go[3] = {1, gsy, gsz};
        int gp[3], gm[3];
        bool any = false;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            gp[d] = __ldg(gid + gc + go[d]);
            gm[d] = __ldg(gid + gc - go[d]);
            any = any || gp[d] != gm[d];
        }
        if (any) {
            R col[3][3];
            grad_scale(K, gu);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (gp[d] == gm[d]) {
                    col[d][0] = col[d][1] = col[d][2] = R(0);
                } else {
                    const R* cp = tab + gp[d] * NC;
                    const R* cm = tab + gm[d] * NC;
                    gradC_col_f<M, R>([&](int q) { return __ldg(cp + q) - __ldg(cm + q); }, gu, d, col[d]);
                }
            }
#pragma unroll
            for (int r = 0; r < 3; ++r) f[r] = row_gradc(K, f[r], col[0][r], col[1][r], col[2][r]);
        }
    }
    return row_factor(K);
}

}  // namespace ae
