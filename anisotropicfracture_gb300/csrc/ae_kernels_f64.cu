// FP64 instantiation of the operator kernels, plus the FP64-only kernels: boundary
// values, post-processing fields and the single-CTA bottom solver.
#include <type_traits>

#include "ae_bottom_ell.h"
#include "ae_div.h"
#include "ae_kernels.cuh"
#include "ae_krylov.cuh"

#define AE_REAL double
#include "ae_kernels_common.inc"
#undef AE_REAL

namespace ae {

std::atomic<long long> g_kernel_launches{0};

AE_INST_COPY(double, double)
AE_INST_COPY(double, float)

// ------------------------------------------------------------------ BC::Operator::Elastic::Init
// src/BC/Operator/Elastic.H:106-181: boundary values into the rhs on every domain-boundary node.
struct BCVal {
    double v[26][3];
};
__global__ void __launch_bounds__(kBlock) k_bc_init(Geo g, BCP bc, BCVal val, int homogeneous, Reg reg,
                                                    View<double> rhs) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    double n[3];
    const int face = classify<double>(g, i, j, k, n);
    if (face < 0) return;
    const long long o = rhs.at(i, j, k);
    for (int dir = 0; dir < 3; ++dir)
        rhs.p[o + dir * rhs.sc] = (homogeneous && bc.t[face][dir] == DISP) ? 0.0 : val.v[face][dir];
}
void launch_bc_init(const Geo& g, const BCP& bc, const double* val, int homogeneous, View<double> rhs,
                    cudaStream_t st) {
    const Box3 region = box_isect(box_grow(geo_valid(g), g.ng < 2 ? g.ng : 2), geo_domain(g));
    const Reg reg = make_reg(region);
    if (reg.n == 0) return;
    BCVal v;
    for (int f = 0; f < 26; ++f)
        for (int d = 0; d < 3; ++d) v.v[f][d] = val[3 * f + d];
    k_bc_init<<<nblocks(reg.n), kBlock, 0, st>>>(g, bc, v, homogeneous, reg, rhs);
    launched();
}

// ------------------------------------------------------------------ Voronoi stiffness
__global__ void __launch_bounds__(kBlock) k_grains_box(Reg reg, View<const int> ids, View<unsigned short> gid,
                                                       View<double> C, const double* __restrict__ tab, int ng, int nc,
                                                       int* bad) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    const int id = ids.p[ids.at(i, j, k)];
    if (id < 0 || id >= ng) {
        atomicExch(bad, 1);
        return;
    }
    gid.p[gid.at(i, j, k)] = (unsigned short)id;
    const long long o = C.at(i, j, k);
    for (int q = 0; q < nc; ++q) C.p[o + q * C.sc] = tab[id * nc + q];
}
__global__ void k_to_float(const double* __restrict__ a, float* __restrict__ b, int n) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) b[t] = (float)a[t];
}
void launch_grains_box(const Box3& region, View<const int> ids, View<unsigned short> gid, View<double> C,
                       const double* tab, int ng, int nc, float* tab32, int* bad, cudaStream_t st) {
    const Reg reg = make_reg(region);
    if (reg.n > 0) {
        k_grains_box<<<nblocks(reg.n), kBlock, 0, st>>>(reg, ids, gid, C, tab, ng, nc, bad);
        launched();
    }
    k_to_float<<<(ng * nc + 255) / 256, 256, 0, st>>>(tab, tab32, ng * nc);
    launched();
}

// ------------------------------------------------------------------ stiffness from order parameters
// Phase-field mixture, src/Integrator/PhaseFieldMicrostructure.cpp:531-539 with
// Affine::Cubic::Combine (src/Model/Solid/Affine/Cubic.H:70-82): the weight of phase n at a node
// is its mean over the four cells (i-1..i, j-1..j) of cell layer k, divided by the sum of those
// means; stiffness slots and eigenstrain are the weighted sums of the per-phase tables.
// NP: the number of phases, 0 for more than kMixPhases.  Bound by FP64 operations: the means are kept
// instead of formed twice, and the weights are one division and three operations each (the product with
// the reciprocal corrected by its remainder) instead of a division each.  129^3 nodes, three phases with
// eigenstrains: 0.52 -> 0.475 ms.
constexpr int kMixPhases = 6;
template <int NC, int NP>
__global__ void __launch_bounds__(kBlock) k_model_mixture(Reg reg, View<const double> eta, int np_,
                                                          const double* __restrict__ tab,
                                                          const double* __restrict__ f0tab, View<double> C,
                                                          View<double> F0, int* bad) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    const int np = NP ? NP : np_;
    const long long o00 = eta.at(i, j, k), o01 = eta.at(i, j - 1, k);
    const long long o10 = eta.at(i - 1, j, k), o11 = eta.at(i - 1, j - 1, k);
    const auto mean = [&](int n) {
        const double* e = eta.p + n * eta.sc;
        return 0.25 * (e[o00] + e[o01] + e[o10] + e[o11]);
    };
    double sum = 0.0, m[NP ? NP : 1];
#pragma unroll
    for (int n = 0; n < np; ++n) {
        const double v = mean(n);
        if (NP) m[NP ? n : 0] = v;
        sum += v;
    }
    if (sum == 0.0 || isnan(sum)) {
        atomicExch(bad, 1);
        return;
    }
    const double inv = 1.0 / sum;
    double acc[NC], f[9];
    for (int q = 0; q < NC; ++q) acc[q] = 0.0;
    for (int r = 0; r < 9; ++r) f[r] = 0.0;
#pragma unroll
    for (int n = 0; n < np; ++n) {
        const double w = div_by(NP ? m[NP ? n : 0] : mean(n), sum, inv);
#pragma unroll
        for (int q = 0; q < NC; ++q) acc[q] += __ldg(tab + n * NC + q) * w;
        if (F0.p)
#pragma unroll
            for (int r = 0; r < 9; ++r) f[r] += __ldg(f0tab + n * 9 + r) * w;
    }
    const long long o = C.at(i, j, k);
#pragma unroll
    for (int q = 0; q < NC; ++q) C.p[o + q * C.sc] = acc[q];
    if (F0.p) {
        const long long of = F0.at(i, j, k);
#pragma unroll
        for (int r = 0; r < 9; ++r) F0.p[of + r * F0.sc] = f[r];
    }
}
template <int NC>
void mixture_nc(const Reg& reg, View<const double> eta, int np, const double* tab, const double* f0tab, View<double> C,
                View<double> F0, int* bad, cudaStream_t st) {
    const auto go = [&](auto n) {
        k_model_mixture<NC, decltype(n)::value><<<nblocks(reg.n), kBlock, 0, st>>>(reg, eta, np, tab, f0tab, C, F0, bad);
    };
    switch (np) {
        case 1: go(std::integral_constant<int, 1>()); break;
        case 2: go(std::integral_constant<int, 2>()); break;
        case 3: go(std::integral_constant<int, 3>()); break;
        case 4: go(std::integral_constant<int, 4>()); break;
        case 5: go(std::integral_constant<int, 5>()); break;
        case kMixPhases: go(std::integral_constant<int, kMixPhases>()); break;
        default: go(std::integral_constant<int, 0>());
    }
}
void launch_model_mixture(const Box3& region, int nc, View<const double> eta, int np, const double* tab,
                          const double* f0tab, View<double> C, View<double> F0, int* bad, cudaStream_t st) {
    const Reg reg = make_reg(region);
    if (reg.n == 0) return;
    if (nc == 2) mixture_nc<2>(reg, eta, np, tab, f0tab, C, F0, bad, st);
    else if (nc == 9) mixture_nc<9>(reg, eta, np, tab, f0tab, C, F0, bad, st);
    else mixture_nc<21>(reg, eta, np, tab, f0tab, C, F0, bad, st);
    launched();
}

// Isotropic degradation, src/Integrator/PolymerDegradation.cpp:794-833 with
// Degradable::Isotropic::DegradeModulus (src/Model/Solid/LinearElastic/Degradable/Isotropic.H:74-81):
// every node starts undamaged; each valid node takes (lambda0 (1 - e), mu0 (1 - e)) with e the
// mean of an order parameter over the 8 cells around the node.  Each component is averaged and
// range-checked in turn and the last one is kept, as the reference's loop over components does.
__global__ void __launch_bounds__(kBlock) k_model_degraded(Reg reg, Box3 valid, View<const double> eta, int neta,
                                                           double lam0, double mu0, View<double> C, int* bad) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    double lam = lam0, mu = mu0;
    const bool in_valid = i >= valid.lo[0] && i <= valid.hi[0] && j >= valid.lo[1] && j <= valid.hi[1] &&
                          k >= valid.lo[2] && k <= valid.hi[2];
    if (in_valid && neta > 0) {
        const long long c000 = eta.at(i, j, k), c100 = eta.at(i - 1, j, k);
        const long long c010 = eta.at(i, j - 1, k), c110 = eta.at(i - 1, j - 1, k);
        const long long c001 = eta.at(i, j, k - 1), c101 = eta.at(i - 1, j, k - 1);
        const long long c011 = eta.at(i, j - 1, k - 1), c111 = eta.at(i - 1, j - 1, k - 1);
        double e = 0.0;
        for (int n = 0; n < neta; ++n) {
            const double* p = eta.p + n * eta.sc;
            e = 0.125 * (p[c000] + p[c100] + p[c010] + p[c110] + p[c001] + p[c101] + p[c011] + p[c111]);
            if (!(e >= 0.0 && e <= 1.0)) {
                atomicExch(bad, 1);
                return;
            }
        }
        lam = lam0 * (1.0 - e);
        mu = mu0 * (1.0 - e);
    }
    const long long o = C.at(i, j, k);
    C.p[o] = lam;
    C.p[o + C.sc] = mu;
}
void launch_model_degraded(const Box3& region, const Box3& valid, View<const double> eta, int neta, double lam0,
                           double mu0, View<double> C, int* bad, cudaStream_t st) {
    const Reg reg = make_reg(region);
    if (reg.n == 0) return;
    k_model_degraded<<<nblocks(reg.n), kBlock, 0, st>>>(reg, valid, eta, neta, lam0, mu0, C, bad);
    launched();
}

// ------------------------------------------------------------------ Strain / Stress / Energy
// src/Operator/Elastic.cpp:399-572 (valid box, boundary-aware first derivatives).  inside: no face of
// the domain at this node.
__device__ __forceinline__ void grad_at(const Geo& g, const SCoef<double>& K, const View<const double>& u, int i,
                                        int j, int k, double gu[3][3], bool inside = false) {
    const int ci[3] = {i, j, k};
    const long long os[3] = {1, u.sy, u.sz};
    const long long o = u.at(i, j, k);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const double* up = u.p + o + p * u.sc;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const long long s = os[d];
            if (inside) gu[p][d] = (up[s] - up[-s]) * K.h[d];
            else if (ci[d] == g.dlo[d]) gu[p][d] = (up[s] - up[0]) * K.id[d];
            else if (ci[d] == g.dhi[d]) gu[p][d] = (up[0] - up[-s]) * K.id[d];
            else gu[p][d] = (up[s] - up[-s]) * K.h[d];
        }
    }
}
// valid nodes, those off the domain's boundary apart
inline Parts post_parts(const Geo& g) {
    Box3 in = geo_domain(g);
    for (int q = 0; q < 3; ++q) { in.lo[q] += 1; in.hi[q] -= 1; }
    return make_parts(box_isect(geo_valid(g), geo_domain(g)), in);
}
__global__ void __launch_bounds__(kBlock) k_strain(Geo g, SCoef<double> K, Parts parts, View<const double> u,
                                                   View<double> e, int voigt) {
    const bool inside = blockIdx.x >= parts.out_blocks;
    int i, j, k;
    if (!parts_ijk(parts, inside, i, j, k)) return;
    double gu[3][3];
    if (inside) grad_at(g, K, u, i, j, k, gu, true);
    else grad_at(g, K, u, i, j, k, gu);
    double s[3][3];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) s[a][b] = 0.5 * (gu[a][b] + gu[b][a]);
    const long long o = e.at(i, j, k);
    if (voigt) {
        const double v[6] = {s[0][0], s[1][1], s[2][2], s[1][2], s[2][0], s[0][1]};
        for (int q = 0; q < 6; ++q) e.p[o + q * e.sc] = v[q];
    } else {
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) e.p[o + (3 * a + b) * e.sc] = s[a][b];
    }
}
// Bound by FP64 operations (57 for a cubic stress, 6 more for the energy).  129^3 cubic nodes: 0.377 ms
// either, now 0.245: interior blocks without the boundary's selections, and the energy
// W(grad u) + sum 1/2 sigma : eps as sigma : grad u where sigma is symmetric.
template <int M>
__global__ void __launch_bounds__(kBlock) k_stress(Geo g, SCoef<double> K, Parts parts, View<const double> C,
                                                   View<const double> u, View<double> sg, int voigt, int energy) {
    constexpr int NC = NCoef<M>::value;
    const bool inside = blockIdx.x >= parts.out_blocks;
    int i, j, k;
    if (!parts_ijk(parts, inside, i, j, k)) return;
    double gu[3][3], s[3][3], a[NC];
    if (inside) grad_at(g, K, u, i, j, k, gu, true);
    else grad_at(g, K, u, i, j, k, gu);
    const long long cc = C.at(i, j, k);
#pragma unroll
    for (int q = 0; q < NC; ++q) a[q] = C.p[cc + q * C.sc];
    stress_of<M, double>(a, gu, s);
    const long long o = sg.at(i, j, k);
    if (energy) {
        // W(gradu) = trace(0.5 gradu^T (C gradu)), then += sum 0.5 sig:eps (Elastic.cpp:557-569)
        double w;
        if (M == DIAG) {
            w = 0.0;
            for (int ii = 0; ii < 3; ++ii) {
                double tt = 0.0;
                for (int jj = 0; jj < 3; ++jj) tt += gu[jj][ii] * s[jj][ii];
                w += 0.5 * tt;
            }
            for (int m = 0; m < 3; ++m)
                for (int n = 0; n < 3; ++n) w += .5 * s[m][n] * (.5 * (gu[m][n] + gu[n][m]));
        } else {
            w = s[0][0] * gu[0][0] + s[1][1] * gu[1][1] + s[2][2] * gu[2][2] + s[0][1] * (gu[0][1] + gu[1][0]) +
                s[0][2] * (gu[0][2] + gu[2][0]) + s[1][2] * (gu[1][2] + gu[2][1]);
        }
        sg.p[o] = w;
    } else if (voigt) {
        const double v[6] = {s[0][0], s[1][1], s[2][2], s[1][2], s[2][0], s[0][1]};
        for (int q = 0; q < 6; ++q) sg.p[o + q * sg.sc] = v[q];
    } else {
        for (int a2 = 0; a2 < 3; ++a2)
            for (int b = 0; b < 3; ++b) sg.p[o + (3 * a2 + b) * sg.sc] = s[a2][b];
    }
}
void launch_strain(const Geo& g, View<const double> u, View<double> e, int voigt, cudaStream_t st) {
    const Parts parts = post_parts(g);
    const unsigned nb = parts_blocks(parts);
    if (nb == 0) return;
    k_strain<<<nb, kBlock, 0, st>>>(g, make_scoef<double>(g), parts, u, e, voigt);
    launched();
}
static void launch_stress_energy(const OpParams& P, View<const double> C, View<const double> u, View<double> s, int voigt,
                                 int energy, cudaStream_t st) {
    const Parts parts = post_parts(P.g);
    const unsigned nb = parts_blocks(parts);
    if (nb == 0) return;
    dispatch_model<double>(P.model, [&](auto m) {
        k_stress<decltype(m)::value><<<nb, kBlock, 0, st>>>(P.g, make_scoef<double>(P.g), parts, C, u, s, voigt, energy);
    });
    launched();
}
void launch_stress(const OpParams& P, View<const double> C, View<const double> u, View<double> s, int voigt,
                   cudaStream_t st) {
    launch_stress_energy(P, C, u, s, voigt, 0, st);
}
void launch_energy(const OpParams& P, View<const double> C, View<const double> u, View<double> w, cudaStream_t st) {
    launch_stress_energy(P, C, u, w, 0, 1, st);
}

// ------------------------------------------------------------------ Solver::Nonlocal::Newton<T>
// DW(grad u) = C : (grad u - F0) for the linear and affine models (kinematic variable grad u:
// src/Model/Solid/Linear/Cubic.H:64-67, src/Model/Solid/Affine/Cubic.H:38-41).
// grad u with Numeric::GetStencil relative to the box bx (one-sided on its faces).
__device__ __forceinline__ void grad_box(const Box3& bx, const SCoef<double>& K, const View<const double>& u, int i,
                                         int j, int k, double gu[3][3]) {
    const int ci[3] = {i, j, k};
    const long long os[3] = {1, u.sy, u.sz};
    const long long o = u.at(i, j, k);
    for (int p = 0; p < 3; ++p) {
        const double* up = u.p + o + p * u.sc;
        for (int d = 0; d < 3; ++d) {
            const long long s = os[d];
            if (ci[d] == bx.lo[d]) gu[p][d] = (up[s] - up[0]) * K.id[d];
            else if (ci[d] == bx.hi[d]) gu[p][d] = (up[0] - up[-s]) * K.id[d];
            else gu[p][d] = (up[s] - up[-s]) * K.h[d];
        }
    }
}
template <int M>
__device__ __forceinline__ void newton_sigma(const View<const double>& C, const View<const double>& F0, int i, int j,
                                             int k, double gu[3][3], double s[3][3]) {
    constexpr int NC = NCoef<M>::value;
    double a[NC];
    const long long cc = C.at(i, j, k);
    for (int q = 0; q < NC; ++q) a[q] = C.p[cc + q * C.sc];
    if (F0.p) {
        const long long of = F0.at(i, j, k);
        for (int p = 0; p < 3; ++p)
            for (int d = 0; d < 3; ++d) gu[p][d] -= F0.p[of + (3 * p + d) * F0.sc];
    }
    stress_of<M, double>(a, gu, s);
}
// dw on bx2 = grow(valid, 2) ∩ domain (src/Solver/Nonlocal/Newton.H:45-76)
template <int M>
__global__ void __launch_bounds__(kBlock) k_newton_dw(SCoef<double> K, Reg reg, Box3 bx2, View<const double> C,
                                                      View<const double> u, View<const double> F0, View<double> dw) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    double gu[3][3], s[3][3];
    grad_box(bx2, K, u, i, j, k, gu);
    newton_sigma<M>(C, F0, i, j, k, gu, s);
    const long long o = dw.at(i, j, k);
    for (int p = 0; p < 3; ++p)
        for (int d = 0; d < 3; ++d) dw.p[o + (3 * p + d) * dw.sc] = s[p][d];
}
// rhs on bx1 = grow(valid, 1) ∩ domain (src/Solver/Nonlocal/Newton.H:80-135): BC rows with
// sigma = dw on the domain boundary (faces classified against bx1), b - div(dw) inside
__global__ void __launch_bounds__(kBlock) k_newton_rhs(Geo g, BCP bc, SCoef<double> K, Parts parts, Box3 bx1,
                                                       View<const double> u, View<const double> b,
                                                       View<const double> dw, View<double> rhs) {
    const bool inside = blockIdx.x >= parts.out_blocks;
    int i, j, k;
    if (!parts_ijk(parts, inside, i, j, k)) return;
    const long long ob = b.at(i, j, k), orr = rhs.at(i, j, k), ow = dw.at(i, j, k);
    const bool bnd = !inside && (i == g.dlo[0] || i == g.dhi[0] || j == g.dlo[1] || j == g.dhi[1] || k == g.dlo[2] ||
                                 k == g.dhi[2]);
    if (bnd) {
        double gu[3][3], s[3][3], n[3];
        grad_box(bx1, K, u, i, j, k, gu);
        for (int p = 0; p < 3; ++p)
            for (int d = 0; d < 3; ++d) s[p][d] = dw.p[ow + (3 * p + d) * dw.sc];
        Geo gb = g;
        for (int d = 0; d < 3; ++d) { gb.dlo[d] = bx1.lo[d]; gb.dhi[d] = bx1.hi[d]; }
        const int face = classify<double>(gb, i, j, k, n);
        const long long ou = u.at(i, j, k);
        for (int r = 0; r < 3; ++r) {
            double v = 0.0;
            if (face >= 0) {
                const unsigned char tp = bc.t[face][r];
                if (tp == DISP) v = u.p[ou + r * u.sc];
                else if (tp == TRAC) v = s[r][0] * n[0] + s[r][1] * n[1] + s[r][2] * n[2];
                else if (tp == NEUMANN) v = gu[r][0] * n[0] + gu[r][1] * n[1] + gu[r][2] * n[2];
            }
            rhs.p[orr + r * rhs.sc] = b.p[ob + r * b.sc] - v;
        }
        return;
    }
    const long long os[3] = {1, dw.sy, dw.sz};
    for (int p = 0; p < 3; ++p) {
        double div = 0.0;
        for (int d = 0; d < 3; ++d) {
            const double* w = dw.p + ow + (3 * p + d) * dw.sc;
            div += (w[os[d]] - w[-os[d]]) * K.h[d];  // the reference divides by 2 and dx: 18 divisions a node
        }
        rhs.p[orr + p * rhs.sc] = b.p[ob + p * b.sc] - div;
    }
}
// Newton::DW and Newton::W on valid ∩ domain, stencils relative to the domain
// (src/Solver/Nonlocal/Newton.H:233-333); half = 0.5, or 1 for Affine::Isotropic
// (src/Model/Solid/Affine/Isotropic.H:31-34)
template <int M>
__global__ void __launch_bounds__(kBlock) k_newton_post(Geo g, SCoef<double> K, Reg reg, View<const double> C,
                                                        View<const double> u, View<const double> F0, View<double> dw,
                                                        View<double> w, double half) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    double gu[3][3], s[3][3];
    grad_at(g, K, u, i, j, k, gu);
    newton_sigma<M>(C, F0, i, j, k, gu, s);  // gu now holds grad u - F0
    if (dw.p) {
        const long long o = dw.at(i, j, k);
        for (int p = 0; p < 3; ++p)
            for (int d = 0; d < 3; ++d) dw.p[o + (3 * p + d) * dw.sc] = s[p][d];
    }
    if (w.p) {
        double tr = 0.0;
        for (int p = 0; p < 3; ++p)
            for (int d = 0; d < 3; ++d) tr += gu[p][d] * s[p][d];
        w.p[w.at(i, j, k)] = half * tr;
    }
}
void launch_newton_residual(const OpParams& P, View<const double> C, View<const double> u, View<const double> b,
                            View<const double> F0, View<double> dw, View<double> rhs, cudaStream_t st) {
    const Box3 bx2 = box_isect(box_isect(box_grow(geo_valid(P.g), 2), geo_domain(P.g)), geo_store(P.g));
    const Box3 bx1 = box_isect(box_isect(box_grow(geo_valid(P.g), 1), geo_domain(P.g)), geo_store(P.g));
    const SCoef<double> K = make_scoef<double>(P.g);
    const Reg r2 = make_reg(bx2);
    if (r2.n == 0) return;
    dispatch_model<double>(P.model, [&](auto m) {
        k_newton_dw<decltype(m)::value><<<nblocks(r2.n), kBlock, 0, st>>>(K, r2, bx2, C, u, F0, dw);
    });
    launched();
    const Parts p1 = make_parts(bx1, geo_interior(P.g));
    k_newton_rhs<<<parts_blocks(p1), kBlock, 0, st>>>(P.g, P.bc, K, p1, bx1, u, b, cview(dw), rhs);
    launched();
}
void launch_newton_post(const OpParams& P, View<const double> C, View<const double> u, View<const double> F0,
                        View<double> dw, View<double> w, double half, cudaStream_t st) {
    const Reg reg = make_reg(box_isect(geo_valid(P.g), geo_domain(P.g)));
    if (reg.n == 0) return;
    dispatch_model<double>(P.model, [&](auto m) {
        k_newton_post<decltype(m)::value><<<nblocks(reg.n), kBlock, 0, st>>>(P.g, make_scoef<double>(P.g), reg, C, u,
                                                                              F0, dw, w, half);
    });
    launched();
}

// ------------------------------------------------------------------ NeoHookean (finite kinematics)
// Model::Solid::Elastic::NeoHookean (src/Model/Solid/Elastic/NeoHookean.H:19-66) at F = I + grad u.
// G = F^-T is the signed cofactor matrix of F times 1 / det F; J23 = |det F|^(2/3) from the cube
// root r as (r r + 2 |det F| / r) / 3, in which r's own rounding cancels: 0.6e-16 from the exact power
// in the mean, as pow, at a fraction of its FP64 operations (r r alone is 1.1e-16 off); tr = F : F.
struct NeoKin {
    double F[3][3], G[3][3], J, J23, tr;
};
__device__ __forceinline__ void neo_kin(const double gu[3][3], NeoKin& n) {
    for (int p = 0; p < 3; ++p)
        for (int d = 0; d < 3; ++d) n.F[p][d] = gu[p][d] + (p == d ? 1.0 : 0.0);
    const auto& F = n.F;
    double cof[3][3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
            cof[i][j] = F[i1][j1] * F[i2][j2] - F[i1][j2] * F[i2][j1];
        }
    n.J = F[0][0] * cof[0][0] + F[1][0] * cof[1][0] + F[2][0] * cof[2][0];
    const double inv = 1.0 / n.J;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) n.G[i][j] = cof[i][j] * inv;
    const double aJ = fabs(n.J), root = cbrt(aJ), q = aJ / root;
    n.J23 = aJ > 0. && aJ < 1e308 ? q + fma_rn(root, root, -q) * (1. / 3.) : aJ;  // 0, inf and NaN pass through
    double tr = 0.0;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) tr += F[i][j] * F[i][j];
    n.tr = tr;
}
// NeoHookean::DW (NeoHookean.H:28-39), mu (F / J23 - tr G / (3 J23)) + kappa (J - 1) J G, with one
// division: mu / J23 times F - tr / 3 G (the difference first, as written there), plus a multiple of G
__device__ __forceinline__ void neo_dw(const NeoKin& n, double mu, double kappa, double dw[3][3]) {
    const double a = mu / n.J23, c = kappa * (n.J - 1) * n.J, t = n.tr * (1. / 3.);
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) dw[i][j] = a * (n.F[i][j] - t * n.G[i][j]) + c * n.G[i][j];
}
// NeoHookean::DDW (NeoHookean.H:40-66): with a = mu / J23 and b = kappa J the entry (i, j, k, l) is
//   a (delta_ik delta_jl - 2/3 (F_ij G_kl + G_ij F_kl) + 2/9 tr G_ij G_kl + 1/3 tr G_il G_kj)
//     + b ((2 J - 1) G_ij G_kl + (1 - J) G_il G_kj)
//   = a delta_ik delta_jl + H_ij G_kl - E_ij F_kl + T_il G_kj,
// H = (2/9 a tr + b (2 J - 1)) G - 2/3 a F, E = 2/3 a G, T = (1/3 a tr + b (1 - J)) G: three operations
// an entry instead of about sixteen.  97^3 nodes, all of k_neohookean: 1.32 -> 0.55 ms (memory 0.06).
struct NeoDD {
    double a, H[3][3], E[3][3], T[3][3];
};
__device__ __forceinline__ void neo_dd(const NeoKin& n, double mu, double kappa, NeoDD& q) {
    q.a = mu / n.J23;
    const double b = kappa * n.J, a23 = q.a * (2. / 3.), at = q.a * n.tr;
    const double h = at * (2. / 9.) + b * (2. * n.J - 1.), t = at * (1. / 3.) + b * (1. - n.J);
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            q.H[i][j] = h * n.G[i][j] - a23 * n.F[i][j];
            q.E[i][j] = a23 * n.G[i][j];
            q.T[i][j] = t * n.G[i][j];
        }
}
__device__ __forceinline__ double neo_ddw(const NeoKin& n, const NeoDD& q, int i, int j, int k, int l) {
    const double v = q.H[i][j] * n.G[k][l] - q.E[i][j] * n.F[k][l] + q.T[i][l] * n.G[k][j];
    return i == k && j == l ? v + q.a : v;
}
// Newton::prepareForSolve with kinematic variable F (src/Solver/Nonlocal/Newton.H:45-76) on
// bx2 = grow(valid, 2) ∩ domain: dw = DW(F), and the level's stiffness C = DDW(F) in the 45
// Sym::Major slots.  The reference assigns ddw(i,j,k,l) in (i, j, k, l) order through the shared
// slot of A(3i+j, 3k+l) and A(3k+l, 3i+j), so each slot ends up holding the value evaluated with
// (i, j) the larger row index of the pair: that is the evaluation made here.
__global__ void __launch_bounds__(kBlock) k_neohookean(SCoef<double> K, Reg reg, Box3 bx2, View<const double> u,
                                                       double mu, double kappa, View<double> dw, View<double> C) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    double gu[3][3], w[3][3];
    grad_box(bx2, K, u, i, j, k, gu);
    NeoKin n;
    neo_kin(gu, n);
    neo_dw(n, mu, kappa, w);
    const long long o = dw.at(i, j, k);
    for (int p = 0; p < 3; ++p)
        for (int d = 0; d < 3; ++d) dw.p[o + (3 * p + d) * dw.sc] = w[p][d];
    const long long oc = C.at(i, j, k);
    NeoDD q;
    neo_dd(n, mu, kappa, q);
#pragma unroll
    for (int I = 0; I < 9; ++I)
#pragma unroll
        for (int Kk = I; Kk < 9; ++Kk)
            C.p[oc + major_slot(I, Kk) * C.sc] = neo_ddw(n, q, Kk / 3, Kk % 3, I / 3, I % 3);
}
// Newton::W and Newton::DW with kinematic variable F on valid ∩ domain, stencils relative to
// the domain (src/Solver/Nonlocal/Newton.H:233-333)
__global__ void __launch_bounds__(kBlock) k_neohookean_post(Geo g, SCoef<double> K, Reg reg, View<const double> u,
                                                            double mu, double kappa, View<double> dw,
                                                            View<double> w) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    double gu[3][3];
    grad_at(g, K, u, i, j, k, gu);
    NeoKin n;
    neo_kin(gu, n);
    if (dw.p) {
        double s[3][3];
        neo_dw(n, mu, kappa, s);
        const long long o = dw.at(i, j, k);
        for (int p = 0; p < 3; ++p)
            for (int d = 0; d < 3; ++d) dw.p[o + (3 * p + d) * dw.sc] = s[p][d];
    }
    // NeoHookean::W (NeoHookean.H:19-27)
    if (w.p) {
        double e = 0.0;
        e += 0.5 * mu * (n.tr / n.J23 - 3.);
        e += 0.5 * kappa * (n.J - 1.0) * (n.J - 1.0);
        w.p[w.at(i, j, k)] = e;
    }
}
void launch_neohookean_residual(const OpParams& P, View<const double> u, View<const double> b, double mu,
                                double kappa, View<double> C, View<double> dw, View<double> rhs, cudaStream_t st) {
    const Box3 bx2 = box_isect(box_isect(box_grow(geo_valid(P.g), 2), geo_domain(P.g)), geo_store(P.g));
    const Box3 bx1 = box_isect(box_isect(box_grow(geo_valid(P.g), 1), geo_domain(P.g)), geo_store(P.g));
    const SCoef<double> K = make_scoef<double>(P.g);
    const Reg r2 = make_reg(bx2);
    if (r2.n == 0) return;
    k_neohookean<<<nblocks(r2.n), kBlock, 0, st>>>(K, r2, bx2, u, mu, kappa, dw, C);
    launched();
    const Parts p1 = make_parts(bx1, geo_interior(P.g));
    k_newton_rhs<<<parts_blocks(p1), kBlock, 0, st>>>(P.g, P.bc, K, p1, bx1, u, b, cview(dw), rhs);
    launched();
}
void launch_neohookean_post(const Geo& g, View<const double> u, double mu, double kappa, View<double> dw,
                            View<double> w, cudaStream_t st) {
    const Reg reg = make_reg(box_isect(geo_valid(g), geo_domain(g)));
    if (reg.n == 0) return;
    k_neohookean_post<<<nblocks(reg.n), kBlock, 0, st>>>(g, make_scoef<double>(g), reg, u, mu, kappa, dw, w);
    launched();
}

// ------------------------------------------------------------------ bottom solve (one CTA)
// MLMG::actualBottomSolve + MLCGSolver::solve_cg / solve_bicgstab (krylov_bottom); the whole
// Krylov loop runs inside one thread block on the coarsest level (ng = 0, storage = domain).
// C, D and invD are either the level's global arrays or their copies in shared memory
// (SMEM = true: plain loads instead of __ldg).
template <int M, bool SMEM>
struct BottomOps {
    const BottomArgs& a;
    SCoef<double> K;
    View<const double> Cv;
    const double* D;
    const double* invD;
    int sy, sz, nn;  // the coarsest level is small: 32-bit index arithmetic
    int nx, ny, nz;
    __device__ BottomOps(const BottomArgs& aa, const double* C, const double* D_, const double* invD_)
        : a(aa), D(D_), invD(invD_) {
        K = aa.K;
        const Geo& g = aa.P.g;
        nx = g.vhi[0] - g.vlo[0] + 1;
        ny = g.vhi[1] - g.vlo[1] + 1;
        nz = g.vhi[2] - g.vlo[2] + 1;
        sy = nx;
        sz = nx * ny;
        nn = sz * nz;
        Cv.p = C;
        Cv.lo[0] = g.vlo[0]; Cv.lo[1] = g.vlo[1]; Cv.lo[2] = g.vlo[2];
        Cv.sy = sy; Cv.sz = sz; Cv.sc = nn;
    }
    // out = A x over every node
    __device__ void apply(const double* x, double* out, BlkRed&) const {
        const Geo& g = a.P.g;
        for (int t = threadIdx.x; t < nn; t += blockDim.x) {
            const int k = t / sz, rem = t - k * sz;
            const int j = rem / nx, i = rem - j * nx;
            double v[3];
            const double f = apply_node<M, double, !SMEM>(g, K, a.P.bc, a.P.uniform, Cv.p, nn, t, sy, sz, x, nn, t, sy, sz,
                                         i + g.vlo[0], j + g.vlo[1], k + g.vlo[2], v);
            out[t] = f * v[0];
            out[t + nn] = f * v[1];
            out[t + 2 * nn] = f * v[2];
        }
        __syncthreads();
    }
    __device__ void residual(const double* x, const double* b, double* r, BlkRed& sh) const {
        apply(x, r, sh);
        for (int t = threadIdx.x; t < 3 * nn; t += blockDim.x) r[t] = b[t] - r[t];
        __syncthreads();
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
    // one Fsmooth call: a.sweeps damped-Jacobi sweeps (ng = 0: every node is updated)
    __device__ void smooth(double* x, const double* b, double* tmp, BlkRed& sh) const {
        for (int s = 0; s < a.sweeps; ++s) {
            apply(x, tmp, sh);
            for (int t = threadIdx.x; t < 3 * nn; t += blockDim.x) {
                const double xv = x[t];
                const double rx = tmp[t] - xv * D[t];
                x[t] = (1.0 - a.omega) * xv + a.omega * (b[t] - rx) * invD[t];
            }
            __syncthreads();
        }
    }
};

// SMEM = true: the whole level (C, D, invD, b, x and the 8 work vectors, bottom_smem_doubles)
// lives in dynamic shared memory; x is copied back at the end.
template <int M, bool SMEM>
__global__ void __launch_bounds__(kBottomThreads) k_bottom(BottomArgs a) {
    __shared__ BlkRed sh;
    extern __shared__ double smem[];
    constexpr int NC = NCoef<M>::value;
    const int N = (int)(3 * a.nn);
    const double* Cp = a.C;
    const double* Dp = a.D;
    const double* invDp = a.invD;
    double* x = a.x;
    const double* b = a.b;
    double* work = a.work;
    if (SMEM) {
        double* sC = smem;
        double* sD = sC + NC * a.nn;
        double* sI = sD + N;
        double* sb = sI + N;
        double* sx = sb + N;
        for (long long t = threadIdx.x; t < NC * a.nn; t += blockDim.x) sC[t] = a.C[t];
        for (int t = threadIdx.x; t < N; t += blockDim.x) {
            sD[t] = a.D[t];
            sI[t] = a.invD[t];
            sb[t] = a.b[t];
            sx[t] = a.x[t];
        }
        __syncthreads();
        Cp = sC; Dp = sD; invDp = sI; b = sb; x = sx;
        work = sx + N;
    }
    const BottomOps<M, SMEM> ops(a, Cp, Dp, invDp);
    const KrylovParams kp{a.bottom, a.maxiter, a.reltol, a.nuf};
    const int ret = krylov_bottom(ops, kp, N, x, b, work, sh);
    if (ret != 0 && ret != 9 && threadIdx.x == 0 && a.fail_count) atomicAdd(a.fail_count, 1);
    if (SMEM) {
        for (int t = threadIdx.x; t < N; t += blockDim.x) a.x[t] = x[t];
    }
}

// doubles of dynamic shared memory the SMEM variant needs for nn nodes
__host__ __device__ constexpr long long bottom_smem_doubles(int nc, long long nn) { return (nc + 36) * nn; }

// Levels whose arrays fit the default 48 KB of dynamic shared memory (no function attribute,
// so the launch is legal inside stream capture) run from shared memory; larger ones from global.
void launch_bottom(const BottomArgs& a, cudaStream_t st) {
    dispatch_model4<double>(a.P.model, [&](auto m) {
        constexpr int Mv = decltype(m)::value;
        const size_t bytes = (size_t)bottom_smem_doubles(NCoef<Mv>::value, a.nn) * sizeof(double);
        if (bytes <= kBottomSmemBytes) k_bottom<Mv, true><<<1, kBottomThreads, bytes, st>>>(a);
        else k_bottom<Mv, false><<<1, kBottomThreads, 0, st>>>(a);
    });
    launched();
}

// Mixed precision on a refined patch: the FP32 correction e was just added to the FP64 solution
// x.  The outermost ghost ring of the patch (grow(valid, 2)) has no equation of its own; in the
// FP64 solve it only ever receives coarse corrections interpolated to it, so there it equals the
// interpolation of the coarse solution.  The FP32 cycle interpolates in FP32, and its rounding
// would stay in the ring (nothing corrects it) and bias the interface rows.  Here the ring's
// increment is replaced by the coarse FP32 correction interpolated in FP64:
//   x_ring += interp(e_coarse) - e_ring.
__global__ void __launch_bounds__(kBlock) k_ring_interp_fix(Reg reg, Geo gf, View<double> x, View<const float> ecrse,
                                                            View<const float> efine) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    const bool ring = i == gf.vlo[0] - 2 || i == gf.vhi[0] + 2 || j == gf.vlo[1] - 2 || j == gf.vhi[1] + 2 ||
                      k == gf.vlo[2] - 2 || k == gf.vhi[2] + 2;
    if (!ring) return;
    for (int n = 0; n < 3; ++n) {
        const double v = interp_at<double, float>(ecrse, i, j, k, n);
        x.p[x.at(i, j, k) + n * x.sc] += v - (double)efine.p[efine.at(i, j, k) + n * efine.sc];
    }
}

void launch_ring_interp_fix(const Geo& gf, View<double> x, View<const float> ecrse, View<const float> efine,
                            cudaStream_t st) {
    if (gf.ng < 2) return;
    const Reg reg = make_reg(box_isect(geo_store(gf), geo_domain(gf)));
    if (reg.n == 0) return;
    k_ring_interp_fix<<<nblocks(reg.n), kBlock, 0, st>>>(reg, gf, x, ecrse, efine);
    launched();
}

// ------------------------------------------------------------------ assembled bottom operator
// The coarsest level's operator as an explicit FP64 matrix, for the bottom solve.  GB300 issues
// FP64 at a small fraction of its FP32 rate, and the stencil form of the level operator costs a few
// hundred FP64 instructions per node on one SM; the assembled rows cost one FMA per nonzero.  Column
// j is the operator applied to the unit vector e_j (so every entry is the stencil's own coefficient
// sum for that pair of unknowns); its nonzeros are packed on the device, a warp per row.

// block j: column j of the dense N x N matrix A (row-major); E holds one unit vector per block
template <int M>
__global__ void __launch_bounds__(128) k_bottom_assemble(BottomArgs a, double* A, double* E) {
    const long long nn = a.nn, N = 3 * nn;
    const long long j = blockIdx.x;
    double* e = E + j * N;
    for (int t = threadIdx.x; t < N; t += blockDim.x) e[t] = (t == j) ? 1.0 : 0.0;
    __syncthreads();
    const Geo& g = a.P.g;
    const int nx = g.vhi[0] - g.vlo[0] + 1, ny = g.vhi[1] - g.vlo[1] + 1;
    const long long sy = nx, sz = (long long)nx * ny;
    for (long long t = threadIdx.x; t < nn; t += blockDim.x) {
        const int k = (int)(t / sz), rem = (int)(t - (long long)k * sz);
        const int jj = rem / nx, i = rem - jj * nx;
        double v[3];
        const double f = apply_node<M, double, true>(g, a.K, a.P.bc, a.P.uniform, a.C, nn, t, sy, sz, e, nn, t, sy, sz, i + g.vlo[0],
                                    jj + g.vlo[1], k + g.vlo[2], v);
        A[t * N + j] = f * v[0];
        A[(t + nn) * N + j] = f * v[1];
        A[(t + 2 * nn) * N + j] = f * v[2];
    }
}
void launch_bottom_assemble(const BottomArgs& a, double* A, double* E, cudaStream_t st) {
    dispatch_model4<double>(a.P.model, [&](auto m) {
        k_bottom_assemble<decltype(m)::value><<<(unsigned)(3 * a.nn), 128, 0, st>>>(a, A, E);
    });
    launched();
}

// Packing the nonzeros here instead of copying the dense matrix (19 MB for 1536 unknowns) to the host and packing
// there: the first FP64 solve of a preparation is charged with all of the assembly.  8^3 nodes, 21 slots, first
// solve over a repeated one: 3.3 ms with the packing on the host, 0.9 here.
constexpr int kPackThreads = 128;
__global__ void __launch_bounds__(kPackThreads) k_csr_count(const double* __restrict__ A, int N, int* __restrict__ count) {
    const int r = (int)((blockIdx.x * kPackThreads + threadIdx.x) / 32), lane = threadIdx.x & 31;
    if (r >= N) return;
    int n = 0;
    for (int c = lane; c < N; c += 32) n += A[(long long)r * N + c] != 0.0;
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) count[r] = n;
}
__global__ void __launch_bounds__(kPackThreads) k_csr_fill(const double* __restrict__ A, int N, const int* __restrict__ rowptr,
                                                           int* __restrict__ col, double* __restrict__ val) {
    const int r = (int)((blockIdx.x * kPackThreads + threadIdx.x) / 32), lane = threadIdx.x & 31;
    if (r >= N) return;
    int at = rowptr[r];
    for (int c0 = 0; c0 < N; c0 += 32) {
        const int c = c0 + lane;
        const double v = c < N ? A[(long long)r * N + c] : 0.0;
        const unsigned ball = __ballot_sync(0xffffffffu, v != 0.0);
        if (v != 0.0) {
            const int q = at + __popc(ball & ((1u << lane) - 1u));
            col[q] = c;
            val[q] = v;
        }
        at += __popc(ball);
    }
}
void launch_csr_count(const double* A, int N, int* count, cudaStream_t st) {
    k_csr_count<<<(unsigned)((N * 32 + kPackThreads - 1) / kPackThreads), kPackThreads, 0, st>>>(A, N, count);
    launched();
}
void launch_csr_fill(const double* A, int N, const int* rowptr, int* col, double* val, cudaStream_t st) {
    k_csr_fill<<<(unsigned)((N * 32 + kPackThreads - 1) / kPackThreads), kPackThreads, 0, st>>>(A, N, rowptr, col, val);
    launched();
}

// Krylov operations over the CSR rows (fixed order: deterministic).  With chunks (part != null)
// a thread sums the products of a chunk into part[], then a thread per row adds its chunks in
// order; else one thread per row.
struct CsrOps {
    const BottomArgs& a;
    const int* rowptr;
    const int* col;
    const double* val;
    int N;
    const int* cptr = nullptr;
    const int* rch = nullptr;
    double* part = nullptr;
    int nchunk = 0;
    __device__ void apply(const double* x, double* out, BlkRed&) const {
        if (part) {
            for (int c = threadIdx.x; c < nchunk; c += blockDim.x) {
                double s = 0.0;
                for (int q = cptr[c]; q < cptr[c + 1]; ++q) s += val[q] * x[col[q]];
                part[c] = s;
            }
            __syncthreads();
            for (int r = threadIdx.x; r < N; r += blockDim.x) {
                double s = part[rch[r]];
                for (int c = rch[r] + 1; c < rch[r + 1]; ++c) s += part[c];
                out[r] = s;
            }
        } else {
            for (int r = threadIdx.x; r < N; r += blockDim.x) {
                double s = 0.0;
                for (int q = rowptr[r]; q < rowptr[r + 1]; ++q) s += val[q] * x[col[q]];
                out[r] = s;
            }
        }
        __syncthreads();
    }
    __device__ void residual(const double* x, const double* b, double* r, BlkRed& sh) const {
        apply(x, r, sh);
        for (int t = threadIdx.x; t < N; t += blockDim.x) r[t] = b[t] - r[t];
        __syncthreads();
    }
    __device__ double dot(const double* x, const double* y, BlkRed& sh) const {
        double s = 0.0;
        for (int t = threadIdx.x; t < N; t += blockDim.x) s += x[t] * y[t];
        return blk_sum(s, sh);
    }
    __device__ double ninf(const double* x, BlkRed& sh) const {
        double s = 0.0;
        for (int t = threadIdx.x; t < N; t += blockDim.x) s = fmax(s, fabs(x[t]));
        return blk_max(s, sh);
    }
    // one Fsmooth call with the level's FP64 diagonal (the same update as the stencil form)
    __device__ void smooth(double* x, const double* b, double* tmp, BlkRed& sh) const {
        for (int s = 0; s < a.sweeps; ++s) {
            apply(x, tmp, sh);
            for (int t = threadIdx.x; t < N; t += blockDim.x) {
                const double xv = x[t];
                const double rx = tmp[t] - xv * a.D[t];
                x[t] = (1.0 - a.omega) * xv + a.omega * (b[t] - rx) * a.invD[t];
            }
            __syncthreads();
        }
    }
};

// the matrix and the vectors in dynamic shared memory when they fit (SMEM), else from global
template <bool SMEM>
__global__ void __launch_bounds__(kBottomThreads) k_bottom_csr(BottomArgs a, BottomCsr m) {
    __shared__ BlkRed sh;
    extern __shared__ double smem[];
    const int N = (int)(3 * a.nn);
    double* x = a.x;
    const double* b = a.b;
    double* work = a.work;
    const int* rowptr = m.rowptr;
    const int* col = m.col;
    const double* val = m.val;
    if (SMEM) {
        double* sval = smem;
        double* sb = sval + m.nnz;
        double* sx = sb + N;
        double* sw = sx + N;
        double* spart = sw + 8 * N;
        int* srow = reinterpret_cast<int*>(spart + (m.cptr ? m.nchunk : 0));
        int* scol = srow + N + 1;
        int* scp = scol + m.nnz;
        int* src = scp + m.nchunk + 1;
        for (long long t = threadIdx.x; t < m.nnz; t += blockDim.x) { sval[t] = m.val[t]; scol[t] = m.col[t]; }
        for (long long t = threadIdx.x; t <= N; t += blockDim.x) srow[t] = m.rowptr[t];
        for (int t = threadIdx.x; t < N; t += blockDim.x) { sb[t] = a.b[t]; sx[t] = a.x[t]; }
        if (m.cptr) {
            for (int t = threadIdx.x; t <= m.nchunk; t += blockDim.x) scp[t] = m.cptr[t];
            for (int t = threadIdx.x; t <= N; t += blockDim.x) src[t] = m.rch[t];
        }
        __syncthreads();
        rowptr = srow; col = scol; val = sval; b = sb; x = sx; work = sw;
        if (m.cptr) {
            const CsrOps ops{a, rowptr, col, val, N, scp, src, spart, m.nchunk};
            const KrylovParams kp{a.bottom, a.maxiter, a.reltol, a.nuf};
            const int ret = krylov_bottom(ops, kp, N, x, b, work, sh);
            if (ret != 0 && ret != 9 && threadIdx.x == 0 && a.fail_count) atomicAdd(a.fail_count, 1);
            for (int t = threadIdx.x; t < N; t += blockDim.x) a.x[t] = x[t];
            return;
        }
    }
    const CsrOps ops{a, rowptr, col, val, N};
    const KrylovParams kp{a.bottom, a.maxiter, a.reltol, a.nuf};
    const int ret = krylov_bottom(ops, kp, N, x, b, work, sh);
    if (ret != 0 && ret != 9 && threadIdx.x == 0 && a.fail_count) atomicAdd(a.fail_count, 1);
    if (SMEM) {
        for (int t = threadIdx.x; t < N; t += blockDim.x) a.x[t] = x[t];
    }
}

size_t bottom_csr_smem_bytes(long long N, long long nnz, long long nchunk) {
    return (size_t)(nnz + 10 * N + nchunk) * sizeof(double) + (size_t)(N + 1 + nnz + nchunk + 1 + N + 1) * sizeof(int);
}

// one thread per row or chunk, rounded up to whole warps
void launch_bottom_csr(const BottomArgs& a, const BottomCsr& m, cudaStream_t st) {
    const int N = (int)(3 * a.nn);
    const int threads = (int)std::min<long long>(kBottomThreads, (std::max(N, m.nchunk) + 31) / 32 * 32);
    const size_t bytes = bottom_csr_smem_bytes(N, m.nnz, m.cptr ? m.nchunk : 0);
    if (bytes <= kBottomSmemBytes) k_bottom_csr<true><<<1, threads, bytes, st>>>(a, m);
    else k_bottom_csr<false><<<1, threads, 0, st>>>(a, m);
    launched();
}

// ------------------------------------------------------------------ four-warp bottom solve
// The Krylov loop of krylov_bottom on up to 768 unknowns: four warps, vectors in registers, the
// matrix in shared memory.
//
// What bounds it: FP64 issue.  A sub-partition of a GB300 SM takes a warp-wide DFMA every 64 cycles,
// whatever lanes are active (a dependent one after 74, a division about 560), so the time of an
// iteration is the number of warp-wide FP64 instructions on the busiest sub-partition.  A 256-thread
// block puts two warps on each and makes every one of them join each reduction and repeat each
// division.  Here there is one warp per sub-partition, and
//   - the product's chunks are dealt to the warps by length; a long row's chunk sums are added by 8
//     lanes;
//   - sum of squares and max-norm of r share a reduction, the max on integer bit patterns (REDUX);
//   - rho / p.Ap and 1 / rho (for the next beta) are one division instruction, on two lanes;
//   - a reduction needs one barrier.
// Measured on the 3^3-node coarsest level (81 unknowns), a call of 200 CG iterations: 256-thread
// block on the assembled matrix 0.95 ms, on the stencil (the FP64 solve) 2.54 ms, one warp 0.80 ms,
// this kernel 0.54 ms (loads unrolled four steps ahead: 0.60).  648 unknowns, BiCGStab: 4.2 ms in
// the block, 2.7 ms here.
struct QuadShared {
    double part[2][kEllWarps];
    unsigned long long top[2][kEllWarps];
};
// |v| as bits; NaN counts as 0, as fmax drops it
__device__ __forceinline__ unsigned long long abs_bits(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return b > 0x7ff0000000000000ull ? 0ull : b;
}
// a < b for non-negative doubles
__device__ __forceinline__ bool lt_bits(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); }
__device__ __forceinline__ bool is_zero(double a) { return (__double_as_longlong(a) << 1) == 0; }

// E: unknowns per thread (slots t, t + 128, ...)
template <int E>
struct QuadEll {
    const double* val;
    const unsigned short* col;
    const int* goff;
    const int* slot;
    double* part;  // chunk sums
    double* xs;    // the vector multiplied
    QuadShared* sh;
    int g0, g1;    // this warp's groups
    int lane, warp, buf;
    int rows[E];
    int most[E];   // most chunks of a row of this warp in each layer, long rows apart
    bool wide[E];  // a long row among them

    // out = A v
    __device__ __forceinline__ void apply(const double (&v)[E], double (&out)[E]) const {
#pragma unroll
        for (int e = 0; e < E; ++e) xs[threadIdx.x + kEllThreads * e] = v[e];
        __syncthreads();
        for (int g = g0; g < g1; ++g) {
            const int w = slot[32 * g + lane], len = (w >> 16) - 1;
            const int base = goff[g] + lane;
            double s = 0.0;
            for (int q = 0; q < len; ++q) s = fma(val[base + 32 * q], xs[col[base + 32 * q]], s);
            if (w) part[w & 0xffff] = s;
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int first = rows[e] & 0xffff, n = rows[e] >> 16;
            const bool mine = n <= kEllLongRow;
            const auto at = [&](int c) { return mine && c < n ? part[first + c] : 0.0; };
            double s = at(0);
            if (most[e] > 2) s = (s + at(1)) + (at(2) + at(3));
            else if (most[e] > 1) s = s + at(1);
            if (wide[e]) {
                const int w = __shfl_sync(0xffffffffu, rows[e], lane & 24), n8 = w >> 16, f8 = w & 0xffff;
                double t = 0.0;
                if (n8 > kEllLongRow) {
                    t = (lane & 7) < n8 ? part[f8 + (lane & 7)] : 0.0;
                    for (int c = (lane & 7) + 8; c < n8; c += 8) t += part[f8 + c];
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (!mine) s = t;
            }
            out[e] = s;
        }
    }
    // the sum of s over the block; with TOP also the max of the bit patterns m
    template <bool TOP>
    __device__ __forceinline__ double reduce(double s, unsigned long long m, double& top) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        unsigned long long t = 0;
        if (TOP) {
            const unsigned h = __reduce_max_sync(0xffffffffu, (unsigned)(m >> 32));
            const unsigned l = __reduce_max_sync(0xffffffffu, (unsigned)(m >> 32) == h ? (unsigned)m : 0u);
            t = ((unsigned long long)h << 32) | l;
        }
        // two buffers: a warp may be writing the next sum while another still reads this one
        buf ^= 1;
        if (lane == 0) {
            sh->part[buf][warp] = s;
            if (TOP) sh->top[buf][warp] = t;
        }
        __syncthreads();
        if (TOP)
            top = __longlong_as_double((long long)max(max(sh->top[buf][0], sh->top[buf][1]),
                                                      max(sh->top[buf][2], sh->top[buf][3])));
        return (sh->part[buf][0] + sh->part[buf][1]) + (sh->part[buf][2] + sh->part[buf][3]);
    }
    __device__ __forceinline__ double dot(const double (&x)[E], const double (&y)[E]) {
        double s = x[0] * y[0], none;
#pragma unroll
        for (int e = 1; e < E; ++e) s = fma(x[e], y[e], s);
        return reduce<false>(s, 0, none);
    }
    // the dot product x.y and the max-norm of r
    __device__ __forceinline__ double dot_max(const double (&x)[E], const double (&y)[E], const double (&r)[E],
                                              double& rmax) {
        double s = x[0] * y[0];
        unsigned long long m = abs_bits(r[0]);
#pragma unroll
        for (int e = 1; e < E; ++e) {
            s = fma(x[e], y[e], s);
            m = max(m, abs_bits(r[e]));
        }
        return reduce<true>(s, m, rmax);
    }
};

// the quotients a / b and c / d as one division
__device__ __forceinline__ void div2(double a, double b, double c, double d, int lane, double& q0, double& q1) {
    const double q = (lane == 1 ? c : a) / (lane == 1 ? d : b);
    q0 = __shfl_sync(0xffffffffu, q, 0);
    q1 = __shfl_sync(0xffffffffu, q, 1);
}
template <class R, int E>
__global__ void __launch_bounds__(kEllThreads) k_bottom_quad(BottomArgs a, BottomEll m, const R* __restrict__ bg,
                                                             R* __restrict__ xg) {
    extern __shared__ double smem[];
    __shared__ QuadShared shared;
    const int tid = threadIdx.x;
    QuadEll<E> A;
    double* sval = smem;
    A.part = sval + m.nval;
    A.xs = A.part + m.nchunk;
    int* sgoff = reinterpret_cast<int*>(A.xs + kEllThreads * E);
    int* sslot = sgoff + m.ngroups + 1;
    unsigned short* scol = reinterpret_cast<unsigned short*>(sslot + 32 * m.ngroups);
    for (int t = tid; t < m.nval; t += kEllThreads) {
        sval[t] = __ldg(m.val + t);
        scol[t] = __ldg(m.col + t);
    }
    for (int t = tid; t <= m.ngroups; t += kEllThreads) sgoff[t] = __ldg(m.goff + t);
    for (int t = tid; t < 32 * m.ngroups; t += kEllThreads) sslot[t] = __ldg(m.slot + t);
    A.val = sval;
    A.col = scol;
    A.goff = sgoff;
    A.slot = sslot;
    A.sh = &shared;
    A.lane = tid & 31;
    A.warp = tid >> 5;
    A.buf = 0;
    A.g0 = __ldg(m.wgrp + A.warp);
    A.g1 = __ldg(m.wgrp + A.warp + 1);
    int pm[E];
    double b[E], x[E], r[E], p[E], q[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int t = tid + kEllThreads * e;
        const bool in = t < kEllThreads * m.layers;
        A.rows[e] = in ? __ldg(m.rows + t) : 0;
        pm[e] = in ? __ldg(m.perm + t) : -1;
        const unsigned n = (unsigned)A.rows[e] >> 16;
        A.most[e] = (int)__reduce_max_sync(0xffffffffu, n <= (unsigned)kEllLongRow ? n : 0u);
        A.wide[e] = __any_sync(0xffffffffu, n > (unsigned)kEllLongRow);
        b[e] = pm[e] >= 0 ? (double)bg[pm[e]] : 0.0;
        x[e] = 0.0;
        r[e] = b[e];  // the correction starts at zero
    }
    double rnorm = 0.0;
    double rho = A.dot_max(r, r, r, rnorm);
    const double rnorm0 = rnorm, stop = a.reltol * rnorm0;
    int ret = 0;
    if (!is_zero(rnorm0)) {
        if (a.bottom == 0) {
            double rho_1 = 0.0, inv_1 = 0.0;
            for (int iter = 1; iter <= a.maxiter; ++iter) {
                if (is_zero(rho)) { ret = 1; break; }
                if (iter == 1) {
#pragma unroll
                    for (int e = 0; e < E; ++e) p[e] = r[e];
                } else {
                    const double beta = div_by(rho, rho_1, inv_1);
#pragma unroll
                    for (int e = 0; e < E; ++e) p[e] = fma(beta, p[e], r[e]);
                }
                A.apply(p, q);
                const double pw = A.dot(p, q);
                if (is_zero(pw)) { ret = 1; break; }
                double alpha;
                div2(rho, pw, 1.0, rho, A.lane, alpha, inv_1);
#pragma unroll
                for (int e = 0; e < E; ++e) r[e] = fma(-alpha, q[e], r[e]);
                rho_1 = rho;
                rho = A.dot_max(r, r, r, rnorm);
#pragma unroll
                for (int e = 0; e < E; ++e) x[e] = fma(alpha, p[e], x[e]);
                if (lt_bits(rnorm, stop)) break;
            }
        } else {
            double rh[E], v[E], tt[E];
            double rho_1 = 0.0, inv_1 = 0.0, alpha = 0.0, omega = 0.0, inv_omega = 0.0;
#pragma unroll
            for (int e = 0; e < E; ++e) { rh[e] = r[e]; p[e] = 0.0; v[e] = 0.0; }
            for (int iter = 1; iter <= a.maxiter; ++iter) {
                if (is_zero(rho)) { ret = 1; break; }
                if (iter == 1) {
#pragma unroll
                    for (int e = 0; e < E; ++e) p[e] = r[e];
                } else {
                    const double beta = div_by(rho, rho_1, inv_1) * div_by(alpha, omega, inv_omega);
#pragma unroll
                    for (int e = 0; e < E; ++e) p[e] = fma(beta, fma(-omega, v[e], p[e]), r[e]);
                }
                A.apply(p, v);
                const double rhTv = A.dot(rh, v);
                if (is_zero(rhTv)) { ret = 2; break; }
                div2(rho, rhTv, 1.0, rho, A.lane, alpha, inv_1);
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    r[e] = fma(-alpha, v[e], r[e]);
                    x[e] = fma(alpha, p[e], x[e]);
                }
                // the max-norm of r ends the iteration when it is small; t = A r does no harm then
                A.apply(r, tt);
                const double t_t = A.dot_max(tt, tt, r, rnorm);
                if (lt_bits(rnorm, stop)) break;
                const double t_r = A.dot(tt, r);
                if (is_zero(t_t)) { ret = 3; break; }
                div2(t_r, t_t, t_t, t_r, A.lane, omega, inv_omega);
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    x[e] = fma(omega, r[e], x[e]);
                    r[e] = fma(-omega, tt[e], r[e]);
                }
                rho_1 = rho;
                rho = A.dot_max(rh, r, r, rnorm);
                if (lt_bits(rnorm, stop)) break;
                if (is_zero(omega)) { ret = 4; break; }
            }
        }
        if (ret == 0 && lt_bits(stop, rnorm)) ret = 8;
    }
    // MLMG: the correction is kept when the residual fell, and on failure nuf smoother calls from
    // zero take its place
    const bool keep = ret == 0 && lt_bits(rnorm, rnorm0);
    if (ret != 0) {
        double D[E], I[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            x[e] = 0.0;
            D[e] = pm[e] >= 0 ? __ldg(a.D + pm[e]) : 0.0;
            I[e] = pm[e] >= 0 ? __ldg(a.invD + pm[e]) : 0.0;
        }
        for (int s = 0; s < a.nuf * a.sweeps; ++s) {
            A.apply(x, q);
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const double rx = q[e] - x[e] * D[e];
                x[e] = (1.0 - a.omega) * x[e] + a.omega * (b[e] - rx) * I[e];
            }
        }
        if (tid == 0 && a.fail_count) atomicAdd(a.fail_count, 1);
    }
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (pm[e] >= 0) xg[pm[e]] = (R)(ret != 0 || keep ? x[e] : 0.0);
}

namespace {
constexpr size_t kQuadSmemMax = 200 * 1024;
// E: the instantiations (layers rounded up)
template <class F>
void quad_by_layers(int layers, F&& f) {
    if (layers <= 1) f(std::integral_constant<int, 1>());
    else if (layers <= 2) f(std::integral_constant<int, 2>());
    else if (layers <= 3) f(std::integral_constant<int, 3>());
    else f(std::integral_constant<int, kBottomQuadLayers>());
}
template <int E>
size_t quad_smem_bytes(const BottomEll& m) {
    return sizeof(double) * (size_t)(m.nval + m.nchunk + kEllThreads * E) + sizeof(int) * (size_t)(33 * m.ngroups + 1) +
           sizeof(unsigned short) * (size_t)m.nval;
}
}  // namespace

bool bottom_quad_init(const BottomEll& m) {
    if (m.layers > kBottomQuadLayers) return false;
    bool ok = false;
    quad_by_layers(m.layers, [&](auto e) {
        constexpr int E = decltype(e)::value;
        const size_t bytes = quad_smem_bytes<E>(m);
        ok = bytes <= kQuadSmemMax;
        if (ok && bytes > kBottomSmemBytes) {  // beyond the default: raise the limit, once and for all sizes
            AE_CUDA_CHECK(cudaFuncSetAttribute(k_bottom_quad<double, E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kQuadSmemMax));
            AE_CUDA_CHECK(cudaFuncSetAttribute(k_bottom_quad<float, E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kQuadSmemMax));
        }
    });
    return ok;
}

template <class R>
void launch_bottom_quad(const BottomArgs& a, const BottomEll& m, const R* b, R* x, cudaStream_t st) {
    quad_by_layers(m.layers, [&](auto e) {
        constexpr int E = decltype(e)::value;
        k_bottom_quad<R, E><<<1, kEllThreads, quad_smem_bytes<E>(m), st>>>(a, m, b, x);
    });
    launched();
}
template void launch_bottom_quad<double>(const BottomArgs&, const BottomEll&, const double*, double*, cudaStream_t);
template void launch_bottom_quad<float>(const BottomArgs&, const BottomEll&, const float*, float*, cudaStream_t);

// Linear::solveaffine's right-hand side (src/Solver/Nonlocal/Linear.H:62-89): with r = 0 - A 0,
// the negated apply of zero, rhs += r on nodes inside the domain, nothing on its boundary.
__global__ void __launch_bounds__(kBlock) k_affine_rhs(Geo g, Reg reg, View<double> rhs, View<const double> r) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= reg.n) return;
    int i, j, k;
    reg_ijk(reg, t, i, j, k);
    if (i == g.dlo[0] || i == g.dhi[0] || j == g.dlo[1] || j == g.dhi[1] || k == g.dlo[2] || k == g.dhi[2]) return;
    const long long o = rhs.at(i, j, k), q = r.at(i, j, k);
#pragma unroll
    for (int n = 0; n < 3; ++n) rhs.p[o + n * rhs.sc] += r.p[q + n * r.sc];
}
void launch_affine_rhs(const Geo& g, const Box3& region, View<double> rhs, View<const double> r, cudaStream_t st) {
    const Reg reg = make_reg(region);
    if (reg.n == 0) return;
    k_affine_rhs<<<nblocks(reg.n), kBlock, 0, st>>>(g, reg, rhs, r);
    launched();
}

}  // namespace ae
