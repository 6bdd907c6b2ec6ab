// D3Q19 lattice constants and the per-cell collision arithmetic shared by the
// lattice and immersed-boundary kernels.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "bib_internal.h"

namespace bib {

// Velocity set in the reference order, src/latticeBoltzmann/nearestNeighborLattices3D.hh:165-197
// (c[i] = -c[i+9]).
__host__ __device__ constexpr int cx(int i) {
    return (i == 1 || i == 4 || i == 5 || i == 6 || i == 7) ? -1 : ((i == 10 || i == 13 || i == 14 || i == 15 || i == 16) ? 1 : 0);
}
__host__ __device__ constexpr int cy(int i) {
    return (i == 2 || i == 4 || i == 8 || i == 9 || i == 14) ? -1 : ((i == 5 || i == 11 || i == 13 || i == 17 || i == 18) ? 1 : 0);
}
__host__ __device__ constexpr int cz(int i) {
    return (i == 3 || i == 6 || i == 8 || i == 16 || i == 18) ? -1 : ((i == 7 || i == 9 || i == 12 || i == 15 || i == 17) ? 1 : 0);
}
__host__ __device__ constexpr int opposite(int i) { return i == 0 ? 0 : (i < 10 ? i + 9 : i - 9); }

template <class C>
__host__ __device__ constexpr C weight(int i) {
    return i == 0 ? C(1) / C(3) : ((cx(i) * cx(i) + cy(i) * cy(i) + cz(i) * cz(i)) == 1 ? C(1) / C(18) : C(1) / C(36));
}

// ---------------------------------------------------------------- storage
// Populations are stored as f-bar = f - t_i; FP16 storage keeps f-bar * scale.
template <class T>
struct Store;
template <>
struct Store<double> {
    using C = double;
    using F = double;
    using U = double;  // velocity field
    static __device__ __forceinline__ double load(const double* p, float) { return __ldg(p); }
    static __device__ __forceinline__ void store(double* p, double v, float) { *p = v; }
};
template <>
struct Store<float> {
    using C = float;
    using F = float;
    using U = float;
    static __device__ __forceinline__ float load(const float* p, float) { return __ldg(p); }
    static __device__ __forceinline__ void store(float* p, float v, float) { *p = v; }
};
template <>
struct Store<__half> {
    using C = float;
    using F = float;
    using U = __half;  // the velocity field in FP16 too: it only feeds the interpolation
    static __device__ __forceinline__ float load(const __half* p, float inv_scale) {
        return __half2float(__ldg(p)) * inv_scale;
    }
    static __device__ __forceinline__ void store(__half* p, float v, float scale) { *p = __float2half_rn(v * scale); }
};

// ---------------------------------------------------------------- moments
// get_rhoBar_j (partial sums), src/latticeBoltzmann/momentTemplates3D.h:350-423
template <class C>
__device__ __forceinline__ void rho_bar_j(const C* f, C& rb, C* j) {
    const C sxm = f[1] + f[4] + f[5] + f[6] + f[7];
    const C sxp = f[10] + f[13] + f[14] + f[15] + f[16];
    const C sym = f[2] + f[4] + f[8] + f[9] + f[14];
    const C syp = f[5] + f[11] + f[13] + f[17] + f[18];
    const C szm = f[3] + f[6] + f[8] + f[16] + f[18];
    const C szp = f[7] + f[9] + f[12] + f[15] + f[17];
    const C sx0 = f[0] + f[2] + f[3] + f[8] + f[9] + f[11] + f[12] + f[17] + f[18];
    rb = sxm + sx0 + sxp;
    j[0] = sxp - sxm;
    j[1] = syp - sym;
    j[2] = szp - szm;
}
// ExternalForceDynamics::computeVelocity, src/basicDynamics/externalForceDynamics.hh:59-74
template <class C>
__device__ __forceinline__ void velocity_with_force(const C* f, const C* F, C* u) {
    C rb, j[3];
    rho_bar_j(f, rb, j);
    const C inv = C(1) / (rb + C(1));
    u[0] = j[0] * inv + F[0] / C(2);
    u[1] = j[1] * inv + F[1] / C(2);
    u[2] = j[2] * inv + F[2] / C(2);
}

// bgk_ma2_equilibrium, src/latticeBoltzmann/dynamicsTemplates3D.h:675-678
template <class C>
__device__ __forceinline__ C bgk_equilibrium(int i, C rhoBar, C invRho, const C* j, C jSqr) {
    const C c_j = C(cx(i)) * j[0] + C(cy(i)) * j[1] + C(cz(i)) * j[2];
    return weight<C>(i) * (rhoBar + C(3) * c_j + invRho * (C(4.5) * c_j * c_j - C(1.5) * jSqr));
}

// Collision of one cell, every kernel and every precision.  BGK_GUO_VOF is
// GuoExternalForceVOFDynamics::collide (src/fsi/VariableViscosityDynamics.hh:151-172): with
// u = j/rho + F/2, rho = rhoBar + 1, the BGK equilibrium of J = rho u
// (bgk_ma2_collision_base, src/latticeBoltzmann/dynamicsTemplates3D.h:770-838) plus the Guo term of
// VariableViscosityDynamics.hh:47-129,
// t_i (1 - w/2) [3 (c_i - u).F + 9 (c_i.u)(c_i.F)], collapse to
//     f_i' = (1 - w) f_i + t_i [A + c_i.H + (c_i.u)(c_i.K)]
//     H = 3 w rho u + 3 mu F,  K = 4.5 w rho u + 9 mu F,  A = w rhoBar - u.K / 3,
// mu = 1 - w/2, evaluated once per opposite pair (i, i+9) (c_{i+9} = -c_i).  BGK without
// forcing is the same with F = 0 and u = j/rho (BGKdynamics::collide,
// src/basicDynamics/isoThermalDynamics.hh:329-340); TRT is Ginzburg's two-relaxation-time split
// around the same equilibrium (no reference counterpart).  The populations may carry a common scale S
// (FP16 storage keeps f-bar * S): moments are unscaled once, post-collision values come out
// in scaled units.  FP64 is bound by its arithmetic: with
// A by its own products, the scale of FP16 storage (1) and the rates worked out per cell a step of one FP64
// capsule in 64^3 took 138 us, so 132.
// BGK keeps the weights outside the brackets: with w t_i rounded once and folded in, its FP32 mass drifts.  TRT has
// them folded into the rates: the density's deviation from 1 drifts by 6e-8 of itself per step at omega 1.25, 2e-8 at 1.3
// (BGK 2e-8; 64^3 FP32, 1000 steps).  Every product that meets a sum is written as fmac, so that all kernels and
// the packed pairs round alike.

// c_i . (a, b, c) of the populations 10..18, whose first component that is not zero is 1, with the zero
// components left out: multiplications by 0 are not removed by the compiler under IEEE semantics
// (0 * inf is NaN), so they are not written.
template <class C>
__device__ __forceinline__ C cdot(int i, C a, C b, C c) {
    if (cx(i) != 0) {
        if (cy(i) != 0) return cy(i) > 0 ? a + b : a - b;
        if (cz(i) != 0) return cz(i) > 0 ? a + c : a - c;
        return a;
    }
    if (cy(i) != 0) return cz(i) == 0 ? b : (cz(i) > 0 ? b + c : b - c);
    return c;
}
__device__ __forceinline__ float fmac(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmac(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float recip(float a) { return 1.0f / a; }
__device__ __forceinline__ double recip(double a) { return 1.0 / a; }

// Two cells' FP32 values in one register pair: an instruction for both, rounded as for one.
struct F2 {
    float2 v;
    F2() = default;
    __device__ __forceinline__ explicit F2(float a) : v(make_float2(a, a)) {}
    __device__ __forceinline__ F2(float a, float b) : v(make_float2(a, b)) {}
    __device__ __forceinline__ explicit F2(float2 a) : v(a) {}
};
__device__ __forceinline__ F2 fmac(F2 a, F2 b, F2 c) { return F2(__ffma2_rn(a.v, b.v, c.v)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return F2(__fadd2_rn(a.v, make_float2(-b.v.x, -b.v.y))); }
__device__ __forceinline__ F2 operator-(F2 a) { return F2(-a.v.x, -a.v.y); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return F2(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 recip(F2 a) { return F2(1.0f / a.v.x, 1.0f / a.v.y); }

template <class C, int COLL>
__host__ __device__ __forceinline__ RelaxRates<C> relax_rates(C w, C wm, C S) {
    const bool trt = COLL == BIB_COLLISION_TRT;
    RelaxRates<C> r;
    r.omo = C(1) - w;
    r.w = w;
    r.m = trt ? (C(3) * wm * S) * weight<C>(4) : C(3) * (C(1) - C(0.5) * w);
    r.t0 = (trt ? w * S : S) * weight<C>(0);
    r.t = (trt ? w * S : S) * weight<C>(4);
    r.a = C(1) - C(0.5) * (w + wm);
    r.b = C(0.5) * (wm - w);
    return r;
}

// Moments of the incoming state: rhoBar, rho, j and 1/rho, unscaled (SCALED: the populations carry the
// scale whose inverse is invS).
template <class C>
struct CellMoments {
    C rb, rho, j0, j1, j2, invRho;
};
template <class C, bool SCALED>
__device__ __forceinline__ CellMoments<C> moments_compact(const C* f, C invS) {
    const C sxm = f[1] + f[4] + f[5] + f[6] + f[7];
    const C sxp = f[10] + f[13] + f[14] + f[15] + f[16];
    const C sym = f[2] + f[4] + f[8] + f[9] + f[14];
    const C syp = f[5] + f[11] + f[13] + f[17] + f[18];
    const C szm = f[3] + f[6] + f[8] + f[16] + f[18];
    const C szp = f[7] + f[9] + f[12] + f[15] + f[17];
    const C sx0 = f[0] + f[2] + f[3] + f[8] + f[9] + f[11] + f[12] + f[17] + f[18];
    const C sum = sxm + sx0 + sxp;
    CellMoments<C> m;
    m.rb = SCALED ? sum * invS : sum;
    m.rho = SCALED ? fmac(sum, invS, C(1)) : sum + C(1);
    m.j0 = SCALED ? (sxp - sxm) * invS : sxp - sxm;
    m.j1 = SCALED ? (syp - sym) * invS : syp - sym;
    m.j2 = SCALED ? (szp - szm) * invS : szp - szm;
    m.invRho = recip(m.rho);
    return m;
}

// The velocity j/rho + F_prev/2 of the incoming state (the reference's computeVelocity).
template <class C>
__device__ __forceinline__ void velocity_compact(const CellMoments<C>& m, const C* Fprev, C* u) {
    u[0] = fmac(m.j0, m.invRho, C(0.5) * Fprev[0]);
    u[1] = fmac(m.j1, m.invRho, C(0.5) * Fprev[1]);
    u[2] = fmac(m.j2, m.invRho, C(0.5) * Fprev[2]);
}

// Relaxation of one cell from its moments (scaled populations in, scaled populations out).
template <class C, int COLL>
__device__ __forceinline__ void relax_compact(C* f, const C* F, const RelaxRates<C>& r, const CellMoments<C>& m) {
    const C j0 = m.j0, j1 = m.j1, j2 = m.j2;
    if constexpr (COLL == BIB_COLLISION_TRT) {
        // Two relaxation times around the BGK equilibrium of j: the symmetric part of each
        // pair (i, i+9) relaxes with omega, the antisymmetric part with omega_minus;
        // feq+ = t_i (rhoBar + 4.5 (c.j)^2 / rho - 1.5 j.j / rho), feq- = 3 t_i c.j.
        // Collected per pair: f_i' = a f_i + b f_i+9 + (w feq+ + w- feq-) and f_i+9' = a f_i+9 +
        // b f_i + (w feq+ - w- feq-), with a = 1 - (w + w-)/2 and b = (w- - w)/2.
        const C jj = fmac(j2, j2, fmac(j1, j1, j0 * j0));
        const C base = fmac(C(-1.5) * m.invRho, jj, m.rb), B = r.t * base, h = r.t * (C(4.5) * m.invRho);
        const C B2 = B + B, h2 = h + h, mp = r.m, mp2 = mp + mp;
        f[0] = fmac(r.omo, f[0], r.t0 * base);
#pragma unroll
        for (int i = 1; i < 10; ++i) {
            const bool axis = i < 4;
            const C cj = cdot<C>(i + 9, j0, j1, j2);
            const C P = fmac((axis ? h2 : h) * cj, cj, axis ? B2 : B);
            const C fi = f[i], fo = f[i + 9];
            f[i] = fmac(r.a, fi, fmac(r.b, fo, fmac(axis ? -mp2 : -mp, cj, P)));
            f[i + 9] = fmac(r.a, fo, fmac(r.b, fi, fmac(axis ? mp2 : mp, cj, P)));
        }
    } else {
        const C wr = r.w * m.rho, c3 = C(3) * wr, c45 = C(4.5) * wr;
        C u[3], H[3], K[3];
        const C j[3] = {j0, j1, j2};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if constexpr (COLL == BIB_COLLISION_BGK_GUO_VOF) {
                const C mF = r.m * F[a];
                u[a] = fmac(j[a], m.invRho, C(0.5) * F[a]);
                H[a] = fmac(c3, u[a], mF);
                K[a] = fmac(c45, u[a], C(3) * mF);
            } else {
                u[a] = j[a] * m.invRho;
                H[a] = c3 * u[a];
                K[a] = c45 * u[a];
            }
        }
        const C A = fmac(C(-1.0 / 3.0), fmac(u[2], K[2], fmac(u[1], K[1], u[0] * K[0])), r.w * m.rb);
        const C tp = r.t, tp2 = tp + tp;
        f[0] = fmac(r.omo, f[0], r.t0 * A);
#pragma unroll
        for (int i = 1; i < 4; ++i) {
            const C P = tp2 * fmac(u[i - 1], K[i - 1], A);
            f[i] = fmac(r.omo, f[i], fmac(-tp2, H[i - 1], P));
            f[i + 9] = fmac(r.omo, f[i + 9], fmac(tp2, H[i - 1], P));
        }
#pragma unroll
        for (int i = 4; i < 10; ++i) {
            const C cu = cdot<C>(i + 9, u[0], u[1], u[2]), cK = cdot<C>(i + 9, K[0], K[1], K[2]);
            const C cH = cdot<C>(i + 9, H[0], H[1], H[2]);
            const C P = tp * fmac(cu, cK, A);
            f[i] = fmac(r.omo, f[i], fmac(-tp, cH, P));
            f[i + 9] = fmac(r.omo, f[i + 9], fmac(tp, cH, P));
        }
    }
}

// The compact operators at unit scale (FP64 / FP32 populations held as f-bar): omega_minus is the
// TRT rate of the antisymmetric parts, unused otherwise.
template <class C, int COLL>
__device__ __forceinline__ void collide_unscaled(C* f, const C* F, C omega, C omega_minus) {
    relax_compact<C, COLL>(f, F, relax_rates<C, COLL>(omega, omega_minus, C(1)), moments_compact<C, false>(f, C(1)));
}

__host__ __device__ inline int64_t wrap_index(int64_t i, int64_t n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

}  // namespace bib
