// Fast FP64 form of the split sweeps: batch members of precision
// CFD_PREC_FP64_FAST.
//
// The method and the reference semantics are those of the plain FP64
// sweeps (cfd_sweep.cuh and cfd_physics.cuh, which restate the reference line
// by line: E/sourcecode/euler_rowsweep.cpp:10-95, euler_colsweep.cpp:10-114,
// E/headers/flux_solver_MUSCLhancock.hpp:128-227,
// E/headers/riemann_solver_HLLC.hpp:50-145 and their A/ counterparts),
// computed for throughput instead of bit identity:
//   * multiply-adds as FMAs, each written as one (see below);
//   * reciprocals and square roots from the hardware approximations
//     (PTX rcp.approx.ftz.f64, rsqrt.approx.ftz.f64) refined by one
//     Newton-Raphson / Householder step to about one ulp, and one reciprocal
//     per divisor shared by every quotient over it (1/rho of a state,
//     1/(S - u*) for both star factors, 1/eps of a mixture);
//   * the primitive Jacobian product with its zero entries dropped;
//   * face states passed to the Riemann solver as primitives (no conserved
//     round trip), with the reference's physicality tests restated on them:
//     rho > 0 and p + gamma p_inf >= 0 (Euler: e >= 0); for Allaire the
//     snapping of near-zero partial densities and near-0/1 volume fractions
//     (A/headers/misc.hpp:251-266) and then the same tests;
//   * the conservative update applied face by face as the fluxes arrive.
// No sum here has a plain product for an operand: it is an fma, or the product
// is a mul().  The compiler may otherwise contract the two in one copy of the
// code and not in another, and the copies (a loop unrolled by two, each set of
// options) would give different bits: a strip's rows fall to the one or the
// other copy by the strip's length, which a member's company in the batch sets.
// It agrees with the reference to a relative L1 density error far below the
// 1e-12 bound of the plain form over the benchmarked runs (measured by the
// tests against the bit-identical form), not bit for bit.
//
// Storage: the packed planes of the mixed form (cfd_mixed.cuh) hold FP64
// values instead of (value, compensation) pairs: components 0-1 as one
// double2 in the "value" float4 plane, 2-3 as one double2 in the
// "compensation" float4 plane, and for Allaire E and z as one double each in
// the two float2 planes.  Both forms take 8 bytes per component, so a member
// needs the same memory in either.
//
// Kernels: the x sweep by warp segments (lanes hold 32 consecutive cells of
// a row, neighbours by shuffles) and the y sweep by marching strips (a lane
// walks up its column with the stencil window in registers), the two
// barrier-free forms of cfd_march.cuh, over the same tile lists.
#pragma once

#include "cfd_march.cuh"

namespace cfd {
namespace fast {

using mixed::Inst;
using mixed::MixedArgs;
using mixed::TileGeom;

// A product that is not contracted into the sums it feeds.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }

// Per-tile FP64 constants held in registers.
struct DPar {
    double g1, p1, gm1, gp1;  // gamma, p_inf, gamma - 1, gamma p_inf (material 1)
    double i1, i2, c1, c2;    // 1/(g1-1), 1/(g2-1), g1 p1/(g1-1), g2 p2/(g2-1)
    int flags;
    __device__ __forceinline__ int limiter() const { return flags & 3; }
    __device__ __forceinline__ bool pvrs() const { return (flags >> 2) & 1; }
    __device__ __forceinline__ bool godunov() const { return (flags >> 3) & 1; }
    __device__ __forceinline__ bool stiff() const { return (flags >> 4) & 1; }
    // p + p_inf and p + gamma p_inf (no addition for a gas)
    __device__ __forceinline__ double plus_p1(double p) const { return stiff() ? p + p1 : p; }
    __device__ __forceinline__ double plus_gp1(double p) const { return stiff() ? p + gp1 : p; }
};

// The parameters of an instance; OPT >= 0: the options its launch is compiled
// for (cfd_march.cuh).
template <int OPT>
__device__ __forceinline__ DPar load_dpar(const Inst& I) {
    DPar P;
    P.g1 = I.eos.g1;
    P.p1 = I.eos.p1;
    P.gm1 = I.eos.gm1_1;
    P.gp1 = I.eos.gp1;
    P.i1 = I.pd[0];
    P.i2 = I.pd[1];
    P.c1 = I.pd[2];
    P.c2 = I.pd[3];
    P.flags = OPT >= 0 ? OPT : I.flags;
    if (OPT >= 0 && !(OPT & mixed::MF_STIFF)) P.p1 = P.gp1 = P.c1 = P.c2 = 0.0;
    return P;
}

// 1/x: the hardware approximation refined by one cubic Newton-Raphson step,
// y (1 + e + e^2) with e = 1 - x y, which takes the approximation's relative
// error to its cube (about one ulp after rounding).
__device__ __forceinline__ double rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// 1/sqrt(a): the hardware approximation refined by one Householder step of
// order 3, y (1 + e/2 + 3 e^2/8) with e = 1 - a y^2.  The approximation is
// taken of a + 1e-300, which is a for every a above 1e-284 and keeps y finite
// for a = 0; NaN for a < 0.
__device__ __forceinline__ double rsqrt_f(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a + 1e-300));
    const double e = fma(-a * y, y, 1.0);
    return fma(y * fma(0.375, e, 0.5), e, y);
}
// sqrt(a), and sqrt(a / b) = a / sqrt(a b) without the division; 0 for a = 0.
__device__ __forceinline__ double sqrt_f(double a) { return mul(a, rsqrt_f(a)); }
__device__ __forceinline__ double sqrt_ratio(double a, double b) { return mul(a, rsqrt_f(mul(a, b))); }

__device__ __forceinline__ int hi32(double x) { return __double2hiint(x); }
constexpr unsigned kInfHi = 0x7ff00000u;   // high word of infinity
constexpr unsigned kSnapHi = 0x3d720000u;  // just above 1e-12

__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }

// Primitive state of a conserved one, with the reciprocals it took:
// W = (rho, u, v, p) for Euler (E/headers/misc_euler.hpp:63-79),
// (rho1 z, rho2 (1-z), u, v, p, z) for Allaire (A/headers/misc.hpp:130-147,
// pressure A/headers/mixturemodel.hpp:18-24 as p = (rho e - eps k) / eps).
template <int MODEL>
struct Prim64 {
    double W[ModelTraits<MODEL>::NV];
    double r;   // 1/rho
    double ie;  // Allaire: 1/eps
    double kn;  // Allaire: eps k
};

template <int MODEL>
__device__ __forceinline__ void mix_eps_kn(const DPar& P, double z, double& eps, double& kn) {
    const double omz = 1.0 - z;
    eps = fma(z, P.i1, omz * P.i2);
    kn = P.stiff() ? fma(z, P.c1, omz * P.c2) : 0.0;
}

template <int MODEL>
__device__ __forceinline__ void c2p(const DPar& P, const double* U, Prim64<MODEL>& Q) {
    if constexpr (MODEL == MODEL_EULER) {
        Q.r = rcp(U[0]);
        const double u = mul(U[1], Q.r), v = mul(U[2], Q.r);
        const double re = fma(-0.5, fma(U[1], u, U[2] * v), U[3]);  // rho e
        Q.W[0] = U[0];
        Q.W[1] = u;
        Q.W[2] = v;
        Q.W[3] = P.stiff() ? fma(P.gm1, re, -P.gp1) : mul(P.gm1, re);
    } else {
        Q.r = rcp(U[0] + U[1]);
        const double u = mul(U[2], Q.r), v = mul(U[3], Q.r);
        const double re = fma(-0.5, fma(U[2], u, U[3] * v), U[4]);
        double eps;
        mix_eps_kn<MODEL>(P, U[5], eps, Q.kn);
        Q.ie = rcp(eps);
        Q.W[0] = U[0];
        Q.W[1] = U[1];
        Q.W[2] = u;
        Q.W[3] = v;
        Q.W[4] = mul(re - Q.kn, Q.ie);
        Q.W[5] = U[5];
    }
}

// rho c^2 of a primitive state: gamma (p + p_inf) (E/headers/stiffened_gas_eos.hpp:78-81),
// (k + p (1/eps + 1)) for a mixture (A/headers/mixturemodel.hpp:34-40).
template <int MODEL>
__device__ __forceinline__ double rho_c2(const DPar& P, const double* W, double ie, double kn) {
    if constexpr (MODEL == MODEL_EULER) return P.g1 * P.plus_p1(W[3]);
    else return fma(kn + W[4], ie, W[4]);
}

// The physicality test of a face state (E/headers/flux_solver_MUSCLhancock.hpp:178-189,
// 212-223): rho > 0 and e >= 0; for Allaire after the snapping of the
// mutating assert, which changes the state the Riemann solver receives.
template <int MODEL>
__device__ __forceinline__ bool phys(const DPar& P, double* W) {
    if constexpr (MODEL == MODEL_EULER) {
        return W[0] > 0.0 && P.plus_gp1(W[3]) >= 0.0;
    } else {
        if (fabs(W[0]) < 1e-12) W[0] = 0.0;
        if (fabs(W[1]) < 1e-12) W[1] = 0.0;
        if (fabs(W[5]) < 1e-12) W[5] = 0.0;
        if (fabs(W[5] - 1.0) < 1e-12) W[5] = 1.0;
        double eps, kn;
        mix_eps_kn<MODEL>(P, W[5], eps, kn);
        return W[0] >= 0.0 && W[1] >= 0.0 && W[0] + W[1] > 0.0 && W[5] >= 0.0 && W[5] <= 1.0 &&
               fma(W[4], eps, kn) >= 0.0;
    }
}

// Slope limiters (E/headers/flux_solver_MUSCLhancock.hpp:30-89; van Leer
// 2 a b / (a + b) where a b > 0).
__device__ __forceinline__ double limit(int lim, double a, double b) {
    switch (lim) {
        case LIM_VANLEER: {
            const double ab = a * b;
            return ab > 0.0 ? 2.0 * ab * rcp(a + b) : 0.0;
        }
        case LIM_MC: {
            // the smallest in size of (a + b)/2, 2 a, 2 b where the signs agree, else 0
            const double x = 2.0 * (fabs(b) < fabs(a) ? b : a), m = 0.5 * (a + b);
            return (hi32(a) ^ hi32(b)) >= 0 ? (fabs(m) < fabs(x) ? m : x) : 0.0;
        }
        case LIM_UNLIMITED:
            return 0.5 * (a + b);
        default: {
            // minmod: the smaller in size where the signs agree, else 0
            const double x = fabs(b) < fabs(a) ? b : a;
            return (hi32(a) ^ hi32(b)) >= 0 ? x : 0.0;
        }
    }
}

template <int NV>
__device__ __forceinline__ void limit_all(int lim, const double* Wm, const double* W,
                                          const double* Wp, double* d) {
    switch (lim) {
        case LIM_VANLEER:
#pragma unroll
            for (int q = 0; q < NV; ++q) d[q] = limit(LIM_VANLEER, W[q] - Wm[q], Wp[q] - W[q]);
            break;
        case LIM_MC:
#pragma unroll
            for (int q = 0; q < NV; ++q) d[q] = limit(LIM_MC, W[q] - Wm[q], Wp[q] - W[q]);
            break;
        case LIM_UNLIMITED:
#pragma unroll
            for (int q = 0; q < NV; ++q) d[q] = limit(LIM_UNLIMITED, W[q] - Wm[q], Wp[q] - W[q]);
            break;
        default:
#pragma unroll
            for (int q = 0; q < NV; ++q) d[q] = limit(LIM_MINMOD, W[q] - Wm[q], Wp[q] - W[q]);
    }
}

// The largest and the smallest high word of component q over four states.
template <int NV>
__device__ __forceinline__ void hi_range(int q, const double* a, const double* b, const double* c,
                                         const double* d, unsigned& lo, unsigned& up) {
    const unsigned x = hi32(a[q]), y = hi32(b[q]), z = hi32(c[q]), w = hi32(d[q]);
    lo = min(min(x, y), min(z, w));
    up = max(max(x, y), max(z, w));
}

// Evolved face states of a cell (E/headers/flux_solver_MUSCLhancock.hpp:195-201):
// Wp/Wm = W +/- d/2 - (dt/(2 dx)) A(W) d with the primitive Jacobian of
// E/headers/misc_euler.hpp:102-119 (A/headers/misc.hpp:189-205), zero entries
// dropped; okp / okm: the slope-extrapolated and the evolved high / low state
// are physical.  Most cells pass on their high words alone: every density
// normal and positive (Allaire: zero, or above the snapping threshold, as
// z and 1 - z), every pressure positive or zero.  Those are sufficient, a
// mixture's eps and eps k being >= 0, and leave nothing to snap; only other
// cells are tested (and snapped) state by state.
template <int MODEL>
__device__ __forceinline__ void face_states(const DPar& P, const Prim64<MODEL>& Q, const double* d,
                                            double s, double* Wp, double* Wm, bool& okp, bool& okm) {
    using T = ModelTraits<MODEL>;
    constexpr int NV = T::NV;
    const double* W = Q.W;
    double E[NV], D[NV], X[NV];
    const double rc2 = rho_c2<MODEL>(P, W, Q.ie, Q.kn);
    const double su = s * W[T::IM];
    if constexpr (MODEL == MODEL_EULER) {
        X[0] = fma(su, d[0], (s * W[0]) * d[1]);
        X[1] = fma(su, d[1], (s * Q.r) * d[3]);
        X[3] = fma(su, d[3], (s * rc2) * d[1]);
    } else {
        const double sd = s * d[2];
        X[0] = fma(su, d[0], W[0] * sd);
        X[1] = fma(su, d[1], W[1] * sd);
        X[2] = fma(su, d[2], (s * Q.r) * d[4]);
        X[4] = fma(su, d[4], rc2 * sd);
    }
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        E[q] = fma(0.5, d[q], W[q]);
        D[q] = fma(-0.5, d[q], W[q]);
        if (q == T::IT || q == 5) {  // X = su d alone
            Wp[q] = fma(-su, d[q], E[q]);
            Wm[q] = fma(-su, d[q], D[q]);
        } else {
            Wp[q] = E[q] - X[q];
            Wm[q] = D[q] - X[q];
        }
    }
    bool ok;
    unsigned lo, up, lop, upp;
    hi_range<NV>(0, E, D, Wp, Wm, lo, up);
    if constexpr (MODEL == MODEL_EULER) {
        hi_range<NV>(3, E, D, Wp, Wm, lop, upp);
        ok = (lo >= 1u) & (max(up, upp) < kInfHi);
    } else {
        unsigned lo1, up1, lo5, up5;
        hi_range<NV>(1, E, D, Wp, Wm, lo1, up1);
        hi_range<NV>(4, E, D, Wp, Wm, lop, upp);
        hi_range<NV>(5, E, D, Wp, Wm, lo5, up5);
        // 1 - z of the four
        const double o[4] = {1.0 - E[5], 1.0 - D[5], 1.0 - Wp[5], 1.0 - Wm[5]};
        const unsigned loz = min(min((unsigned)hi32(o[0]), (unsigned)hi32(o[1])),
                                 min((unsigned)hi32(o[2]), (unsigned)hi32(o[3])));
        const unsigned upz = max(max((unsigned)hi32(o[0]), (unsigned)hi32(o[1])),
                                 max((unsigned)hi32(o[2]), (unsigned)hi32(o[3])));
        ok = (max(max(max(up, up1), max(upp, up5)), upz) < kInfHi) & ((lo >= kSnapHi) | (up == 0u)) &
             ((lo1 >= kSnapHi) | (up1 == 0u)) & ((lo5 >= kSnapHi) | (up5 == 0u)) &
             ((loz >= kSnapHi) | (upz == 0u)) & (max(lo, lo1) != 0u);
    }
    okp = okm = ok;
    if (!ok) {
        okp = phys<MODEL>(P, E);
        okm = phys<MODEL>(P, D);
        okp &= phys<MODEL>(P, Wp);
        okm &= phys<MODEL>(P, Wm);
    }
}

// Sound speed of a primitive state from its own reciprocals.
template <int MODEL>
__device__ __forceinline__ double sound(const DPar& P, const double* W, double r, double ie,
                                        double kn) {
    return sqrt_f(mul(rho_c2<MODEL>(P, W, ie, kn), r));
}

// HLLC flux from primitive face states (E/headers/riemann_solver_HLLC.hpp:50-145,
// A/headers/riemann_solver_HLLC.hpp:49-150; PVRS wave speeds restated from its
// commented block :84-107 with A/headers/riemann_solver_PVRS.hpp:85 and
// A/headers/mixturemodel.hpp:42-52).  F[NV] = u*, F[NV + 1] = z* (Allaire,
// A/headers/flux_solver_MUSCLhancock.hpp:375).  The side is selected by the
// sign bit of u* (+0 goes left), as the reference's copysign blend does.
template <int MODEL>
__device__ __forceinline__ void hllc(const DPar& P, const double* WL, const double* WR, double* F) {
    using T = ModelTraits<MODEL>;
    constexpr int NV = T::NV;
    double rhoL, rhoR, uL, uR, pL, pR, cL, cR;
    double eL = 1.0, eR = 1.0, knL = 0.0, knR = 0.0, MLe = 0.0, MRe = 0.0;  // Allaire: eps, eps k, eps rho
    if constexpr (MODEL == MODEL_EULER) {
        rhoL = WL[0];
        rhoR = WR[0];
        uL = WL[1];
        uR = WR[1];
        pL = WL[3];
        pR = WR[3];
        cL = sqrt_ratio(P.g1 * P.plus_p1(pL), rhoL);
        cR = sqrt_ratio(P.g1 * P.plus_p1(pR), rhoR);
    } else {
        rhoL = WL[0] + WL[1];
        rhoR = WR[0] + WR[1];
        uL = WL[2];
        uR = WR[2];
        pL = WL[4];
        pR = WR[4];
        mix_eps_kn<MODEL>(P, WL[5], eL, knL);
        mix_eps_kn<MODEL>(P, WR[5], eR, knR);
        // c^2 = (k + p (1/eps + 1))/rho = (eps k + p + p eps)/(eps rho)
        MLe = eL * rhoL;
        MRe = eR * rhoR;
        cL = sqrt_ratio(fma(pL, eL, knL + pL), MLe);
        cR = sqrt_ratio(fma(pR, eR, knR + pR), MRe);
    }
    double SL, SR;
    if (MODEL == MODEL_ALLAIRE && P.pvrs()) {
        const double ppv =
            dmax(0.0, fma(0.5, pL + pR, ((0.5 * (uL - uR)) * (0.5 * (rhoL + rhoR))) * (0.5 * (cL + cR))));
        // shock_speed_jump: sqrt(((p* + k) + ((p* + p)/2)/eps) / rho)
        SL = uL - (ppv > pL ? sqrt_ratio(fma(ppv, eL, fma(0.5, ppv + pL, knL)), MLe) : cL);
        SR = uR + (ppv > pR ? sqrt_ratio(fma(ppv, eR, fma(0.5, ppv + pR, knR)), MRe) : cR);
    } else {
        const double us = uL + uR, ca = 0.5 * (cL + cR);
        SL = dmin(fma(0.5, us, -ca), uL - cL);
        SR = dmax(fma(0.5, us, ca), uR + cR);
    }
    const double mL = mul(rhoL, SL - uL), mR = mul(rhoR, SR - uR);
    // u* = num/den; its sign, and 1/(S - u*) = den/(S den - num), do not wait
    // for the quotient
    const double num = fma(-mR, uR, fma(mL, uL, pR - pL)), den = mL - mR;
    const bool left = (hi32(num) ^ hi32(den)) >= 0;
    // per-element selects (a pointer to either side would go through local memory)
    const double rho = left ? rhoL : rhoR, u = left ? uL : uR, p = left ? pL : pR;
    const double v = left ? WL[T::IT] : WR[T::IT];
    const double Sk = left ? SL : SR, wave = left ? dmin(0.0, SL) : dmax(0.0, SR);
    const double q = den * rcp(fma(Sk, den, -num));  // 1/(S - u*)
    const double u_star = mul(num, rcp(den));
    const double fac = mul(Sk - u, q);  // (S - u)/(S - u*)
    // The passive components' flux U u + w (fac U - U) is U A; the normal
    // momentum's rho (u^2 + w (fac u* - u)) + p; the energy's star state
    // fac (E + (u* - u)(rho u* + p/(S - u))) - E gives E A + p u
    // + w (u* - u)(fac rho u* + p/(S - u*))
    const double A = fma(wave, fac - 1.0, u);
    double re;
    if constexpr (MODEL == MODEL_EULER) {
        re = P.plus_gp1(p) * P.i1;
    } else {
        const double eps = left ? eL : eR, kn = left ? knL : knR;
        re = fma(p, eps, kn);  // (p + k) eps
    }
    const double E = fma(0.5 * rho, fma(u, u, v * v), re);
    const double m = mul(rho, A), fu = mul(fac, u_star);
    if constexpr (MODEL == MODEL_EULER) {
        F[0] = m;
    } else {
        F[0] = mul(left ? WL[0] : WR[0], A);
        F[1] = mul(left ? WL[1] : WR[1], A);
        F[5] = 0.0;
        F[NV + 1] = left ? WL[5] : WR[5];
    }
    F[T::IM] = fma(rho, fma(wave, fu - u, u * u), p);
    F[T::IT] = mul(m, v);
    F[T::IE] = fma(wave * (u_star - u), fma(rho, fu, p * q), fma(E, A, p * u));
    F[NV] = u_star;
}

// Allaire z update (A/headers/zupdate.hpp:44-49 upwind, :62-67 second
// order), clipped to [z_min, 1 - z_min] (or [0, 1]).
__device__ __forceinline__ double z_new(bool god, double k, double zL, double z, double zR,
                                        double usL, double usR, double zsL, double zsR,
                                        double z_min) {
    double nz;
    if (god)
        nz = fma(-k, fma(zR - z, dmin(0.0, usR), (z - zL) * dmax(0.0, usL)), z);
    else
        nz = fma(-k, fma(-z, usR - usL, fma(usR, zsR, -usL * zsL)), z);
    const double lo = z_min > 0.0 ? z_min : 0.0, hi = z_min > 0.0 ? 1.0 - z_min : 1.0;
    return dmax(dmin(hi, nz), lo);
}

// Euler: the new state has rho > 0 and rho E >= |m|^2 / 2, i.e. e >= 0.
__device__ __forceinline__ bool euler_physical(const double* N) {
    return N[0] > 0.0 && fma(N[0], N[3], -0.5 * fma(N[1], N[1], N[2] * N[2])) >= 0.0;
}

// Post-update repairs of the reference: Allaire's snapping assert on the new
// state (A/sourcecode/allaire_diffuse_rowsweep.cpp:49, misc.hpp:251-266),
// Euler's density / energy restore from the old state
// (E/sourcecode/euler_rowsweep.cpp:47-82) when rho or e of the new state is
// negative (the caller reads the old state again then; it is rare).
template <int MODEL>
__device__ __forceinline__ void repair(double* N, const double* Uold) {
    if constexpr (MODEL == MODEL_ALLAIRE) {
        // nothing to snap where the four sizes clear the threshold
        const unsigned lo = min(min((unsigned)hi32(N[0]) & 0x7fffffffu, (unsigned)hi32(N[1]) & 0x7fffffffu),
                                min((unsigned)hi32(N[5]) & 0x7fffffffu, (unsigned)hi32(N[5] - 1.0) & 0x7fffffffu));
        if (lo >= kSnapHi) return;
        if (fabs(N[0]) < 1e-12) N[0] = 0.0;
        if (fabs(N[1]) < 1e-12) N[1] = 0.0;
        if (fabs(N[5]) < 1e-12) N[5] = 0.0;
        if (fabs(N[5] - 1.0) < 1e-12) N[5] = 1.0;
    } else {
        if (euler_physical(N)) return;
        double rho = N[0];
        const double u = N[1] / rho, v = N[2] / rho;
        double e = fma(-0.5, fma(u, u, v * v), N[3] / rho);
        const double ro = Uold[0];
        const double uo = Uold[1] / ro, vo = Uold[2] / ro;
        const double eo = fma(-0.5, fma(uo, uo, vo * vo), Uold[3] / ro);
        if (rho <= 1e-12) rho = ro;
        if (e <= 1e-12) e = eo;
        // the pressure of (e, rho) taken back to conserved: rho e + rho |u|^2 / 2
        N[0] = rho;
        N[1] = rho * u;
        N[2] = rho * v;
        N[3] = fma(0.5 * rho, fma(u, u, v * v), rho * e);
    }
}

// The planes of one state buffer of an FP64 member (see the storage note),
// held in registers: the stores of a sweep go through pointers the compiler
// cannot tell apart from the member descriptor, so reading the descriptor's
// pointers again after every store would cost a global load each time.
struct Planes64 {
    double2* a;  // components 0-1
    double2* b;  // components 2-3
    double* c;   // Allaire E
    double* d;   // Allaire z
};

template <int MODEL>
__device__ __forceinline__ Planes64 planes64(const Inst& I, int buf) {
    Planes64 p;
    p.a = reinterpret_cast<double2*>(I.q4[buf][0]);
    p.b = reinterpret_cast<double2*>(I.q4[buf][1]);
    p.c = MODEL == MODEL_ALLAIRE ? reinterpret_cast<double*>(I.q2[buf][0]) : nullptr;
    p.d = MODEL == MODEL_ALLAIRE ? reinterpret_cast<double*>(I.q2[buf][1]) : nullptr;
    return p;
}

// FP64 cell at element offset `off` of a buffer that the sweep only reads.
template <int MODEL>
__device__ __forceinline__ void load64(const Planes64& P, long long off, double* U) {
    const double2 a = __ldg(P.a + off);
    const double2 b = __ldg(P.b + off);
    U[0] = a.x;
    U[1] = a.y;
    U[2] = b.x;
    U[3] = b.y;
    if constexpr (MODEL == MODEL_ALLAIRE) {
        U[4] = __ldg(P.c + off);
        U[5] = __ldg(P.d + off);
    }
}

template <int MODEL>
__device__ __forceinline__ void store64(const Planes64& P, long long off, const double* U) {
    P.a[off] = make_double2(U[0], U[1]);
    P.b[off] = make_double2(U[2], U[3]);
    if constexpr (MODEL == MODEL_ALLAIRE) {
        P.c[off] = U[4];
        P.d[off] = U[5];
    }
}

// Wave speeds |u| + c, |v| + c and the mass terms of a new (unrotated) state
// (E/sourcecode/euler_timestep.cpp:9-26, A/sourcecode/allaire_diffuse_timestep.cpp:10-29).
template <int MODEL>
__device__ __forceinline__ void speeds(const DPar& P, const double* N, double& su, double& sv,
                                       double& m1, double& m2) {
    using MT = ModelTraits<MODEL>;
    Prim64<MODEL> Q;
    c2p<MODEL>(P, N, Q);
    const double c = sound<MODEL>(P, Q.W, Q.r, Q.ie, Q.kn);
    su = fabs(Q.W[MT::IM]) + c;
    sv = fabs(Q.W[MT::IT]) + c;
    m1 = N[0];
    m2 = MODEL == MODEL_ALLAIRE ? N[1] : 0.0;
}

// ---- y sweep by marching strips ---------------------------------------------

// Rows staged ahead through shared memory: a lane copies the cells of rows
// k+1 .. k+kAhead of its column global -> shared with cp.async while it
// computes row k, so no registers are held by the loads in flight; per slot
// NU 16-byte units per lane (components 0-1, 2-3, and for Allaire E and z),
// lane-major.  Euler's ring has kAhead + 2 slots: the slot refilled at row k
// is the one read at row k - 2, so row k - 1 is still there when row k
// computes and its update starts from it there rather than from registers
// (8 fewer registers, y sweep 0.448 -> 0.421 ms at 4096^2).  Allaire, 2 CTAs
// per SM either way, measured 1.5 % slower like that; it carries row k - 1
// in registers and refills the slot read at row k - 1 (kAhead + 1 slots).
constexpr int kAhead = 3;
template <int MODEL>
__host__ __device__ constexpr bool march64_reread() {
    return MODEL == MODEL_EULER;
}
template <int MODEL>
__host__ __device__ constexpr int march64_slots() {
    return kAhead + (march64_reread<MODEL>() ? 2 : 1);
}
template <int MODEL>
__host__ __device__ constexpr int stage_units() {
    return MODEL == MODEL_ALLAIRE ? 3 : 2;
}
template <int MODEL>
__host__ __device__ constexpr int march64_smem_bytes() {
    return 4 * march64_slots<MODEL>() * stage_units<MODEL>() * 32 * 16;  // 4 warps per CTA
}

template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Starts copying the cell at element offset `off` into slot `s` of this lane.
template <int MODEL>
__device__ __forceinline__ void stage_issue(char* stg, int s, const Planes64& P, long long off) {
    constexpr int NU = stage_units<MODEL>();
    mixed::cp_async16(stg + ((s * NU + 0) * 32) * 16, P.a + off);
    mixed::cp_async16(stg + ((s * NU + 1) * 32) * 16, P.b + off);
    if constexpr (MODEL == MODEL_ALLAIRE) {
        mixed::cp_async8(stg + ((s * NU + 2) * 32) * 16, P.c + off);
        mixed::cp_async8(stg + ((s * NU + 2) * 32) * 16 + 8, P.d + off);
    }
}

template <int MODEL>
__device__ __forceinline__ void stage_read(const char* stg, int s, double* U) {
    constexpr int NU = stage_units<MODEL>();
    const double2 a = *reinterpret_cast<const double2*>(stg + ((s * NU + 0) * 32) * 16);
    const double2 b = *reinterpret_cast<const double2*>(stg + ((s * NU + 1) * 32) * 16);
    U[0] = a.x;
    U[1] = a.y;
    U[2] = b.x;
    U[3] = b.y;
    if constexpr (MODEL == MODEL_ALLAIRE) {
        const double2 c = *reinterpret_cast<const double2*>(stg + ((s * NU + 2) * 32) * 16);
        U[4] = c.x;
        U[5] = c.y;
    }
}
// A lane walks up its column from row r0 - 2 to r1 + 1 (two halo rows at each
// end, mirrored at the domain edges as pre_sweep fills them,
// E/sourcecode/euler_ppsweep.cpp:7-118).  Loading row k completes the slope
// and face states of row k - 1, the flux at the face between rows k - 2 and
// k - 1, and the update of row k - 2.  Carried from row to row: the
// primitive states of rows k - 1 and k - 2 (and 1/rho, 1/eps of row k - 1),
// the evolved high-face state of row k - 2 and the partly updated state of
// row k - 2 (its low-face flux applied); the raw state of row k - 1 is read
// again from its staging slot (Euler) or carried (Allaire).
template <int MODEL, int OPT>
__device__ __forceinline__ void march64_strip(const MixedArgs& A, const TileGeom& g, int part) {
    using MT = ModelTraits<MODEL>;
    constexpr int NV = MT::NV;
    const int lane = threadIdx.x & 31;
    const Inst& I = A.insts[g.inst];
    const DPar P = load_dpar<OPT>(I);
    DevState* st = I.st;
    const double dt = st->dt;
    const double s_half = 0.5 * (dt / (I.fix_dy ? I.dy : I.dx));  // the reference: dx (quirk)
    const double k_upd = dt / I.dy;
    const int ny = g.len, nx = g.wid;
    const int col = g.b_org + lane;
    const bool live = col < nx;
    const int c = min(col, nx - 1);
    const int r0 = min(g.a_org + 2 + part * mixed::part_rows(A), ny);
    const int r1 = min(min(r0 + mixed::part_rows(A), g.a_org + 2 + A.rows), ny);
    // the x sweep's output -> the current buffer
    const Planes64 pin = planes64<MODEL>(I, g.cur ^ 1), pout = planes64<MODEL>(I, g.cur);
    const long long pitch = I.pitch;
    const bool wall_lo = (I.flags >> 7) & 1, wall_hi = (I.flags >> 8) & 1;
    const bool god = P.godunov();
    const int lim = P.limiter();
    const double z_min = I.z_min;

    auto src_row = [&](int k, bool& neg) {
        neg = false;
        int r = k;
        if (k < 0) {
            r = -k - 1;
            neg = wall_lo;
        } else if (k >= ny) {
            r = 2 * ny - 1 - k;
            neg = wall_hi;
        }
        return min(max(r, 0), ny - 1);
    };

    Prim64<MODEL> Q1, Q2;          // rows k-1, k-2
    double A2[NV], Pp[NV];         // partly updated row k-2, high face of row k-2
    bool okp = false;              // whether Pp may be used
    double usL = 0.0, zsL = 0.0;   // u*, z* at the low face of row k-2
    double z3 = 0.0;               // z of row k-3 (upwind z update)
    double rmu = 0.0, rmv = 0.0, rm1 = 0.0, rm2 = 0.0;
#pragma unroll
    for (int q = 0; q < NV; ++q) Q1.W[q] = Q2.W[q] = A2[q] = Pp[q] = 0.0;
    Q1.r = Q1.ie = Q1.kn = Q2.r = Q2.ie = Q2.kn = 0.0;

    // this lane's staging slots; rows r0-2 .. r0-3+kAhead in flight first
    extern __shared__ __align__(16) char fast_stage[];
    constexpr bool reread = march64_reread<MODEL>();
    constexpr int NS = march64_slots<MODEL>();
    double H1c[NV];  // raw row k-1 in the sweep frame (when carried)
#pragma unroll
    for (int q = 0; q < NV; ++q) H1c[q] = 0.0;
    char* stg = fast_stage + (threadIdx.x >> 5) * (NS * stage_units<MODEL>() * 32 * 16) + 16 * lane;
    bool dummy;
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
        if (r0 < r1)  // a part without rows copies none: nothing below would wait for them
            stage_issue<MODEL>(stg, j, pin, src_row(r0 - 2 + j, dummy) * pitch + c);
        mixed::cp_async_commit();
    }
    int slot = 0;

    // Euler: unrolled by two, so that the two-row window changes roles
    // instead of being copied (y sweep 2 % faster; no change for Allaire)
#pragma unroll(MODEL == MODEL_EULER ? 2 : 1)
    for (int k = r0 < r1 ? r0 - 2 : r1 + 2; k <= r1 + 1; ++k) {
        double h[NV];
        bool neg;
        src_row(k, neg);
        cp_async_wait<kAhead - 1>();  // row k has arrived
        stage_read<MODEL>(stg, slot, h);
        const int slot1 = slot == 0 ? NS - 1 : slot - 1;                   // row k - 1
        const int refill = !reread ? slot1 : slot >= 2 ? slot - 2 : slot + NS - 2;  // row k - 1 or k - 2
        if (k + kAhead <= r1 + 1)
            stage_issue<MODEL>(stg, refill, pin, src_row(k + kAhead, dummy) * pitch + c);
        mixed::cp_async_commit();
        slot = slot == NS - 1 ? 0 : slot + 1;
        // sweep frame: mirror sign, then (u, v) -> (v, -u) (E/sourcecode/euler_colsweep.cpp:22-29)
        {
            const double m = h[MT::IM], n = neg ? -h[MT::IT] : h[MT::IT];
            h[MT::IM] = n;
            h[MT::IT] = -m;
        }
        Prim64<MODEL> Q0;
        c2p<MODEL>(P, h, Q0);

        // slope and face states of row k-1
        double Pn[NV], Mn[NV];
        bool okn = false, okm = false;
        if (k >= r0 && !god) {
            double d[NV];
            limit_all<NV>(lim, Q2.W, Q1.W, Q0.W, d);
            face_states<MODEL>(P, Q1, d, s_half, Pn, Mn, okn, okm);
        } else {
#pragma unroll
            for (int q = 0; q < NV; ++q) Pn[q] = Mn[q] = Q1.W[q];
        }

        if (k >= r0 + 1) {
            // flux at the face between rows k-2 and k-1
            double F[NV + 2];
            const bool first = god || !(okp && okm);
            if (god || __any_sync(0xffffffffu, first)) {  // rare in second order
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    Pp[q] = first ? Q2.W[q] : Pp[q];
                    Mn[q] = first ? Q1.W[q] : Mn[q];
                }
            }
            hllc<MODEL>(P, Pp, Mn, F);

            if (k >= r0 + 2) {  // row k-2 is complete
                const int row = k - 2;
                double N[NV];
#pragma unroll
                for (int q = 0; q < NV; ++q) N[q] = fma(-k_upd, F[q], A2[q]);
                if constexpr (MODEL == MODEL_ALLAIRE)
                    N[5] = z_new(god, k_upd, z3, A2[5], Q1.W[5], usL, F[NV], zsL, F[NV + 1], z_min);
                {  // rotate back (E/sourcecode/euler_colsweep.cpp:66-73)
                    const double t = N[MT::IM];
                    N[MT::IM] = -N[MT::IT];
                    N[MT::IT] = t;
                }
                if constexpr (MODEL == MODEL_EULER) {
                    if (!euler_physical(N)) {  // the stored old state, for the restore
                        double Uo[NV];
                        load64<MODEL>(pin, row * pitch + c, Uo);
                        repair<MODEL>(N, Uo);
                    }
                } else {
                    repair<MODEL>(N, nullptr);
                }
                if (live) {
                    store64<MODEL>(pout, row * pitch + c, N);
                    double su, sv, m1, m2;
                    speeds<MODEL>(P, N, su, sv, m1, m2);
                    rmu = dmax(rmu, su);
                    rmv = dmax(rmv, sv);
                    rm1 += m1;
                    rm2 += m2;
                }
            }
            // row k-1 takes the flux at its low face (it is updated only
            // when inside the strip, so never a mirrored row)
            double H1[NV];
            if constexpr (reread) {
                stage_read<MODEL>(stg, slot1, H1);
                const double m = H1[MT::IM];
                H1[MT::IM] = H1[MT::IT];
                H1[MT::IT] = -m;
            } else {
#pragma unroll
                for (int q = 0; q < NV; ++q) H1[q] = H1c[q];
            }
#pragma unroll
            for (int q = 0; q < NV; ++q) A2[q] = fma(k_upd, F[q], H1[q]);
            if constexpr (MODEL == MODEL_ALLAIRE) {
                A2[5] = H1[5];
                z3 = Q2.W[5];
                usL = F[NV];
                zsL = F[NV + 1];
            }
        }

        // shift the window
        Q2 = Q1;
        Q1 = Q0;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            Pp[q] = Pn[q];
            if constexpr (!reread) H1c[q] = h[q];
        }
        okp = okn;
    }

    mixed::march_reduce(I, g.ltile * A.split + part, rmu, rmv, rm1, rm2);
}

// Euler bounded to 128 registers for 4 CTAs per SM: its y sweep measured
// faster than at the 3 CTAs of its unbounded register count; Allaire runs 2.
template <int MODEL, int OPT>
__global__ void __launch_bounds__(128, MODEL == MODEL_EULER ? 4 : 2) fast_march_kernel(MixedArgs A) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // close_steps may be scheduled
    const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int w = gw; w < A.ntiles * A.split; w += nw) {
        const TileGeom g = mixed::tile_geom<DIR_Y, mixed::kMarchMaxRows, 32>(A, w / A.split);
        if (!g.skip) march64_strip<MODEL, OPT>(A, g, w % A.split);
    }
}

// ---- x sweep by warp segments -----------------------------------------------
// The 32 lanes hold 32 consecutive cells of a row (kSegCells outputs and a
// 2-cell halo at each end); neighbour values come from the adjacent lanes by
// shuffles.  A warp walks the rows of its tile (A.rows, chosen per launch).
template <int N>
__device__ __forceinline__ void shfl_up64(const double* x, double* y) {
#pragma unroll
    for (int q = 0; q < N; ++q) y[q] = __shfl_up_sync(0xffffffffu, x[q], 1);
}
template <int N>
__device__ __forceinline__ void shfl_down64(const double* x, double* y) {
#pragma unroll
    for (int q = 0; q < N; ++q) y[q] = __shfl_down_sync(0xffffffffu, x[q], 1);
}

constexpr int kSegSlots = kAhead + 1;
template <int MODEL>
__host__ __device__ constexpr int segment64_smem_bytes() {
    return 4 * kSegSlots * stage_units<MODEL>() * 32 * 16;  // 4 warps per CTA
}

template <int MODEL, int OPT>
__device__ __forceinline__ void segment64_tile(const MixedArgs& A, const TileGeom& g, int row_begin, int row_end) {
    using MT = ModelTraits<MODEL>;
    constexpr int NV = MT::NV;
    const int lane = threadIdx.x & 31;
    const Inst& I = A.insts[g.inst];
    const DPar P = load_dpar<OPT>(I);
    const double dt = I.st->dt;
    const double s_half = 0.5 * (dt / I.dx);
    const double k_upd = dt / I.dx;
    const int nx = g.len, ny = g.wid;
    const Planes64 pin = planes64<MODEL>(I, g.cur), pout = planes64<MODEL>(I, g.cur ^ 1);
    const long long pitch = I.pitch;
    const bool god = P.godunov();
    const int lim = P.limiter();
    const double z_min = I.z_min;
    // this lane's column and its mirrored source (pre_sweep's fill)
    const int ga = g.a_org + lane;
    int src = ga;
    bool neg = false;
    if (ga < 0) {
        src = -ga - 1;
        neg = (I.flags >> 5) & 1;
    } else if (ga >= nx) {
        src = 2 * nx - 1 - ga;
        neg = (I.flags >> 6) & 1;
    }
    src = min(max(src, 0), nx - 1);
    const bool writer = lane >= 2 && lane < 2 + mixed::kSegCells && ga < nx;
    row_end = min(row_end, ny);

    // rows staged kAhead ahead, the slot refilled at row r the one read at row r - 1
    extern __shared__ __align__(16) char seg64_stage[];
    char* stg = seg64_stage + (threadIdx.x >> 5) * (kSegSlots * stage_units<MODEL>() * 32 * 16) + 16 * lane;
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
        if (row_begin + j < row_end) stage_issue<MODEL>(stg, j, pin, (row_begin + j) * pitch + src);
        mixed::cp_async_commit();
    }
    int slot = 0;
    for (int row = row_begin; row < row_end; ++row) {
        double h[NV];
        cp_async_wait<kAhead - 1>();  // row `row` has arrived
        stage_read<MODEL>(stg, slot, h);
        if (row + kAhead < row_end)
            stage_issue<MODEL>(stg, slot == 0 ? kSegSlots - 1 : slot - 1, pin, (row + kAhead) * pitch + src);
        mixed::cp_async_commit();
        slot = slot == kSegSlots - 1 ? 0 : slot + 1;
        if (neg) h[MT::IM] = -h[MT::IM];
        Prim64<MODEL> Q;
        c2p<MODEL>(P, h, Q);
        double Wl[NV], Wr[NV];
        shfl_up64<NV>(Q.W, Wl);
        if (!god || MODEL == MODEL_ALLAIRE) shfl_down64<NV>(Q.W, Wr);  // first order: Allaire's z only

        // slope and face states of this cell (used by lanes 1..30)
        double Pf[NV], Mf[NV];
        bool okp = false, okm = false;
        if (!god) {
            double d[NV];
            limit_all<NV>(lim, Wl, Q.W, Wr, d);
            face_states<MODEL>(P, Q, d, s_half, Pf, Mf, okp, okm);
        }

        // HLLC at this cell's low face (between the lane below and this one)
        double F[NV + 2];
        {
            double PL[NV];
            unsigned okL = 0;  // bit l: lane l - 1's high-face state may be used
            if (!god) {
                shfl_up64<NV>(Pf, PL);
                okL = __ballot_sync(0xffffffffu, okp) << 1;
            }
            const bool first = god || (!(((okL >> lane) & 1u) && okm) && lane >= 2);
            if (god || __any_sync(0xffffffffu, first)) {  // rare in second order
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    PL[q] = first ? Wl[q] : PL[q];
                    Mf[q] = first ? Q.W[q] : Mf[q];
                }
            }
            hllc<MODEL>(P, PL, Mf, F);
        }
        double FR[NV + 2];  // Euler's update needs only the NV fluxes, not u*
        shfl_down64<MODEL == MODEL_EULER ? NV : NV + 2>(F, FR);

        // update (lanes 2 .. 2 + kSegCells - 1)
        double N[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) N[q] = fma(k_upd, F[q] - FR[q], h[q]);
        if constexpr (MODEL == MODEL_ALLAIRE)
            N[5] = z_new(god, k_upd, Wl[5], h[5], Wr[5], F[NV], FR[NV], F[NV + 1], FR[NV + 1], z_min);
        if (writer) {  // interior cells: h is the stored old state
            repair<MODEL>(N, h);
            store64<MODEL>(pout, row * pitch + ga, N);
        }
    }
}

// Euler 5 CTAs per SM (96 registers), Allaire 4 (128: 25 % faster than the 3
// of its unbounded count when that was measured); 6 and 5 spill and measured
// 5 and 11 % slower.
//
// Both sweeps wait on FP64 latency at 16-20 warps per SM, with the FP64 pipe
// half busy: at 2048^2 Euler the x sweep runs 369 thread instructions a cell,
// about 155 of them FP64, and the y sweep 384, against 533 and 520 before
// minmod took seven instructions, the physicality tests were made on high
// words, first-order faces were left to a vote, HLLC's star state was reduced
// to one reciprocal that does not wait for u*, sound speeds took one
// reciprocal root and the options were fixed at compile time: x 96.7 -> 74.5
// us, y 108.4 -> 90.7 us a sweep (71.5 since a warp takes one tile, 84.2 since
// close_steps closes the steps; 73.0 and 84.5 with every multiply-add written
// out).  Allaire at 2048x1024 (880 -> 558 instructions in x): x 90.6 -> 63.8 us,
// y 121.1 -> 87.6, then 84.6 us.
template <int MODEL, int OPT>
__global__ void __launch_bounds__(128, MODEL == MODEL_EULER ? 5 : 4) fast_segment_x_kernel(MixedArgs A) {
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (w >= A.ntiles * A.split) return;
    const TileGeom g = mixed::tile_geom<DIR_X, mixed::kSegCells, mixed::kSegRows>(A, w / A.split);
    if (g.skip) return;
    const int n = mixed::part_rows(A), r = g.b_org + (w % A.split) * n;  // this warp's rows
    segment64_tile<MODEL, OPT>(A, g, r, min(r + n, g.b_org + A.rows));
}

}  // namespace fast
}  // namespace cfd
