// The bit-identical FP64 form through shared reciprocals.
//
// Quotients.  The bit-identical form keeps every division of the reference,
// each rounded to nearest.  Most of them share a divisor with others (three or four
// quotients over one density, two or three over one mixture coefficient), or
// divide by a material constant, so the correctly rounded reciprocal
// y = RN(1/b) is formed once and each quotient takes three operations:
//
//     q0 = RN(a y),   r = RN(b q0 - a),   q = RN(q0 - r y)
//
// which is Markstein's division (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990;
// J.-M. Muller et al., "Handbook of Floating-Point Arithmetic", ch. 4).  With
// mantissas scaled to integers A, B in [2^52, 2^53) and errors in ulps of the
// quotient:
//   * |q0 - a/b| < 1.5, and r is exact when |q0 - a/b| <= 1;
//   * the last operation rounds a/b + (a/b - q0)(by - 1), and a/b is never
//     closer than 1/(2B) to the midpoint of two neighbours.  Next to a
//     midpoint at distance 1/2 from q0 the deviation is at most
//     (1/2)|by - 1| <= B 2^-107 (1 + d) for a reciprocal within
//     (1/2)(1 + d) ulp, below 1/(2B) whenever B^2 (1 + d) < 2^106;
//   * a midpoint at distance 3/2 comes within reach only for A and B both
//     within 8 of 2^53, and for those (A and B within 200 of 2^53, all pairs)
//     the result is RN(a/b), by exact integer arithmetic.
// So y = RN(1/b) serves every divisor, and a y within (1/2)(1 + 2^-48) ulp
// every divisor whose mantissa is not within 16 of 2^53 (near_top).
//
// The reciprocal: the hardware approximation (PTX rcp.approx.ftz.f64; over
// all leading 20 mantissa bits |1 - b y| <= 2^-19.9) refined by a cubic step
// and a final Newton step.  The final step rounds (1/b)(1 - e^2) with
// |e| <= 2^-53 (1 + 2^-6); it could only miss RN(1/b) for a B in
// [2^53/1.2, 2^53) that divides 2^106 - 1, and the only one is 2^53 - 1 (a
// value just below a power of two, which densities near 1 do take).  There
// it gives the power of two below, and RN(1/b) is the next number up.
//
// Square roots: the hardware approximation of 1/sqrt(a) (PTX
// rsqrt.approx.ftz.f64) refined by one Householder step of order 3 (A. S.
// Householder, "The Numerical Treatment of a Single Nonlinear Equation", 1970),
// y (1 + e/2 + 3 e^2/8) with e = 1 - a y^2, then one Newton step on the root
// itself, its residual exact by FMA (Markstein, above): g1 = RN(g + r h) with
// g = RN(a y), h = y/2, r = RN(a - g^2); then
// c = (a - g1^2) h is sqrt(a) - g1 to a relative 2^-40, and g1 is the correctly
// rounded root whenever |c| is below half an ulp of g1 by its high word.  It
// is for all but about one operand in a million; the others take the ordinary
// root.
//
// The guards (pos_ok and friends) keep exponents away from overflow and
// underflow, where r would not be exact: divisors within 2^-100 .. 2^100,
// numerators within 2^-863 .. 2^864 in size or exactly zero.  The sign of a
// zero quotient over a positive divisor is the one of the division: b q0 - a
// is +0 for a zero a of either sign, and q0 - (+0) y keeps q0.
//
// Every function below returns whether its guards held and the state it
// formed is physical by the reference's tests, decided with a margin that
// rounding cannot cross; where one returns false its results are not used,
// and the caller takes the functions of cfd_physics.cuh for the whole update
// (the reference's divisions and tests, with their events).
#pragma once

#include "cfd_physics.cuh"

namespace cfd {

__device__ __forceinline__ unsigned hi_word(double x) { return (unsigned)__double2hiint(x); }
__device__ __forceinline__ unsigned lo_word(double x) { return (unsigned)__double2loint(x); }

constexpr unsigned kNumLo = 0x0a000000u, kNumHi = 0x75f00000u;  // 2^-863 .. 2^864
constexpr unsigned kDivLo = 0x39b00000u, kDivHi = 0x46300000u;  // 2^-100 .. 2^100

// x > 0 within the numerators' range.
__device__ __forceinline__ bool pos_ok(double x) {
    return hi_word(x) - kNumLo < kNumHi - kNumLo;
}
// |x| within the numerators' range, or x = 0 (of either sign).
__device__ __forceinline__ bool num_ok(double x) {
    const unsigned t = hi_word(x) & 0x7fffffffu;
    return (t - kNumLo < kNumHi - kNumLo) | ((t | lo_word(x)) == 0u);
}
// 0 < |x| < 2^-863.
__device__ __forceinline__ bool tiny(double x) {
    const unsigned t = hi_word(x) & 0x7fffffffu;
    return (t < kNumLo) & ((t | lo_word(x)) != 0u);
}
// |x| within the numerators' range.
__device__ __forceinline__ bool abs_ok(double x) {
    return (hi_word(x) & 0x7fffffffu) - kNumLo < kNumHi - kNumLo;
}
// x > 0 within the divisors' range.
__device__ __forceinline__ bool div_ok(double x) {
    return hi_word(x) - kDivLo < kDivHi - kDivLo;
}
// The divisors that need RN(1/b) itself (a superset of those within 16 of
// 2^53 by mantissa).
__device__ __forceinline__ bool near_top(double b) {
    return ((hi_word(b) | 0xfff00000u) & lo_word(b)) >= 0xffffffc0u;
}

// a / b as written, for branches that are rarely taken: the compiler would
// otherwise evaluate a short division on both sides of the branch.
__device__ __forceinline__ double div_cold(double a, double b) {
    double q;
    asm volatile("div.rn.f64 %0, %1, %2;" : "=d"(q) : "d"(a), "d"(b));
    return q;
}

// One Newton step on a reciprocal: y (1 + e), e = 1 - b y.
__device__ __forceinline__ double rcp_step(double b, double y) {
    return __fma_rn(__fma_rn(-b, y, 1.0), y, y);
}
// RN(1/b) for div_ok(b).
__device__ __forceinline__ double rcp_rn(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = __fma_rn(-b, y, 1.0);
    y = rcp_step(b, __fma_rn(__fma_rn(e, e, e), y, y));
    // B = 2^53 - 1
    const int top = ((hi_word(b) | 0xfff00000u) & lo_word(b)) == 0xffffffffu;
    return __hiloint2double(__double2hiint(y), __double2loint(y) | top);
}
// RN(a/b) for div_ok(b), num_ok(a) and y = RN(1/b), or, where b is not
// near_top, a y within (1/2)(1 + 2^-48) ulp of 1/b.
__device__ __forceinline__ double quot_rn(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(-__fma_rn(b, q, -a), y, q);
}

// RN(sqrt(a)) for pos_ok(a); false where the rounding is too close to call.
__device__ __forceinline__ bool sqrt_rn(double a, double& s) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = __fma_rn(-__dmul_rn(a, y), y, 1.0);
    y = __fma_rn(__dmul_rn(y, e), __fma_rn(0.375, e, 0.5), y);
    const double g = __dmul_rn(a, y);
    const double h = __hiloint2double(__double2hiint(y) - 0x100000, __double2loint(y));  // y / 2
    s = __fma_rn(__fma_rn(-g, g, a), h, g);
    const double c = __dmul_rn(__fma_rn(-s, s, a), h);
    // half an ulp of s (of the binade below at a power of two)
    const unsigned half = ((hi_word(s) - 1u) & 0x7ff00000u) - (53u << 20);
    return (hi_word(c) & 0x7fffffffu) < half;
}

// ---- the physics -------------------------------------------------------------

struct MixR {
    double eps, k, ie;  // ie = 1/eps
};
template <int MODEL> struct PrimR {
    double W[ModelTraits<MODEL>::NV];
    double rho, r;  // r = 1/rho
    MixR mix;       // Allaire only
};
// A face state as the Riemann solver uses it.
template <int MODEL> struct Side {
    double U[ModelTraits<MODEL>::NV];
    double rho, u, p, c;
    MixR mix;  // Allaire only
};

// e > 0 clears 1e-13 (e + ke) for ke = ss/2 by orders of magnitude:
// e 2^bits > ss up to a factor of 2, from the high words alone.
__device__ __forceinline__ bool clear_margin(double e, double ss, int bits) {
    return (int)hi_word(e) + (bits << 20) > (int)hi_word(ss);
}
// x = 0, or x above the snapping threshold (1e-12) of the mutating check.
__device__ __forceinline__ bool unsnapped(double x) {
    return (hi_word(x) - 0x3d720000u < kNumHi - 0x3d720000u) | ((hi_word(x) | lo_word(x)) == 0u);
}

// mix_coeffs
__device__ __forceinline__ bool mix_rn(const Eos& q, double z, MixR& m) {
    const double omz = 1.0 - z;
    bool ok = (q.shared_ok != 0) & num_ok(z) & num_ok(omz);
    m.eps = quot_rn(z, q.gm1_1, q.r1) + quot_rn(omz, q.gm1_2, q.r2);
    double t1 = (z * q.g1) * q.p1;
    if (q.p1 != 0.0) {
        ok &= num_ok(t1);
        t1 = quot_rn(t1, q.gm1_1, q.r1);
    }
    double t2 = (omz * q.g2) * q.p2;
    if (q.p2 != 0.0) {
        ok &= num_ok(t2);
        t2 = quot_rn(t2, q.gm1_2, q.r2);
    }
    const double num = t1 + t2;
    ok &= div_ok(m.eps) & num_ok(num);
    m.ie = rcp_rn(m.eps);
    m.k = quot_rn(num, m.eps, m.ie);
    return ok;
}

// rho c^2 up to the division by rho: the numerator under the root of
// sg_soundspeed and mix_soundspeed.
template <int MODEL>
__device__ __forceinline__ double sound_num(const Eos& q, double p, const MixR& m) {
    if constexpr (MODEL == MODEL_EULER) return q.g1 * (p + q.p1);
    else return m.k + p * (m.ie + 1.0);
}

// The two velocities.  Ahead of a wave the momenta fall off cell by cell until
// they underflow, so tiny ones are common in quiescent gas and are divided in
// place; leaving them to the plain update sent a good part of the segments of
// small grids there.  Huge ones need no test: their squares overflow, and the
// test of e or of the sound speed fails.
__device__ __forceinline__ void velocities_rn(double m, double n, double rho, double r, double& u,
                                              double& v) {
    u = quot_rn(m, rho, r);
    v = quot_rn(n, rho, r);
    if (tiny(m) | tiny(n)) {
        u = div_cold(m, rho);
        v = div_cold(n, rho);
    }
}

// cons_to_prim, with the reference's test of the state.
template <int MODEL>
__device__ __forceinline__ bool c2p_rn(const Eos& q, const double* U, PrimR<MODEL>& P) {
    constexpr int IM = ModelTraits<MODEL>::IM, IE = ModelTraits<MODEL>::IE;
    P.rho = U[0];
    if constexpr (MODEL == MODEL_ALLAIRE) P.rho = U[0] + U[1];
    P.r = rcp_rn(P.rho);
    bool ok = div_ok(P.rho) & pos_ok(U[IE]);
    double u, v;
    velocities_rn(U[IM], U[IM + 1], P.rho, P.r, u, v);
    const double e = quot_rn(U[IE], P.rho, P.r) - (0.5 * ((u * u) + (v * v)));
    ok &= (int)hi_word(e) >= 0;  // e >= 0 (not -0, which the plain test settles)
    P.W[0] = U[0];
    P.W[IM] = u;
    P.W[IM + 1] = v;
    if constexpr (MODEL == MODEL_EULER) {
        P.W[IE] = ((q.gm1_1 * P.rho) * e) - q.gp1;
    } else {
        ok &= mix_rn(q, U[5], P.mix);
        const double re = P.rho * e;
        ok &= num_ok(re) & (U[0] >= 0.0) & (U[1] >= 0.0) & (U[5] >= 0.0) & (U[5] <= 1.0);
        P.W[1] = U[1];
        P.W[IE] = quot_rn(re, P.mix.eps, P.mix.ie) - P.mix.k;
        P.W[5] = U[5];
    }
    return ok;
}

template <int MODEL>
__device__ __forceinline__ bool sound_rn(const Eos& q, const PrimR<MODEL>& P, double& c) {
    const double y = sound_num<MODEL>(q, P.W[ModelTraits<MODEL>::IE], P.mix);
    return sqrt_rn(quot_rn(y, P.rho, P.r), c) & pos_ok(y);
}

// jacobian_times
template <int MODEL>
__device__ __forceinline__ bool jacobian_rn(const Eos& q, const PrimR<MODEL>& P, const double* d,
                                            double s, double* X) {
    const double* W = P.W;
    double c;
    const bool ok = sound_rn<MODEL>(q, P, c);
    if constexpr (MODEL == MODEL_EULER) {
        const double su = s * W[1];
        X[0] = su * d[0] + (s * P.rho) * d[1];
        X[1] = su * d[1] + (s * P.r) * d[3];
        X[2] = su * d[2];
        X[3] = (s * ((P.rho * c) * c)) * d[1] + su * d[3];
    } else {
        const double su = s * W[2];
        X[0] = su * d[0] + (s * W[0]) * d[2];
        X[1] = su * d[1] + (s * W[1]) * d[2];
        X[2] = su * d[2] + (s * P.r) * d[4];
        X[3] = su * d[3];
        X[4] = (s * ((P.rho * c) * c)) * d[2] + su * d[4];
        X[5] = su * d[5];
    }
    return ok;
}

// rp_side of S.U given S.rho, r = 1/S.rho and (Allaire) S.mix.
template <int MODEL>
__device__ __forceinline__ bool side_quotients(const Eos& q, double r, Side<MODEL>& S) {
    constexpr int IM = ModelTraits<MODEL>::IM, IE = ModelTraits<MODEL>::IE;
    const double* U = S.U;
    bool ok = pos_ok(U[IE]);
    double v;
    velocities_rn(U[IM], U[IM + 1], S.rho, r, S.u, v);
    const double e = quot_rn(U[IE], S.rho, r) - (0.5 * ((S.u * S.u) + (v * v)));
    if constexpr (MODEL == MODEL_EULER) {
        S.p = ((q.gm1_1 * S.rho) * e) - q.gp1;
    } else {
        const double re = S.rho * e;
        ok &= num_ok(re);
        S.p = quot_rn(re, S.mix.eps, S.mix.ie) - S.mix.k;
    }
    const double y = sound_num<MODEL>(q, S.p, S.mix);
    return ok & pos_ok(y) & sqrt_rn(quot_rn(y, S.rho, r), S.c);
}

// rp_side of S.U.
template <int MODEL>
__device__ __forceinline__ bool side_from_cons(const Eos& q, Side<MODEL>& S) {
    S.rho = S.U[0];
    if constexpr (MODEL == MODEL_ALLAIRE) S.rho = S.U[0] + S.U[1];
    bool ok = div_ok(S.rho);
    if constexpr (MODEL == MODEL_ALLAIRE) ok &= mix_rn(q, S.U[5], S.mix);
    return ok & side_quotients<MODEL>(q, rcp_rn(S.rho), S);
}

// An evolved face state: prim_to_cons of W, its check, and rp_side of the
// result.  The density, and for Allaire the mixture, of the converted state
// are W's own (nothing is snapped), so the conversions there and back share
// their reciprocals.
template <int MODEL>
__device__ __forceinline__ bool side_from_prim(const Eos& q, const double* W, Side<MODEL>& S) {
    constexpr int IM = ModelTraits<MODEL>::IM, IE = ModelTraits<MODEL>::IE;
    const double u = W[IM], v = W[IM + 1];
    const double ss = (u * u) + (v * v);
    S.rho = W[0];
    if constexpr (MODEL == MODEL_ALLAIRE) S.rho = W[0] + W[1];
    const double r = rcp_rn(S.rho);
    bool ok = div_ok(S.rho);
    double e;
    if constexpr (MODEL == MODEL_EULER) {
        // 1/((gamma - 1) rho) from the two reciprocals, within 2^-51, and one step
        const double x = W[3] + q.gp1, b = q.gm1_1 * S.rho;
        e = quot_rn(x, b, rcp_step(b, r * q.r1));
        if (near_top(b)) e = div_cold(x, b);
        ok &= (q.shared_ok != 0) & pos_ok(x) & div_ok(b);
    } else {
        ok &= mix_rn(q, W[5], S.mix);
        const double x = (W[4] + S.mix.k) * S.mix.eps;
        e = quot_rn(x, S.rho, r);
        ok &= pos_ok(x) & unsnapped(W[0]) & unsnapped(W[1]) & unsnapped(W[5]) & unsnapped(1.0 - W[5]);
        S.U[1] = W[1];
        S.U[5] = W[5];
    }
    S.U[0] = W[0];
    S.U[IM] = S.rho * u;
    S.U[IM + 1] = S.rho * v;
    S.U[IE] = (S.rho * e) + ((0.5 * S.rho) * ss);
    return ok & clear_margin(e, ss, 40) & side_quotients<MODEL>(q, r, S);
}

// Both slope-extrapolated states W + h and W - h (h the half slopes) pass the
// reference's check: densities and pressure bounded from below, speeds from
// above, the energy by a margin that no rounding of the conversion crosses.
template <int MODEL>
__device__ __forceinline__ bool slopes_physical(const Eos& q, const double* W, const double* h) {
    constexpr int IM = ModelTraits<MODEL>::IM, IE = ModelTraits<MODEL>::IE;
    const double um = fabs(W[IM]) + fabs(h[IM]), vm = fabs(W[IM + 1]) + fabs(h[IM + 1]);
    const double ss = __fma_rn(um, um, vm * vm);
    const double p = W[IE] - fabs(h[IE]);
    if constexpr (MODEL == MODEL_EULER) {
        // e = x / (gm1 rho) against ss
        const double x = p + q.gp1, lo = W[0] - fabs(h[0]), up = W[0] + fabs(h[0]);
        return div_ok(lo) & pos_ok(x) & clear_margin(x, (q.gm1_1 * up) * ss, 40);
    } else {
        const double a0 = fabs(h[0]), a1 = fabs(h[1]), a5 = fabs(h[5]);
        const double l0 = W[0] - a0, l1 = W[1] - a1, zl = W[5] - a5, zu = W[5] + a5;
        // rho e = p eps + eps k, linear in z at the lowest pressure: both
        // ends, less 2^-40 of the terms, against rho ss.  2^-14: the snapping
        // of a partial density below 1e-12 may change rho by 2e-6 of it at
        // most where rho > 9.6e-7
        const double A = __fma_rn(q.r2, p, q.c2 - q.cm), B = __fma_rn(q.r1 - q.r2, p, q.c1 - q.c2);
        const double x0 = __fma_rn(zl, B, A), x1 = __fma_rn(zu, B, A);
        const double lo = l0 + l1, b = ((W[0] + a0) + (W[1] + a1)) * ss;
        return (l0 >= 0.0) & (l1 >= 0.0) & (zl >= 0.0) & (zu <= 1.0) & (lo > 9.6e-7) & div_ok(lo) &
               pos_ok(x0) & pos_ok(x1) & clear_margin(x0, b, 14) & clear_margin(x1, b, 14);
    }
}

// hllc_flux.  The wave speeds bracket u* in every ordinary case, so the
// divisors are formed positive, as S_R - u, u - S_L, S_R - u*, u* - S_L and
// the negated denominator of u*; negation is exact.
template <int MODEL>
__device__ __forceinline__ bool hllc_rn(const Eos& q, int wavespeed, const Side<MODEL>& L,
                                        const Side<MODEL>& R, double* F, double& u_star) {
    using T = ModelTraits<MODEL>;
    constexpr int NV = T::NV;
    bool ok = true;
    double SL, SR;
    if (MODEL == MODEL_ALLAIRE && wavespeed == WS_PVRS) {
        const double rho_avg = 0.5 * (L.rho + R.rho);
        const double c_avg = 0.5 * (L.c + R.c);
        const double ppv = smax(0.0, (0.5 * (L.p + R.p)) + (((0.5 * (L.u - R.u)) * rho_avg) * c_avg));
        auto speed = [&](const Side<MODEL>& S) {  // sound speed, or mix_shock_speed_jump
            if (!(ppv > S.p)) return S.c;
            const double pa = 0.5 * (ppv + S.p);
            const double x = (ppv + S.mix.k) + quot_rn(pa, S.mix.eps, S.mix.ie);
            double s;
            ok &= num_ok(pa) & pos_ok(x) & sqrt_rn(quot_rn(x, S.rho, rcp_rn(S.rho)), s);
            return s;
        };
        SL = L.u - speed(L);
        SR = R.u + speed(R);
    } else {
        const double u_avg = 0.5 * (L.u + R.u);
        const double c_avg = 0.5 * (L.c + R.c);
        SL = smin(u_avg - c_avg, L.u - L.c);
        SR = smax(u_avg + c_avg, R.u + R.c);
    }
    const double dSL = SL - L.u, dSR = SR - R.u;
    const double num = ((R.p - L.p) + ((L.rho * L.u) * dSL)) - ((R.rho * R.u) * dSR);
    const double nden = (R.rho * dSR) - (L.rho * dSL);  // the reference's denominator, negated
    double us = quot_rn(-num, nden, rcp_rn(nden));
    if (tiny(num)) us = div_cold(-num, nden);  // as for the velocities
    const bool left = !signbit(us);  // copysign(1.0, u*) == +1
    const double gl = us - SL, gr = SR - us;
    // the side u* selects; per-element selects keep both sides in registers
    double U[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) U[k] = left ? L.U[k] : R.U[k];
    double rho = U[0];
    if constexpr (MODEL == MODEL_ALLAIRE) rho = U[0] + U[1];
    const double u = left ? L.u : R.u, p = left ? L.p : R.p;
    const double g = left ? gl : gr;     // |S - u*|
    const double d = left ? -dSL : dSR;  // |S - u|
    // every divisor above 2^-100, and gl, gr finite below 2^100, which bounds
    // us, SL and SR and so the others; a u* of inf or NaN fails that
    const int low = min(min(min((int)hi_word(gl), (int)hi_word(gr)), min((int)hi_word(-dSL), (int)hi_word(dSR))),
                        (int)hi_word(nden));
    const int high = max(max((int)hi_word(gl), (int)hi_word(gr)), (int)hi_word(nden));
    ok &= (low >= (int)kDivLo) & (high < (int)kDivHi) & abs_ok(p);
    const double fac = quot_rn(d, g, rcp_rn(g));
    double pd = quot_rn(p, d, rcp_rn(d));
    pd = left ? -pd : pd;  // p / (S - u)
    // min(0, S_L) or max(0, S_R)
    const double S = left ? SL : SR;
    const double wave = (left ? SL : -SR) < 0.0 ? S : 0.0;
    double Us[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) Us[k] = fac * U[k];
    Us[T::IM] = (fac * rho) * us;
    Us[T::IE] = fac * (U[T::IE] + ((us - u) * ((rho * us) + pd)));
    double Fp[NV];
    if constexpr (MODEL == MODEL_EULER) {
        Fp[0] = U[0] * u;
        Fp[1] = (U[1] * u) + p;
        Fp[2] = U[2] * u;
        Fp[3] = (U[3] + p) * u;
    } else {
        Fp[0] = U[0] * u;
        Fp[1] = U[1] * u;
        Fp[2] = (U[2] * u) + p;
        Fp[3] = U[3] * u;
        Fp[4] = (U[4] + p) * u;
        Fp[5] = 0.0;
    }
    u_star = us;
#pragma unroll
    for (int k = 0; k < NV; ++k) F[k] = Fp[k] + (wave * (Us[k] - U[k]));
    if constexpr (MODEL == MODEL_ALLAIRE) F[5] = 0.0;
    return ok;
}

// rho E clears |m|^2/2 by 1e-13 of it, more than the rounding of the exact
// test of e >= 0 can amount to.
__device__ __forceinline__ bool surely_energy(double rho, double mu, double mv, double E) {
    return __fma_rn(rho, E, -(0.5 + 1e-13) * __fma_rn(mu, mu, mv * mv)) > 0.0;
}

// wave_speeds of a new state.
template <int MODEL>
__device__ __forceinline__ bool wave_speeds_rn(const Eos& q, const double* U, double& su, double& sv) {
    constexpr int IM = ModelTraits<MODEL>::IM;
    PrimR<MODEL> P;
    double c;
    bool ok = c2p_rn<MODEL>(q, U, P);
    ok &= sound_rn<MODEL>(q, P, c);
    su = fabs(P.W[IM]) + c;
    sv = fabs(P.W[IM + 1]) + c;
    return ok;
}

}  // namespace cfd
