// Mixed-precision split sweeps over a batch of independent solves.
//
// Same numerical method as the plain FP64 path (cfd_physics.cuh and
// cfd_sweep.cuh, which cite the reference) with this precision split:
//   * state: every conserved component stored as an FP32 value plus an FP32
//     compensation word (hi + lo, kept normalised by an error-free sum), so
//     small increments are not lost to FP32 rounding step after step;
//   * reconstruction, slope limiting, the half step and the HLLC solve in
//     FP32 with hardware reciprocal / square-root approximations;
//   * FP64 for the numerator and denominator of the stiffened-gas pressure
//     p = rho e / eps - k of cells with pinf != 0 (pinf up to 6e8 cancels
//     catastrophically in FP32), for the sums of the CFL reduction, for dt
//     and for the time accumulator.
// The face states go to the Riemann solver as primitives, so the pressure
// is never re-derived from a reconstructed FP32 energy.
//
// Batching: one launch sweeps every tile of every active instance.  A tile
// table maps blockIdx to (instance, tile); each instance has its own grid,
// materials, options, buffers and device-resident time state, and its y
// sweep finishes its own wave-speed reduction (last CTA of that instance).
// The batch's y sweep marches strips by default (cfd_march.cuh) and offers
// this tiled form as three alternative shapes with the same results; the x
// sweep uses the warp segments of cfd_march.cuh.  The tiled code is written
// for both directions, but only its y instantiations are launched.
#pragma once

#include "cfd_physics.cuh"
#include "cfd_sweep.cuh"

namespace cfd {
namespace mixed {

// Per-instance descriptor (device memory, one per solve).  The state of a
// cell is stored packed: components 0-3 as one float4 and, for the Allaire
// model, components 4-5 (E, z) as one float2, each with its compensation
// word in a parallel plane, so a cell is read and written with 2 (Euler) or
// 4 (Allaire) vector accesses.
struct Inst {
    float4* q4[2][2];   // [state buffer][0: value, 1: compensation]
    float2* q2[2][2];   // Allaire only
    long long plane;    // cells per plane (pitch * ny)
    int pitch, nx, ny, nv;
    int model, limiter, wavespeed, godunov, fix_dy;
    int bc[4];       // L, R, B, T
    double dx, dy;
    double z_min;
    Eos eos;         // FP64 material parameters
    // FP32 constants of the sweeps (loaded into registers once per tile):
    // g1, p1, g1 - 1, g1 p1, 1/(g1 - 1), 1/(g2 - 1), g1 p1/(g1 - 1), g2 p2/(g2 - 1)
    alignas(16) float pf[8];
    alignas(16) float zf[4];  // z_min and 1 - z_min as value + compensation word
    int flags;       // limiter (bits 0-1), PVRS speeds (2), Godunov (3), stiffened gas (4),
                     // reflective walls L, R, B, T (5-8)
    // FP64 mixture constants for the pressure of stiffened-gas cells:
    // 1/(g1 - 1), 1/(g2 - 1), g1 p1/(g1 - 1), g2 p2/(g2 - 1)
    double pd[4];
    DevState* st;
    double* partials;   // 4 per y tile (marching: per strip part)
    int tiles_x, tiles_y;   // tiles of each sweep
    int max_steps;          // stop after this many steps (and at t >= T)
    int active;             // 0: skip
    int slots, closed;      // marching y sweep: reduction slots in use; the close_steps launch that closes it (0: its last warp)
    int fp64;               // 1: the planes hold FP64 values (fast FP64 form, cfd_fast64.cuh)
};

// One tile of a launch, precomputed on the host when the membership or the
// tile shapes change.
struct alignas(16) TileEnt {
    int inst;          // instance
    int local;         // tile index within the instance
    int a_org, b_org;  // first staged cell along the sweep (halo included), first line
    int len, wid;      // cells along the sweep and lines of the instance
    int max_steps, active;
};

struct MixedArgs {
    Inst* insts;
    const TileEnt* tiles;   // tiles of this launch
    int ntiles;             // tiles of this launch
    int chunk;              // CTA c walks tiles [c * chunk, (c + 1) * chunk) (persistent)
    int rows;               // warp sweeps: rows of a tile
    int split;              // warp sweeps: parts a tile is divided into, a warp each (2^n)
};


// Per-tile constants held in registers (one vector load per tile instead of
// a global load at every use).
struct MPar {
    float g1, p1, gm1, gp1, i1, i2, c1, c2;
    int flags;
    __device__ __forceinline__ int limiter() const { return flags & 3; }
    __device__ __forceinline__ bool pvrs() const { return (flags >> 2) & 1; }
    __device__ __forceinline__ bool godunov() const { return (flags >> 3) & 1; }
    __device__ __forceinline__ bool stiff() const { return (flags >> 4) & 1; }
    // p + p_inf and p + gamma p_inf (no addition for a gas)
    __device__ __forceinline__ float plus_p1(float p) const { return stiff() ? p + p1 : p; }
    __device__ __forceinline__ float plus_gp1(float p) const { return stiff() ? p + gp1 : p; }
};
enum { MF_PVRS = 4, MF_GODUNOV = 8, MF_STIFF = 16, MF_BC = 32 };  // MF_BC << k: wall on side k (L, R, B, T)

__device__ __forceinline__ MPar load_par(const Inst& I) {
    const float4 a = *reinterpret_cast<const float4*>(I.pf);
    const float4 b = *reinterpret_cast<const float4*>(I.pf + 4);
    MPar P;
    P.g1 = a.x; P.p1 = a.y; P.gm1 = a.z; P.gp1 = a.w;
    P.i1 = b.x; P.i2 = b.y; P.c1 = b.z; P.c2 = b.w;
    P.flags = I.flags;
    return P;
}

// Asynchronous global -> shared copies (no registers held while in flight).
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem_dst, const void* gsrc) {
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// FP64 -> FP32 by the conversion alone (with -ftz the cast also tests and
// flushes the result: two more instructions; the results here are pressures,
// densities and steps, far from FP32's denormals, and the FP32 operations on
// them flush one anyway).
__device__ __forceinline__ float to_float(double x) {
    float r;
    asm("cvt.rn.f32.f64 %0, %1;" : "=f"(r) : "d"(x));
    return r;
}
__device__ __forceinline__ float frcp(float x) { return 1.0f / x; }
// Approximate quotient without the operand range scaling of `a / b` (which
// only matters for |b| > 2^126; every divisor here, a density, a pressure,
// a wave speed or a product of them, is many orders of magnitude smaller).
// Measured 3-4 % faster on the sweeps, the same results on every test case.
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }
// sqrt(a / b) for b > 0: the root of the quotient, so that a and b may each take
// FP32's range.  (a rsqrt(a b) is 0 or infinite where the product leaves it; it
// takes 99.0 us a tick of Euler 2048^2 and 96.3 of Allaire 2048x1024, this 99.2
// and 96.9, and that form with a test of its result 98.7 to 100.0 and 101.8 to
// 103.7.)  At least 3e-19, where a is 0 or negative too: a gas of no pressure at
// rest keeps S_L < S_R.
__device__ __forceinline__ float sqrt_ratio(float a, float b) { return sqrtf(fmaxf(1e-37f, fdiv(a, b))); }
// One instruction each (the comparison forms of the reference's std::min and
// std::max take two); a NaN operand gives the other one.
__device__ __forceinline__ float fminf_s(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ float fmaxf_s(float a, float b) { return fmaxf(a, b); }

// The same giving NaN for a NaN operand, for tests that a NaN has to fail.
__device__ __forceinline__ float fmin_n(float a, float b) {
    float r;
    asm("min.NaN.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float fmax_n(float a, float b) {
    float r;
    asm("max.NaN.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// Two FP32 values in one 64-bit register pair: sm_100 adds, multiplies and
// fuses both with one instruction, each rounded as the scalar instruction
// rounds it.  The sweeps are bound by instruction issue, so the component-wise
// parts of the update (slope differences, face states, the compensated sum)
// go through pairs of components.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_get(F2 x, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// y = x over N (even) components, by pairs.
template <int N, class Fn>
__device__ __forceinline__ void pairs(Fn fn) {
#pragma unroll
    for (int q = 0; q < N; q += 2) fn(q);
}

// Mixture coefficients eps(z) = z/(g1-1) + (1-z)/(g2-1) and
// eps k(z) = z g1 p1/(g1-1) + (1-z) g2 p2/(g2-1) in FP32.
__device__ __forceinline__ void mix_f(const MPar& P, float z, float& eps, float& kn) {
    const float omz = 1.0f - z;
    eps = z * P.i1 + omz * P.i2;
    kn = P.stiff() ? z * P.c1 + omz * P.c2 : 0.0f;
}

// Primitive state (rho-split for Allaire: W = rho1 z, rho2 (1-z), u, v, p, z).
template <int MODEL> struct PrimF {
    float W[ModelTraits<MODEL>::NV];
};

// Conserved (hi + lo) -> primitive.  The pressure of a stiffened gas comes
// from the FP64 sum hi + lo.
template <int MODEL>
__device__ __forceinline__ void c2p_mixed(const Inst& I, const MPar& P, const float* hi,
                                          const float* lo, float* W) {
    if constexpr (MODEL == MODEL_EULER) {
        float rho = hi[0];
        float r = frcp(rho);
        float u = hi[1] * r, v = hi[2] * r;
        float p;
        if (!P.stiff()) {
            p = P.gm1 * (hi[3] - 0.5f * (hi[1] * u + hi[2] * v));
        } else {
            double R = (double)hi[0] + (double)lo[0];
            double M1 = (double)hi[1] + (double)lo[1], M2 = (double)hi[2] + (double)lo[2];
            double E = (double)hi[3] + (double)lo[3];
            double re = E - 0.5 * (M1 * M1 + M2 * M2) / R;
            p = to_float(__ldg(&I.eos.gm1_1) * re - __ldg(&I.eos.gp1));
        }
        W[0] = rho;
        W[1] = u;
        W[2] = v;
        W[3] = p;
    } else {
        float rho = hi[0] + hi[1];
        float r = frcp(rho);
        float u = hi[2] * r, v = hi[3] * r;
        float z = hi[5];
        float p;
        if (!P.stiff()) {
            float eps = z * P.i1 + (1.0f - z) * P.i2;
            p = fdiv(hi[4] - 0.5f * (hi[2] * u + hi[3] * v), eps);
        } else {
            // p = (rho e - kn) / eps with rho e = E - |M|^2 / (2 R) and
            // kn = eps k, as (E R - |M|^2/2 - kn R) / (R eps): numerator and
            // denominator in FP64 (the cancellation of p_inf happens in the
            // numerator), the quotient in FP32, the precision of the result
            double R = ((double)hi[0] + (double)lo[0]) + ((double)hi[1] + (double)lo[1]);
            double M1 = (double)hi[2] + (double)lo[2], M2 = (double)hi[3] + (double)lo[3];
            double E = (double)hi[4] + (double)lo[4];
            double zz = (double)hi[5] + (double)lo[5];
            double omz = 1.0 - zz;
            double eps = zz * __ldg(I.pd + 0) + omz * __ldg(I.pd + 1);
            double kn = zz * __ldg(I.pd + 2) + omz * __ldg(I.pd + 3);
            p = fdiv(to_float((E * R - 0.5 * (M1 * M1 + M2 * M2)) - kn * R), to_float(R * eps));
        }
        W[0] = hi[0];
        W[1] = hi[1];
        W[2] = u;
        W[3] = v;
        W[4] = p;
        W[5] = z;
    }
}

// Physical primitive state: the reference's test on the conserved state
// (E/headers/misc_euler.hpp:123-131, A/headers/misc.hpp:228-237) passes,
// i.e. rho >= 0 and e >= 0 (and 0 <= z <= 1, partial densities >= 0).  Its
// e is computed with divisions by rho, so a zero density gives e = NaN and
// fails the test: the density must be strictly positive (a face state of
// zero density taken as physical produced infinite sound speeds and NaN
// fluxes on unlimited slopes at a contact).
template <int MODEL> __device__ __forceinline__ bool phys_prim(const MPar& P, const float* W) {
    if constexpr (MODEL == MODEL_EULER) {
        return W[0] > 0.0f && P.plus_gp1(W[3]) >= 0.0f;
    } else {
        // p + k >= 0  <=>  p eps + kn >= 0 (eps > 0 for 0 <= z <= 1)
        float omz = 1.0f - W[5];
        float eps = W[5] * P.i1 + omz * P.i2, kn = W[5] * P.c1 + omz * P.c2;
        // all six tests evaluated (no short-circuit branches): 2 % faster
        return (W[0] >= 0.0f) & (W[1] >= 0.0f) & (W[0] + W[1] > 0.0f) & (W[5] >= 0.0f) &
               (W[5] <= 1.0f) & (fmaf(W[4], eps, kn) >= 0.0f);
    }
}

// The median of a, b and 0: minmod (the smaller in size where the signs
// agree, else 0) in three instructions: the smaller size with the product's
// sign, clipped at 0, under the sign of a.
__device__ __forceinline__ float median0(float a, float b) {
    float x;
    asm("min.ftz.xorsign.abs.f32 %0, %1, %2;" : "=f"(x) : "f"(a), "f"(b));
    return __int_as_float(__float_as_int(fmaxf(x, 0.0f)) | (__float_as_int(a) & 0x80000000));
}

__device__ __forceinline__ float limit_f(int lim, float a, float b) {
    switch (lim) {
        case LIM_VANLEER:
            return (a * b > 0.0f) ? fdiv(2.0f * a * b, a + b) : 0.0f;
        case LIM_MC:
            return median0(0.5f * (a + b), 2.0f * median0(a, b));
        case LIM_UNLIMITED:
            return 0.5f * (a + b);
        default:
            return median0(a, b);
    }
}

// Limited slopes of all components, d = limit(W - Wm, Wp - W), with the
// limiter chosen once for the cell rather than once per component.
template <int NV>
__device__ __forceinline__ void limit_all(int lim, const float* Wm, const float* W, const float* Wp,
                                          float* d) {
    float a[NV], b[NV];
    pairs<NV>([&](int q) {
        const F2 w = f2(W[q], W[q + 1]);
        f2_get(sub2(w, f2(Wm[q], Wm[q + 1])), a[q], a[q + 1]);
        f2_get(sub2(f2(Wp[q], Wp[q + 1]), w), b[q], b[q + 1]);
    });
    switch (lim) {
        case LIM_VANLEER:
#pragma unroll
            for (int q = 0; q < NV; ++q) d[q] = limit_f(LIM_VANLEER, a[q], b[q]);
            break;
        case LIM_MC:
#pragma unroll
            for (int q = 0; q < NV; ++q) d[q] = limit_f(LIM_MC, a[q], b[q]);
            break;
        case LIM_UNLIMITED:
#pragma unroll
            for (int q = 0; q < NV; ++q) d[q] = limit_f(LIM_UNLIMITED, a[q], b[q]);
            break;
        default:
#pragma unroll
            for (int q = 0; q < NV; ++q) d[q] = limit_f(LIM_MINMOD, a[q], b[q]);
    }
}

// Sound speed of a primitive state.
template <int MODEL> __device__ __forceinline__ float sound_f(const MPar& P, const float* W) {
    if constexpr (MODEL == MODEL_EULER) {
        return sqrt_ratio(P.g1 * P.plus_p1(W[3]), W[0]);
    } else {
        // c^2 = (k + p (1/eps + 1)) / rho = (kn + p (1 + eps)) / (eps rho)
        float omz = 1.0f - W[5];
        float eps = W[5] * P.i1 + omz * P.i2, kn = W[5] * P.c1 + omz * P.c2;
        float rho = W[0] + W[1];
        return sqrt_ratio(fmaf(W[4], 1.0f + eps, kn), eps * rho);
    }
}

// Half-step evolution X = (0.5 dt/dx) A(W) d (primitive Jacobian), rho c^2
// without the root and the division by rho that c itself would take.
template <int MODEL>
__device__ __forceinline__ void jac_f(const MPar& P, const float* W, const float* d, float s,
                                      float* X) {
    if constexpr (MODEL == MODEL_EULER) {
        const float rho = W[0], u = W[1];
        const float rc2 = fmaxf(0.0f, P.g1 * P.plus_p1(W[3]));
        X[0] = s * (u * d[0] + rho * d[1]);
        X[1] = s * (u * d[1] + frcp(rho) * d[3]);
        X[2] = s * (u * d[2]);
        X[3] = s * (rc2 * d[1] + u * d[3]);
    } else {
        const float rho = W[0] + W[1], u = W[2];
        float eps, kn;
        mix_f(P, W[5], eps, kn);
        const float rc2 = fmaxf(0.0f, fdiv(fmaf(W[4], 1.0f + eps, kn), eps));
        X[0] = s * (u * d[0] + W[0] * d[2]);
        X[1] = s * (u * d[1] + W[1] * d[2]);
        X[2] = s * (u * d[2] + frcp(rho) * d[4]);
        X[3] = s * (u * d[3]);
        X[4] = s * (rc2 * d[2] + u * d[4]);
        X[5] = s * (u * d[5]);
    }
}

// Evolved face states of a cell, Wp (high face) and Wm (low face), from its
// slopes d, and whether the reference would use them: each needs its
// slope-extrapolated state and its evolved state physical
// (E/headers/flux_solver_MUSCLhancock.hpp:178-223).  Where the smallest
// values of all four states pass, all pass; only otherwise are they tested one
// by one (for the mixture a pressure >= 0 is sufficient, eps k being >= 0).
template <int MODEL>
__device__ __forceinline__ void face_states(const MPar& P, const float* W, const float* d, float s,
                                            float* Wp, float* Wm, bool& okp, bool& okm) {
    constexpr int NV = ModelTraits<MODEL>::NV;
    float E[NV], D[NV], X[NV];  // slope-extrapolated states (high, low), half step
    jac_f<MODEL>(P, W, d, s, X);
    const F2 half = f2(0.5f, 0.5f), mhalf = f2(-0.5f, -0.5f);
    pairs<NV>([&](int q) {
        const F2 w = f2(W[q], W[q + 1]), dq = f2(d[q], d[q + 1]), x = f2(X[q], X[q + 1]);
        const F2 e = fma2(half, dq, w), m = fma2(mhalf, dq, w);
        f2_get(e, E[q], E[q + 1]);
        f2_get(m, D[q], D[q + 1]);
        f2_get(sub2(e, x), Wp[q], Wp[q + 1]);
        f2_get(sub2(m, x), Wm[q], Wm[q + 1]);
    });
    bool all;
    auto least = [&](int q) {  // the smallest of component q over the four states
        return fmin_n(fmin_n(E[q], D[q]), fmin_n(Wp[q], Wm[q]));
    };
    if constexpr (MODEL == MODEL_EULER) {
        all = (least(0) > 0.0f) & (P.plus_gp1(least(3)) >= 0.0f);
    } else {
        const float zm = fmax_n(fmax_n(E[5], D[5]), fmax_n(Wp[5], Wm[5]));
        const float r1 = least(0), r2 = least(1);
        all = (fmin_n(fmin_n(r1, r2), fmin_n(least(4), least(5))) >= 0.0f) & (zm <= 1.0f) &
              (r1 + r2 > 0.0f);
    }
    okp = okm = all;
    if (!all) {
        okp = phys_prim<MODEL>(P, E) && phys_prim<MODEL>(P, Wp);
        okm = phys_prim<MODEL>(P, D) && phys_prim<MODEL>(P, Wm);
    }
}

// (Multiply-adds beside terms that vanish for a gas are written as fmaf: where
// a launch's options make such a term a constant 0, the compiler would
// otherwise contract the rest differently, and a member's bits would depend on
// its company.)
//
// HLLC flux from primitive face states (same wave-speed estimates and star
// states as hllc_flux in cfd_physics.cuh), F[NV] = u*, F[NV+1] = z* (Allaire).
// With the star factor f = (S - u)/(S - u*), the passive components' flux
// U u + w (f U - U) is U A with A = u + w (f - 1), w the selected wave speed
// clipped at 0, and p/(S - u) enters the energy as f p/(S - u) = p/(S - u*),
// so one reciprocal serves both.
template <int MODEL>
__device__ __forceinline__ void hllc_prim(const MPar& P, const float* WL, const float* WR,
                                          float* F) {
    using T = ModelTraits<MODEL>;
    constexpr int NV = T::NV;
    float rL, rR, uL, uR, pL, pR, cL, cR, epsL = 1.f, knL = 0.f, epsR = 1.f, knR = 0.f;
    float qL = 1.f, qR = 1.f;  // eps rho
    if constexpr (MODEL == MODEL_EULER) {
        rL = WL[0]; uL = WL[1]; pL = WL[3];
        rR = WR[0]; uR = WR[1]; pR = WR[3];
        cL = sqrt_ratio(P.g1 * P.plus_p1(pL), rL);
        cR = sqrt_ratio(P.g1 * P.plus_p1(pR), rR);
    } else {
        rL = WL[0] + WL[1]; uL = WL[2]; pL = WL[4];
        rR = WR[0] + WR[1]; uR = WR[2]; pR = WR[4];
        mix_f(P, WL[5], epsL, knL);
        mix_f(P, WR[5], epsR, knR);
        qL = epsL * rL;
        qR = epsR * rR;
        cL = sqrt_ratio(fmaf(pL, 1.0f + epsL, knL), qL);
        cR = sqrt_ratio(fmaf(pR, 1.0f + epsR, knR), qR);
    }
    float SL, SR;
    if (MODEL == MODEL_ALLAIRE && P.pvrs()) {
        const float ra = 0.5f * (rL + rR), ca = 0.5f * (cL + cR);
        const float ppv = fmaxf(0.0f, 0.5f * (pL + pR) + 0.5f * (uL - uR) * ra * ca);
        // shock_speed_jump: sqrt(((p* + k) + ((p* + p)/2)/eps) / rho)
        SL = uL - (ppv > pL ? sqrt_ratio(fmaf(ppv, epsL, fmaf(0.5f, ppv + pL, knL)), qL) : cL);
        SR = uR + (ppv > pR ? sqrt_ratio(fmaf(ppv, epsR, fmaf(0.5f, ppv + pR, knR)), qR) : cR);
    } else {
        const float ua = 0.5f * (uL + uR), ca = 0.5f * (cL + cR);
        SL = fminf(ua - ca, uL - cL);
        SR = fmaxf(ua + ca, uR + cR);
    }
    const float dSL = SL - uL, dSR = SR - uR;
    const float mL = rL * dSL, mR = rR * dSR;
    const float us = fdiv((pR - pL) + mL * uL - mR * uR, mL - mR);
    const bool left = !signbit(us);
    // per-element selects (a pointer to either side would put both in local memory)
    const float rho = left ? rL : rR, u = left ? uL : uR, p = left ? pL : pR;
    const float Sk = left ? SL : SR, dS = left ? dSL : dSR;
    const float wave = left ? fminf(0.0f, SL) : fmaxf(0.0f, SR);
    const float v = left ? WL[T::IT] : WR[T::IT];
    const float inv = frcp(Sk - us);
    const float fac = dS * inv;
    const float A = u + wave * (fac - 1.0f);
    float re;  // rho e
    if constexpr (MODEL == MODEL_EULER) {
        re = P.plus_gp1(p) * P.i1;
    } else {
        const float eps = left ? epsL : epsR, kn = left ? knL : knR;
        re = fmaf(p, eps, kn);
    }
    const float E = fmaf(0.5f * rho, fmaf(u, u, v * v), re);
    const float m = rho * A;
    if constexpr (MODEL == MODEL_EULER) {
        F[0] = m;
    } else {
        F[0] = (left ? WL[0] : WR[0]) * A;
        F[1] = (left ? WL[1] : WR[1]) * A;
        F[5] = 0.0f;
    }
    F[T::IM] = rho * (u * u + wave * (fac * us - u)) + p;
    F[T::IT] = m * v;
    F[T::IE] = E * A + p * u + (wave * (us - u)) * (fac * rho * us + p * inv);
    F[NV] = us;
    if constexpr (MODEL == MODEL_ALLAIRE) F[NV + 1] = left ? WL[5] : WR[5];
}

// Whether an updated Euler state is sure to keep rho > 0 and rho e > 0
// (p + gamma p_inf > 0): rho E clears |m|^2/2 by more than its rounding.
// Otherwise the caller converts the state and tests it as the reference does.
__device__ __forceinline__ bool euler_sure(const float* h) {
    return (h[0] > 1e-12f) & (h[0] * h[3] > 0.500001f * (h[1] * h[1] + h[2] * h[2]));
}

// hi + lo += d with an error-free transformation (TwoSum), keeping the pair
// normalised.
__device__ __forceinline__ void comp_add(float& hi, float& lo, float d) {
    float y = lo + d;
    float s = hi + y;
    float bp = s - hi;
    float e = (hi - (s - bp)) + (y - bp);
    hi = s;
    lo = e;
}

// The same for a pair, d = k (a - b).
__device__ __forceinline__ void comp_add2(float* hi, float* lo, F2 k, F2 a, F2 b) {
    const F2 h = f2(hi[0], hi[1]);
    const F2 y = fma2(k, sub2(a, b), f2(lo[0], lo[1]));
    const F2 s = add2(h, y);
    const F2 bp = sub2(s, h);
    const F2 e = add2(sub2(h, sub2(s, bp)), sub2(y, bp));
    f2_get(s, hi[0], hi[1]);
    f2_get(e, lo[0], lo[1]);
}
// The conservative update of a cell from the fluxes at its two faces (all
// components; the caller sets Allaire's z, whose flux is 0).
template <int NV>
__device__ __forceinline__ void comp_update(float* h, float* l, float k, const float* FL, const float* FR) {
    const F2 kk = f2(k, k);
    pairs<NV>([&](int q) {
        if (NV == 6 && q == 4) {  // E alone: z has its own update
            comp_add(h[4], l[4], k * (FL[4] - FR[4]));
            return;
        }
        comp_add2(h + q, l + q, kk, f2(FL[q], FL[q + 1]), f2(FR[q], FR[q + 1]));
    });
}

// The planes of one state buffer of a member, held in registers: the stores
// of a sweep go through pointers the compiler cannot tell apart from the
// member descriptor, so reading the descriptor's pointers again after every
// store would cost a global load each time.
struct MPlanes {
    float4 *v4, *c4;  // components 0-3: value, compensation
    float2 *v2, *c2;  // Allaire E, z: value, compensation
};

template <int MODEL>
__device__ __forceinline__ MPlanes mplanes(const Inst& I, int buf) {
    MPlanes q;
    q.v4 = I.q4[buf][0];
    q.c4 = I.q4[buf][1];
    q.v2 = MODEL == MODEL_ALLAIRE ? I.q2[buf][0] : nullptr;
    q.c2 = MODEL == MODEL_ALLAIRE ? I.q2[buf][1] : nullptr;
    return q;
}

template <int MODEL, class Off>
__device__ __forceinline__ void load_cell(const MPlanes& Q, Off off, float* h, float* l) {
    float4 a = __ldg(Q.v4 + off), b = __ldg(Q.c4 + off);
    h[0] = a.x; h[1] = a.y; h[2] = a.z; h[3] = a.w;
    l[0] = b.x; l[1] = b.y; l[2] = b.z; l[3] = b.w;
    if constexpr (MODEL == MODEL_ALLAIRE) {
        float2 c = __ldg(Q.v2 + off), d = __ldg(Q.c2 + off);
        h[4] = c.x; h[5] = c.y;
        l[4] = d.x; l[5] = d.y;
    }
}

template <int MODEL, class Off>
__device__ __forceinline__ void store_cell(const MPlanes& Q, Off off, const float* h, const float* l) {
    Q.v4[off] = make_float4(h[0], h[1], h[2], h[3]);
    Q.c4[off] = make_float4(l[0], l[1], l[2], l[3]);
    if constexpr (MODEL == MODEL_ALLAIRE) {
        Q.v2[off] = make_float2(h[4], h[5]);
        Q.c2[off] = make_float2(l[4], l[5]);
    }
}

template <int MODEL> __device__ __forceinline__ void load_cell(const Inst& I, int buf,
                                                               long long off, float* h, float* l) {
    load_cell<MODEL>(mplanes<MODEL>(I, buf), off, h, l);
}

// The clip of the updated volume fraction to [z_min, 1 - z_min] on a
// compensated z (value h, compensation l).
__device__ __forceinline__ void clip_z(const Inst& I, float& h, float& l) {
    const float4 b = __ldg(reinterpret_cast<const float4*>(I.zf));
    if (h + l < b.x) { h = b.x; l = b.y; }
    if (h + l > b.z) { h = b.z; l = b.w; }
}

template <int MODEL> __device__ __forceinline__ void store_cell(const Inst& I, int buf,
                                                                long long off, const float* h,
                                                                const float* l) {
    store_cell<MODEL>(mplanes<MODEL>(I, buf), off, h, l);
}

// Shared-memory vectors: one float4 (+ one float2 for Allaire) per slot.
template <int MODEL> struct SVec {
    float4* v4;
    float2* v2;
    __device__ __forceinline__ void put(int s, const float* x) const {
        v4[s] = make_float4(x[0], x[1], x[2], x[3]);
        if constexpr (MODEL == MODEL_ALLAIRE) v2[s] = make_float2(x[4], x[5]);
    }
    __device__ __forceinline__ void get(int s, float* x) const {
        float4 a = v4[s];
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        if constexpr (MODEL == MODEL_ALLAIRE) {
            float2 b = v2[s];
            x[4] = b.x; x[5] = b.y;
        }
    }
};

template <int MODEL, int DIR, int TS, int NA>
struct MTile {
    static constexpr int NV = ModelTraits<MODEL>::NV;
    static constexpr int LA = TS + 4;
    static constexpr int NSLOT = LA * NA;
    static constexpr int ST = (DIR == DIR_X) ? 1 : NA;
    static constexpr int VB = (MODEL == MODEL_ALLAIRE) ? 24 : 16;  // bytes of one vector
    static_assert(NSLOT == 256, "one staged cell per thread");
    __device__ static __forceinline__ int slot(int a, int b) {
        return (DIR == DIR_X) ? b * LA + a : a * NA + b;
    }
    __device__ static __forceinline__ void item(int i, int a0, int cnt, int& a, int& b) {
        if (DIR == DIR_X) {
            b = i / cnt;
            a = a0 + i - b * cnt;
        } else {
            a = a0 + i / NA;
            b = i - (i / NA) * NA;
        }
    }
    // vectors per slot: value, compensation, W, W+, W-, flux; u*, z*; flags;
    // then the staging area the next tile's cells are copied into
    // (value and compensation, slot = thread)
    static constexpr int STG = (6 * VB * NSLOT + 8 * NSLOT + NSLOT + 15) / 16 * 16;
    static constexpr int SMEM = STG + 2 * VB * NSLOT;
};

// Where a tile lies and whether it is skipped.
struct TileGeom {
    int inst, ltile, a_org, b_org, len, wid, cur;
    bool skip;
};

template <int DIR, int TS, int NA>
__device__ __forceinline__ TileGeom tile_geom(const MixedArgs& A, int tile) {
    const int4* e = reinterpret_cast<const int4*>(A.tiles + tile);
    const int4 e0 = e[0], e1 = e[1];
    TileGeom g;
    g.inst = e0.x;
    g.ltile = e0.y;
    g.a_org = e0.z;
    g.b_org = e0.w;
    g.len = e1.x;
    g.wid = e1.y;
    const DevState* st = A.insts[g.inst].st;
    g.skip = !e1.w || st->done || st->n >= e1.z;
    g.cur = st->cur;
    return g;
}

// Starts copying this thread's staged cell of a tile (the boundary mirror
// of pre_sweep picks the source cell) into its staging slot.
template <int MODEL, int DIR, int TS, int NA>
__device__ __forceinline__ void tile_issue(const MixedArgs& A, const TileGeom& g, char* smem) {
    using Tl = MTile<MODEL, DIR, TS, NA>;
    const Inst& I = A.insts[g.inst];
    int a, b;
    Tl::item(threadIdx.x, 0, Tl::LA, a, b);
    const int ga = g.a_org + a, gb = g.b_org + b;
    int src = ga;
    if (ga < 0) src = -ga - 1;
    else if (ga >= g.len) src = 2 * g.len - 1 - ga;
    src = min(max(src, 0), g.len - 1);
    const int gbs = min(gb, g.wid - 1);
    const long long off =
        (DIR == DIR_X) ? (long long)gbs * I.pitch + src : (long long)src * I.pitch + gbs;
    const int buf = g.cur ^ (DIR == DIR_Y);
    char* stg = smem + Tl::STG;
    const int t = threadIdx.x;
    cp_async16(stg + 16 * t, I.q4[buf][0] + off);
    cp_async16(stg + 16 * (Tl::NSLOT + t), I.q4[buf][1] + off);
    if constexpr (MODEL == MODEL_ALLAIRE) {
        cp_async8(stg + 32 * Tl::NSLOT + 8 * t, I.q2[buf][0] + off);
        cp_async8(stg + 40 * Tl::NSLOT + 8 * t, I.q2[buf][1] + off);
    }
    cp_async_commit();
}

// Per-thread wave-speed maxima and mass sums of the tiles of a run.
struct RAcc {
    float mu, mv;
    double m1, m2;
};

template <int MODEL, int DIR, int TS, int NA>
__device__ __forceinline__ void mixed_tile(const MixedArgs& A, const TileGeom& g, int next_tile,
                                           char* smem, RAcc& racc, TileGeom& s_next,
                                           float* s_coef) {
    using Tl = MTile<MODEL, DIR, TS, NA>;
    using MT = ModelTraits<MODEL>;
    constexpr int NV = MT::NV, LA = Tl::LA, NSLOT = Tl::NSLOT, ST = Tl::ST;
    const int tid = threadIdx.x;
    auto vec = [&](int k) {
        SVec<MODEL> v;
        v.v4 = reinterpret_cast<float4*>(smem + k * Tl::VB * NSLOT);
        v.v2 = reinterpret_cast<float2*>(smem + k * Tl::VB * NSLOT + 16 * NSLOT);
        return v;
    };
    const SVec<MODEL> sH = vec(0), sL = vec(1), sW = vec(2), sP = vec(3), sM = vec(4), sF = vec(5);
    float2* sUZ = reinterpret_cast<float2*>(smem + 6 * Tl::VB * NSLOT);
    unsigned char* sFl = reinterpret_cast<unsigned char*>(smem + 6 * Tl::VB * NSLOT + 8 * NSLOT);

    const Inst& I = A.insts[g.inst];
    const MPar P = load_par(I);
    // CTA-wide values of this tile, made once by thread 0 during P1 (shared
    // memory): the sweep's coefficients and the geometry of the next tile
    if (tid == 0) {
        const double dt = I.st->dt;
        const double h_flux = (DIR == DIR_X) ? I.dx : (I.fix_dy ? I.dy : I.dx);
        const double h_upd = (DIR == DIR_X) ? I.dx : I.dy;
        s_coef[0] = (float)(0.5 * (dt / h_flux));
        s_coef[1] = (float)(dt / h_upd);
        TileGeom t;
        if (next_tile < A.ntiles) {
            t = tile_geom<DIR, TS, NA>(A, next_tile);
        } else {
            t.inst = -1;
            t.skip = true;
        }
        s_next = t;
    }

    // ---- P1: boundary sign, rotation, conversion of the fetched cell -------
    {
        int a, b;
        Tl::item(tid, 0, LA, a, b);
        float h[NV], l[NV];
        cp_async_wait_all();
        {
            const char* stg = smem + Tl::STG;
            const float4 x = *reinterpret_cast<const float4*>(stg + 16 * tid);
            const float4 y = *reinterpret_cast<const float4*>(stg + 16 * (NSLOT + tid));
            h[0] = x.x; h[1] = x.y; h[2] = x.z; h[3] = x.w;
            l[0] = y.x; l[1] = y.y; l[2] = y.z; l[3] = y.w;
            if constexpr (MODEL == MODEL_ALLAIRE) {
                const float2 z = *reinterpret_cast<const float2*>(stg + 32 * NSLOT + 8 * tid);
                const float2 w = *reinterpret_cast<const float2*>(stg + 40 * NSLOT + 8 * tid);
                h[4] = z.x; h[5] = z.y;
                l[4] = w.x; l[5] = w.y;
            }
        }
        const int ga = g.a_org + a;
        const int wall_lo = (DIR == DIR_X) ? 0 : 2;
        const bool neg = (ga < 0 && ((P.flags >> (5 + wall_lo)) & 1)) ||
                         (ga >= g.len && ((P.flags >> (6 + wall_lo)) & 1));
        if (DIR == DIR_X) {
            if (neg) { h[MT::IM] = -h[MT::IM]; l[MT::IM] = -l[MT::IM]; }
        } else {
            if (neg) { h[MT::IT] = -h[MT::IT]; l[MT::IT] = -l[MT::IT]; }
            float t = h[MT::IM], tl = l[MT::IM];
            h[MT::IM] = h[MT::IT]; l[MT::IM] = l[MT::IT];
            h[MT::IT] = -t; l[MT::IT] = -tl;
        }
        int s = Tl::slot(a, b);
        float W[NV];
        c2p_mixed<MODEL>(I, P, h, l, W);
        sH.put(s, h);
        sL.put(s, l);
        sW.put(s, W);
    }
    __syncthreads();
    // the staging slot is free: start copying this thread's cell of the next tile
    {
        const TileGeom gn = s_next;
        if (!gn.skip) tile_issue<MODEL, DIR, TS, NA>(A, gn, smem);
    }
    const float s_half = s_coef[0];
    const float k_upd = s_coef[1];

    // ---- P2: slopes and evolved face states (primitive) ----------------
    if (!P.godunov() && tid < (LA - 2) * NA) {
        int a, b;
        Tl::item(tid, 1, LA - 2, a, b);
        int s = Tl::slot(a, b);
        float W[NV], Wl[NV], Wr[NV], d[NV], Wp[NV], Wm[NV];
        sW.get(s, W);
        sW.get(s - ST, Wl);
        sW.get(s + ST, Wr);
        limit_all<NV>(P.limiter(), Wl, W, Wr, d);
        bool okp, okm;
        face_states<MODEL>(P, W, d, s_half, Wp, Wm, okp, okm);
        sP.put(s, Wp);
        sM.put(s, Wm);
        sFl[s] = (unsigned char)((okp ? 1 : 0) | (okm ? 2 : 0));
    }
    __syncthreads();

    // ---- P3: HLLC per face -------------------------------------------------
    if (tid < (TS + 1) * NA) {
        int a, b;
        Tl::item(tid, 2, TS + 1, a, b);
        int sR = Tl::slot(a, b), sL = sR - ST;
        float WL[NV], WR[NV];
        bool first = true;
        if (!P.godunov()) {
            unsigned fL = sFl[sL], fR = sFl[sR];
            // zero slopes evolve to the cell state itself; the first-order
            // fallback uses the cell states too
            if ((fL & 1u) && (fR & 2u)) {
                first = false;
                sP.get(sL, WL);
                sM.get(sR, WR);
            }
        }
        if (first) {
            sW.get(sL, WL);
            sW.get(sR, WR);
        }
        float F[NV + 2];
        hllc_prim<MODEL>(P, WL, WR, F);
        sF.put(sR, F);
        sUZ[sR] = make_float2(F[NV], MODEL == MODEL_ALLAIRE ? F[NV + 1] : 0.0f);
    }
    __syncthreads();

    // ---- P4: compensated update, store, reduce -----------------------------
    float r_mu = 0.0f, r_mv = 0.0f;
    double r_m1 = 0.0, r_m2 = 0.0;
    if (tid < TS * NA) {
        int a, b;
        Tl::item(tid, 2, TS, a, b);
        int ga = g.a_org + a, gb = g.b_org + b;
        if (ga < g.len && gb < g.wid) {
            int s = Tl::slot(a, b);
            float hh[NV], ll[NV];
            sH.get(s, hh);
            sL.get(s, ll);
            {
                float FL[NV], FR[NV];
                sF.get(s, FL);
                sF.get(s + ST, FR);
                comp_update<NV>(hh, ll, k_upd, FL, FR);
            }
            if constexpr (MODEL == MODEL_ALLAIRE) {
                float2 uzL = sUZ[s], uzR = sUZ[s + ST];
                float usL = uzL.x, usR = uzR.x, zsL = uzL.y, zsR = uzR.y;
                float z = hh[5];
                float dz;
                if (P.godunov()) {
                    float zL = sH.v2[s - ST].y, zR = sH.v2[s + ST].y;
                    dz = -k_upd * ((zR - z) * fminf_s(0.0f, usR) + (z - zL) * fmaxf_s(0.0f, usL));
                } else {
                    dz = -k_upd * ((usR * zsR - usL * zsL) - z * (usR - usL));
                }
                comp_add(hh[5], ll[5], dz);
                clip_z(I, hh[5], ll[5]);
                if (hh[0] < 0.0f) { hh[0] = 0.0f; ll[0] = 0.0f; }
                if (hh[1] < 0.0f) { hh[1] = 0.0f; ll[1] = 0.0f; }
            }
            if (DIR == DIR_Y) {  // rotate back
                float t = hh[MT::IM], tl = ll[MT::IM];
                hh[MT::IM] = -hh[MT::IT]; ll[MT::IM] = -ll[MT::IT];
                hh[MT::IT] = t; ll[MT::IT] = tl;
            }
            float Wn[NV];
            c2p_mixed<MODEL>(I, P, hh, ll, Wn);
            if constexpr (MODEL == MODEL_EULER) {
                // density / energy restore as in the plain form (rare)
                if (!(hh[0] > 1e-12f) || !(P.plus_gp1(Wn[3]) > 0.0f)) {
                    float oh[NV], ol[NV], Wo[NV];  // the cell before the update
                    sH.get(s, oh);
                    sL.get(s, ol);
                    if (DIR == DIR_Y) {
                        float t2 = oh[MT::IM], t2l = ol[MT::IM];
                        oh[MT::IM] = -oh[MT::IT]; ol[MT::IM] = -ol[MT::IT];
                        oh[MT::IT] = t2; ol[MT::IT] = t2l;
                    }
                    c2p_mixed<MODEL>(I, P, oh, ol, Wo);
                    float rho = hh[0] > 1e-12f ? hh[0] : oh[0];
                    float u = Wn[1], v = Wn[2];
                    float p = (P.plus_gp1(Wn[3]) > 0.0f) ? Wn[3] : Wo[3];
                    hh[0] = rho; ll[0] = 0.f;
                    hh[1] = rho * u; ll[1] = 0.f;
                    hh[2] = rho * v; ll[2] = 0.f;
                    hh[3] = P.plus_gp1(p) * P.i1 + 0.5f * rho * (u * u + v * v); ll[3] = 0.f;
                    Wn[0] = rho;
                    Wn[3] = p;
                }
            }
            long long off = (DIR == DIR_X) ? (long long)gb * I.pitch + ga : (long long)ga * I.pitch + gb;
            store_cell<MODEL>(I, g.cur ^ (DIR == DIR_X), off, hh, ll);
            if (DIR == DIR_Y) {
                float c = sound_f<MODEL>(P, Wn);
                r_mu = fabsf(Wn[MT::IM]) + c;
                r_mv = fabsf(Wn[MT::IT]) + c;
                r_m1 = (double)hh[0] + (double)ll[0];
                if constexpr (MODEL == MODEL_ALLAIRE) r_m2 = (double)hh[1] + (double)ll[1];
            }
        }
    }
    if constexpr (DIR == DIR_Y) {  // this thread's wave speeds and masses
        racc.mu = fmaxf_s(racc.mu, r_mu);  // max of FP32 speeds: exact in FP32
        racc.mv = fmaxf_s(racc.mv, r_mv);
        racc.m1 += r_m1;
        racc.m2 += r_m2;
    }
}

// End of the run of an instance's tiles processed by this CTA (y sweep):
// block-reduce the run's wave speeds and masses into the instance's partial
// slot, count the run's tiles, and let the CTA that completes the count pick
// the instance's dt.  CTA c walks the contiguous tile range
// [c * chunk, (c + 1) * chunk), so it meets an instance (tiles [t0, t0 + n))
// in at most one run, and the CTAs that do are c0 = t0 / chunk ..
// (t0 + n - 1) / chunk: slot c - c0 is written exactly once per sweep.
__device__ __forceinline__ void flush_run(const MixedArgs& A, int inst, int slot, int nslots,
                                          int count, RAcc& racc, double dt) {
    const Inst& I = A.insts[inst];
    DevState* st = I.st;
    __shared__ double red[4][8];
    __shared__ bool is_last;
    const int tid = threadIdx.x;
    double mu = (double)racc.mu, mv = (double)racc.mv, m1 = racc.m1, m2 = racc.m2;
    for (int o = 16; o > 0; o >>= 1) {
        mu = smax(mu, __shfl_down_sync(0xffffffffu, mu, o));
        mv = smax(mv, __shfl_down_sync(0xffffffffu, mv, o));
        m1 += __shfl_down_sync(0xffffffffu, m1, o);
        m2 += __shfl_down_sync(0xffffffffu, m2, o);
    }
    if ((tid & 31) == 0) {
        red[0][tid >> 5] = mu;
        red[1][tid >> 5] = mv;
        red[2][tid >> 5] = m1;
        red[3][tid >> 5] = m2;
    }
    __syncthreads();
    if (tid == 0) {
        mu = red[0][0], mv = red[1][0], m1 = red[2][0], m2 = red[3][0];
        for (int w = 1; w < 8; ++w) {
            mu = smax(mu, red[0][w]);
            mv = smax(mv, red[1][w]);
            m1 += red[2][w];
            m2 += red[3][w];
        }
        double* p = I.partials + 4 * slot;
        p[0] = mu;
        p[1] = mv;
        p[2] = m1;
        p[3] = m2;
        __threadfence();
        unsigned t = atomicAdd(&st->ticket, (unsigned)count);
        is_last = (t + (unsigned)count == (unsigned)I.tiles_y);
    }
    __syncthreads();
    if (is_last) {
        __threadfence();
        finish_reduction(st, I.partials, nslots, 1, dt, 0);
    }
    racc.mu = racc.mv = 0.0f;
    racc.m1 = racc.m2 = 0.0;
}

// Persistent sweep: a fixed grid of CTAs walks the tile list of every
// instance in the launch; each thread loads its cell of the next tile while
// the current tile is being computed.
// Resident CTAs per SM: 3 for the y sweeps the batch launches (4 would suit
// the Euler x form, which the batch does not launch).
template <int MODEL, int DIR, int TS, int NA>
__global__ void __launch_bounds__(256, (MODEL == MODEL_EULER && DIR == DIR_X) ? 4 : 3)
    mixed_sweep_kernel(MixedArgs A) {
    extern __shared__ __align__(16) char msm[];
    __shared__ TileGeom s_next;
    __shared__ float s_coef[2];
    const int t_begin = blockIdx.x * A.chunk;
    const int t_end = min(t_begin + A.chunk, A.ntiles);
    if (t_begin >= t_end) return;
    TileGeom g = tile_geom<DIR, TS, NA>(A, t_begin);
    if (!g.skip) tile_issue<MODEL, DIR, TS, NA>(A, g, msm);
    RAcc racc{0.0f, 0.0f, 0.0, 0.0};
    int run_first = t_begin, run_count = 0;
    for (int tile = t_begin; tile < t_end; ++tile) {
        int next = tile + 1 < t_end ? tile + 1 : A.ntiles;  // A.ntiles: none
        const int inst = g.inst;
        TileGeom gn;
        gn.inst = -1;
        gn.skip = true;
        if (!g.skip) {
            mixed_tile<MODEL, DIR, TS, NA>(A, g, next, msm, racc, s_next, s_coef);
            ++run_count;
            gn = s_next;
        } else if (next < A.ntiles) {
            gn = tile_geom<DIR, TS, NA>(A, next);
            if (!gn.skip) tile_issue<MODEL, DIR, TS, NA>(A, gn, msm);
        }
        bool run_ends = next >= A.ntiles || gn.inst != inst;
        if (DIR == DIR_Y && run_ends && run_count > 0) {
            int t0 = run_first - A.tiles[run_first].local;  // first tile of the instance
            int c0 = t0 / A.chunk;
            int nslots = (t0 + A.insts[inst].tiles_y - 1) / A.chunk - c0 + 1;
            flush_run(A, inst, (int)blockIdx.x - c0, nslots, run_count, racc,
                      A.insts[inst].st->dt);
        }
        if (run_ends) {
            run_count = 0;
            run_first = next;
        }
        g = gn;
        __syncthreads();  // shared memory is reused by the next tile
    }
    cp_async_wait_all();
}

}  // namespace mixed
}  // namespace cfd
