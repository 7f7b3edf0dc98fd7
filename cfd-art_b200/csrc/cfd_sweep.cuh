// Directional sweep kernels of the split finite-volume update (plain FP64).
//
// One launch updates every interior cell along one direction:
//   x-sweep  E/sourcecode/euler_rowsweep.cpp:10-95,
//            A/sourcecode/allaire_diffuse_rowsweep.cpp:10-52
//   y-sweep  E/sourcecode/euler_colsweep.cpp:10-114,
//            A/sourcecode/allaire_diffuse_colsweep.cpp:9-73
// with the ghost-cell fill that precedes each sweep
// (E/sourcecode/euler_ppsweep.cpp:7-118) synthesised while the tile is loaded,
// and, optionally, the CFL wave-speed reduction of the new state
// (E/sourcecode/euler_timestep.cpp:7-44, A/sourcecode/allaire_diffuse_timestep.cpp:8-48)
// fused into the store, finished by the last CTA, which also advances the
// device-resident time and picks the next dt.
//
// Layout in HBM: SoA, one plane per stored component, interior cells only,
// row-major with a padded pitch.
//
// Form: warp segments.  A warp holds 32 consecutive cells along the sweep in
// its lanes (28 outputs, two halo cells at each end) and takes them through
// the whole update in registers: conversion, limited slope, the two evolved
// face states, HLLC at the low face, update, and the wave speeds of the new
// state where the launch reduces them.  Neighbour values come by shuffles, so
// the update needs no barrier and no shared memory; the arithmetic is that of
// cfd_exact.cuh, with the plain functions for a segment any lane of which
// they do not serve.
//
// What bounds it: FP64 work.  At 2048^2 Euler the x sweep runs 858 thread
// instructions per cell, 360 of them on the FP64 pipe (53 % busy, 64 % of the
// issue slots), against 1921 and 478 when every division was made on its own
// and the phases met in shared memory: x 314 -> 165 us, y 426 -> 194 us.
// 4096^2 Euler 2.79 -> 1.34 ms a step, Allaire 2048x1024 0.90 -> 0.36 ms (0.33 with
// its options at compile time), the 200x200 grid 22.0 -> 18.0 us a step, where
// a launch is one pass through the code.
#pragma once

#include "cfd_exact.cuh"

namespace cfd {

enum { DIR_X = 0, DIR_Y = 1 };
enum {
    CNT_UNPHYSICAL_INPUT = 0,  // stencil state failing the reference's assert
    CNT_SLOPE_ZEROED = 1,      // "Unphysical state created by slope extrapolation"
    CNT_FIRST_ORDER = 2,       // "Unphysical state created by time evolution"
    CNT_FIXUP = 3,             // Euler post-update density/energy restore
    CNT_UNPHYSICAL_OUTPUT = 4, // Allaire assert after the z update
    CNT_N = 8
};

// Device-resident time-loop state (headers/simulation.hpp:44-61).
struct DevState {
    double t;      // simulated time of the current state
    double dt;     // dt chosen for the next step from the current state
    double T;      // end time
    double cfl;
    double maxu, maxv;    // max(|u|+c), max(|v|+c) over the current state
    double mass1, mass2;  // sum of density (Allaire: partial densities)
    double dx, dy;
    int n;         // steps taken
    int done;      // t >= T: further steps are no-ops
    unsigned ticket;  // last-CTA-done counter of the reduction
    int cur;       // which of the two state buffers holds the current state
};

struct SweepArgs {
    double* bufs[2];  // the two state buffers; input = bufs[cur ^ in_sel]
    int in_sel;
    int flip_cur;     // the finishing CTA flips DevState::cur (Strang: odd sweep count)
    long long plane;  // elements between component planes
    int pitch;        // elements between rows
    int nx, ny;
    Eos eos;
    int bc_lo, bc_hi;  // reflective walls at the low/high end along the sweep
    int limiter, wavespeed, godunov;
    double z_min;
    double h_flux;    // spacing handed to the flux solver (dx; dx or dy in y)
    double h_upd;     // spacing of the conservative update
    double dt_host;   // dt when use_host_dt
    double dt_scale;  // 1 or 0.5 (Strang half steps)
    int use_host_dt;
    int reduce;       // fuse the wave-speed reduction and the time advance
    int advance_time; // the reduction closes a step: t += dt, n++
    DevState* st;
    double* partials;  // 4 per CTA
    unsigned long long* counters;
};

__device__ __forceinline__ void block_count(unsigned long long* ctr, int idx, bool flag) {
    unsigned m = __ballot_sync(0xffffffffu, flag);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(ctr + idx, (unsigned long long)__popc(m));
}

// dt from the reduced wave speeds: E/sourcecode/euler_timestep.cpp:36-43.
__device__ __forceinline__ double choose_dt(const DevState& s, double maxu, double maxv) {
    double cfl = s.cfl;
    if (s.n < 5) cfl = smin(cfl, 0.2);
    double dt = __dmul_rn(cfl, smin(s.dx / maxu, s.dy / maxv));  // not contracted into the sum
    if (s.t + dt > s.T) dt = s.T - s.t;
    return dt;
}

// Last-CTA finish of the wave-speed reduction.  Partials are combined in CTA
// order, so the mass sums are reproducible run to run.
__device__ inline void finish_reduction(DevState* st, const double* partials, int nblocks,
                                 int advance_time, double dt_used, int flip_cur) {
    __shared__ double red[4][32];
    double mu = 0.0, mv = 0.0, m1 = 0.0, m2 = 0.0;
    // fixed assignment of partials to threads, then a fixed-order tree
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
        mu = smax(mu, partials[4 * b + 0]);
        mv = smax(mv, partials[4 * b + 1]);
        m1 += partials[4 * b + 2];
        m2 += partials[4 * b + 3];
    }
    for (int o = 16; o > 0; o >>= 1) {
        mu = smax(mu, __shfl_down_sync(0xffffffffu, mu, o));
        mv = smax(mv, __shfl_down_sync(0xffffffffu, mv, o));
        m1 += __shfl_down_sync(0xffffffffu, m1, o);
        m2 += __shfl_down_sync(0xffffffffu, m2, o);
    }
    int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        red[0][w] = mu;
        red[1][w] = mv;
        red[2][w] = m1;
        red[3][w] = m2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        mu = red[0][0];
        mv = red[1][0];
        m1 = red[2][0];
        m2 = red[3][0];
        for (int i = 1; i < nw; ++i) {
            mu = smax(mu, red[0][i]);
            mv = smax(mv, red[1][i]);
            m1 += red[2][i];
            m2 += red[3][i];
        }
        DevState s = *st;
        if (advance_time) {
            s.t = s.t + dt_used;
            s.n = s.n + 1;
            if (fabs(s.t - s.T) < 1e-12) s.t = s.T;
        }
        s.maxu = mu;
        s.maxv = mv;
        s.mass1 = m1 * s.dx * s.dy;
        s.mass2 = m2 * s.dx * s.dy;
        s.dt = choose_dt(s, mu, mv);
        s.done = !(s.t < s.T);
        s.ticket = 0;
        if (flip_cur) s.cur ^= 1;
        *st = s;
        __threadfence();
    }
}

// Wave speeds of one stored (unrotated) state, exactly as compute_dt forms
// them.  Returns |u|+c, |v|+c and the mass contributions.
template <int MODEL>
__device__ __forceinline__ void wave_speeds(const Eos& q, const double* U, double& su, double& sv,
                                            double& m1, double& m2) {
    Prim<MODEL> P;
    cons_to_prim<MODEL>(q, U, P);
    double c;
    if constexpr (MODEL == MODEL_EULER) {
        c = sg_soundspeed(q, P.W[3], P.rho);
        m1 = P.rho;
        m2 = 0.0;
    } else {
        c = mix_soundspeed(P.mix, P.rho, P.W[4]);
        m1 = U[0];
        m2 = U[1];
    }
    su = fabs(P.W[ModelTraits<MODEL>::IM]) + c;
    sv = fabs(P.W[ModelTraits<MODEL>::IT]) + c;
}

// One line segment: the warp's 32 lanes hold 32 consecutive cells along the
// sweep (kSegOut outputs, two halo cells at each end), in the sweep frame.
constexpr int kSegOut = 28;

template <int N>
__device__ __forceinline__ void shfl_up_d(const double* x, double* y) {
#pragma unroll
    for (int k = 0; k < N; ++k) y[k] = __shfl_up_sync(0xffffffffu, x[k], 1);
}
template <int N>
__device__ __forceinline__ void shfl_down_d(const double* x, double* y) {
#pragma unroll
    for (int k = 0; k < N; ++k) y[k] = __shfl_down_sync(0xffffffffu, x[k], 1);
}

// Event bits of a lane (counted under CNT_*).
enum { EV_INPUT = 1, EV_ZEROED = 2, EV_FIRST = 4, EV_FIXUP = 8, EV_OUTPUT = 16 };

// What a segment's update needs besides the cells.
struct SegPar {
    Eos q;
    int limiter, wavespeed, godunov;
    double z_min;
};

// z at a face: the side u* selects (A/headers/flux_solver_godunov.hpp:33-34,
// A/headers/flux_solver_MUSCLhancock.hpp:375).
__device__ __forceinline__ double face_z(int godunov, double us, double zL, double zR) {
    const double cs = copysign(1.0, us);
    if (godunov) return (((1.0 + cs) / 2.0) * zL) + (((1.0 - cs) / 2.0) * zR);
    return ((0.5 * (1.0 + cs)) * zL) + ((0.5 * (1.0 - cs)) * zR);
}

// The conservative update from the fluxes at the lane's low face (F, with u*
// and z* behind the components) and, by shuffle, at its high face.
template <int MODEL>
__device__ __forceinline__ void segment_new_state(const SegPar& A, const double* U, const double* F,
                                                  double k_upd, double* N) {
    constexpr int NV = ModelTraits<MODEL>::NV;
    double FR[NV + 2];
    shfl_down_d<MODEL == MODEL_EULER ? NV : NV + 2>(F, FR);
#pragma unroll
    for (int k = 0; k < NV; ++k) N[k] = U[k] + (k_upd * (F[k] - FR[k]));
    if constexpr (MODEL == MODEL_ALLAIRE) {
        double zL = 0.0, zR = 0.0;
        if (A.godunov) {
            zL = __shfl_up_sync(0xffffffffu, U[5], 1);
            zR = __shfl_down_sync(0xffffffffu, U[5], 1);
        }
        N[5] = z_update(A.godunov, k_upd, zL, U[5], zR, F[NV], FR[NV], F[NV + 1], FR[NV + 1], A.z_min);
        bool changed;
        snap_allaire(N, changed);  // live assert(is_physical_state(...))
    }
}

// The update of one segment: U (this lane's conserved state) -> N.  All 32
// lanes take part; N is valid in lanes 2 .. 2 + kSegOut - 1 when every lane
// returns true; `cell` marks the lanes whose N is stored.
template <int MODEL>
__device__ __forceinline__ bool segment_update(const SegPar& A, const double* U, double s_half,
                                               double k_upd, bool cell, double* N) {
    constexpr int NV = ModelTraits<MODEL>::NV;
    const Eos& q = A.q;
    const int lane = threadIdx.x & 31;
    Side<MODEL> L, R;
    bool ok;
    {
        Side<MODEL> S;  // the high face's
        if (!A.godunov) {
            PrimR<MODEL> P;
            ok = c2p_rn<MODEL>(q, U, P);
            double a[NV], b[NV], h[NV], X[NV], Wt[NV];
            shfl_up_d<NV>(P.W, a);
#pragma unroll
            for (int k = 0; k < NV; ++k) a[k] = P.W[k] - a[k];
            shfl_down_d<NV>(a, b);
            limit_diffs<NV>(A.limiter, a, b, h);
            bool in = jacobian_rn<MODEL>(q, P, h, s_half, X);
#pragma unroll
            for (int k = 0; k < NV; ++k) h[k] = 0.5 * h[k];
            in &= slopes_physical<MODEL>(q, P.W, h);
#pragma unroll
            for (int k = 0; k < NV; ++k) Wt[k] = (P.W[k] + h[k]) - X[k];
            in &= side_from_prim<MODEL>(q, Wt, S);
#pragma unroll
            for (int k = 0; k < NV; ++k) Wt[k] = (P.W[k] - h[k]) - X[k];
            in &= side_from_prim<MODEL>(q, Wt, R);
            ok &= in | (lane < 1) | (lane > 2 + kSegOut);
        } else {
#pragma unroll
            for (int k = 0; k < NV; ++k) S.U[k] = U[k];
            ok = side_from_cons<MODEL>(q, S);
            // the reference's test of the stencil states
            const double rho = S.rho;
            if constexpr (MODEL == MODEL_ALLAIRE)
                ok &= (U[0] >= 0.0) & (U[1] >= 0.0) & (U[5] >= 0.0) & (U[5] <= 1.0) &
                      surely_energy(rho, U[2], U[3], U[4]);
            else
                ok &= surely_energy(rho, U[1], U[2], U[3]);
            R = S;
        }
        // the lane below's high-face state is this lane's left state
        shfl_up_d<NV>(S.U, L.U);
        L.rho = L.U[0];
        if constexpr (MODEL == MODEL_ALLAIRE) L.rho = L.U[0] + L.U[1];
        L.u = __shfl_up_sync(0xffffffffu, S.u, 1);
        L.p = __shfl_up_sync(0xffffffffu, S.p, 1);
        L.c = __shfl_up_sync(0xffffffffu, S.c, 1);
        if (MODEL == MODEL_ALLAIRE && A.wavespeed == WS_PVRS) {  // its speeds use the mixture
            L.mix.eps = __shfl_up_sync(0xffffffffu, S.mix.eps, 1);
            L.mix.k = __shfl_up_sync(0xffffffffu, S.mix.k, 1);
            L.mix.ie = __shfl_up_sync(0xffffffffu, S.mix.ie, 1);
        }
    }
    double F[NV + 2];
    const bool fo = hllc_rn<MODEL>(q, A.wavespeed, L, R, F, F[NV]);
    ok &= fo | (lane < 2) | (lane > 2 + kSegOut);
    if constexpr (MODEL == MODEL_ALLAIRE) F[NV + 1] = face_z(A.godunov, F[NV], L.U[5], R.U[5]);
    segment_new_state<MODEL>(A, U, F, k_upd, N);
    bool fine;  // the new state surely passes the reference's test
    if constexpr (MODEL == MODEL_ALLAIRE) {
        const double rho = N[0] + N[1];
        fine = (N[0] >= 0.0) & (N[1] >= 0.0) & (N[5] >= 0.0) & (N[5] <= 1.0) & (rho > 0.0) &
               surely_energy(rho, N[2], N[3], N[4]);
    } else {
        fine = (N[0] > 0.0) & (N[3] > 0.0) & surely_energy(N[0], N[1], N[2], N[3]);
    }
    return ok & (fine | !cell);
}

// The same by the functions of cfd_physics.cuh, with the reference's
// fallbacks and events: `face` marks lanes whose low face belongs to this
// segment, `cell` those whose cell does.  In the y sweep the segment is the
// rotated one; u and v enter the post-update restore symmetrically.
template <int MODEL>
__device__ __noinline__ void segment_update_plain(const SegPar& A, const double* Uin, double s_half,
                                                  double k_upd, bool cell, bool face, double* N,
                                                  unsigned& ev) {
    using MT = ModelTraits<MODEL>;
    constexpr int NV = MT::NV;
    const Eos& q = A.q;
    double U[NV], UL[NV], EL[NV], ER[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) U[k] = Uin[k];
    shfl_up_d<NV>(U, UL);
    Prim<MODEL> P;
    cons_to_prim<MODEL>(q, U, P);
    // the reference's assert on the stencil states
    bool phys;
    if constexpr (MODEL == MODEL_EULER) phys = P.rho >= 0.0 && P.e >= 0.0;
    else phys = is_physical_exact<MODEL>(U);
    if (cell && !phys) ev |= EV_INPUT;
    if (!A.godunov) {
        double a[NV], b[NV], d[NV], X[NV], Wt[NV], Ut[NV], Ep[NV], e;
        shfl_up_d<NV>(P.W, a);
#pragma unroll
        for (int k = 0; k < NV; ++k) a[k] = P.W[k] - a[k];
        shfl_down_d<NV>(a, b);
        limit_diffs<NV>(A.limiter, a, b, d);
        // slope-extrapolated states (check only)
        unsigned fl = 0;
#pragma unroll
        for (int k = 0; k < NV; ++k) Wt[k] = P.W[k] + 0.5 * d[k];
        prim_to_cons<MODEL>(q, Wt, Ut, e);
        if (muscl_check<MODEL>(Ut, Wt, e)) fl |= 1u;  // high face ok
#pragma unroll
        for (int k = 0; k < NV; ++k) Wt[k] = P.W[k] - 0.5 * d[k];
        prim_to_cons<MODEL>(q, Wt, Ut, e);
        if (muscl_check<MODEL>(Ut, Wt, e)) fl |= 2u;  // low face ok
        // half-step evolved states
        jacobian_times<MODEL>(q, P, d, s_half, X);
#pragma unroll
        for (int k = 0; k < NV; ++k) Wt[k] = (P.W[k] + 0.5 * d[k]) - X[k];
        prim_to_cons<MODEL>(q, Wt, Ep, e);
        if (muscl_check<MODEL>(Ep, Wt, e)) fl |= 4u;
#pragma unroll
        for (int k = 0; k < NV; ++k) Wt[k] = (P.W[k] - 0.5 * d[k]) - X[k];
        prim_to_cons<MODEL>(q, Wt, ER, e);
        if (muscl_check<MODEL>(ER, Wt, e)) fl |= 8u;
        shfl_up_d<NV>(Ep, EL);
        const unsigned flL = __shfl_up_sync(0xffffffffu, fl, 1);
        bool ok2 = (flL & 4u) && (fl & 8u);
        if (!((flL & 1u) && (fl & 2u))) {  // zero slopes for this face
            if (face) ev |= EV_ZEROED;
            Prim<MODEL> PL;
            cons_to_prim<MODEL>(q, UL, PL);
            zero_slope_state<MODEL>(q, PL, s_half, true, Wt);
            prim_to_cons<MODEL>(q, Wt, EL, e);
            const bool okL = muscl_check<MODEL>(EL, Wt, e);
            zero_slope_state<MODEL>(q, P, s_half, false, Wt);
            prim_to_cons<MODEL>(q, Wt, ER, e);
            const bool okR = muscl_check<MODEL>(ER, Wt, e);
            ok2 = okL && okR;
        }
        if (!ok2) {
            if (face) ev |= EV_FIRST;
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                EL[k] = UL[k];
                ER[k] = U[k];
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            EL[k] = UL[k];
            ER[k] = U[k];
        }
    }
    double F[NV + 2];
    hllc_flux<MODEL>(q, A.wavespeed, EL, ER, F, F[NV]);
    if constexpr (MODEL == MODEL_ALLAIRE) F[NV + 1] = face_z(A.godunov, F[NV], EL[5], ER[5]);
    double Nn[NV];
    segment_new_state<MODEL>(A, U, F, k_upd, Nn);
    if (cell && !is_physical_exact<MODEL>(Nn)) {
        if constexpr (MODEL == MODEL_ALLAIRE) {
            ev |= EV_OUTPUT;
        } else {
            // E/sourcecode/euler_rowsweep.cpp:47-82: restore rho or e from the
            // old state when the update produced rho or e <= 0
            ev |= EV_FIXUP;
            double rho = Nn[0];
            double u = Nn[1] / rho;
            double v = Nn[2] / rho;
            double e = (Nn[3] / rho) - (0.5 * ((u * u) + (v * v)));
            double rho_old = U[0];
            double u_old = U[1] / rho_old;
            double v_old = U[2] / rho_old;
            double e_old = (U[3] / rho_old) - (0.5 * ((u_old * u_old) + (v_old * v_old)));
            if (rho <= 1e-12) rho = rho_old;
            if (e <= 1e-12) e = e_old;
            double W[4] = {rho, u, v, sg_pressure(q, e, rho)};
            double ee;
            prim_to_cons<MODEL>(q, W, Nn, ee);
        }
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) N[k] = Nn[k];
}

template <int MODEL>
__device__ __noinline__ void plain_speeds(const Eos& q, const double* U, double& su, double& sv) {
    double m1, m2;
    wave_speeds<MODEL>(q, U, su, sv, m1, m2);
}

__device__ __forceinline__ void count_events(unsigned long long* ctr, unsigned ev) {
    if (!__any_sync(0xffffffffu, ev != 0u)) return;
    block_count(ctr, CNT_UNPHYSICAL_INPUT, ev & EV_INPUT);
    block_count(ctr, CNT_SLOPE_ZEROED, ev & EV_ZEROED);
    block_count(ctr, CNT_FIRST_ORDER, ev & EV_FIRST);
    block_count(ctr, CNT_FIXUP, ev & EV_FIXUP);
    block_count(ctr, CNT_UNPHYSICAL_OUTPUT, ev & EV_OUTPUT);
}

// Tiles: x, kSegOut columns by kXRows rows, a row per warp; y, kSegOut rows
// by kYCols columns, a column per warp, staged through shared memory so that
// global accesses are rows of kYCols cells (64 bytes per component).  CTA c of
// G walks the tiles c, c + G, ...; the next tile's cells are copied global ->
// shared with cp.async while the current one is computed.
constexpr int kXRows = 4, kYCols = 8;
constexpr int kYStride = 34;  // doubles per staged column: conflict-free both ways

template <int DIR>
__host__ __device__ constexpr int sweep_threads() {
    return DIR == DIR_X ? 32 * kXRows : 32 * kYCols;
}
template <int MODEL, int DIR>
__host__ __device__ constexpr int sweep_min_ctas() {
    return MODEL == MODEL_EULER ? (DIR == DIR_X ? 4 : 2) : (DIR == DIR_X ? 3 : 1);
}
template <int MODEL, int DIR>
__host__ __device__ constexpr int sweep_smem_bytes() {
    constexpr int NV = ModelTraits<MODEL>::NV;
    return DIR == DIR_X ? 2 * NV * 32 * kXRows * 8 : 2 * NV * kYCols * kYStride * 8;
}
template <int DIR>
__host__ __device__ inline long long sweep_tiles(int nx, int ny) {
    const int len = DIR == DIR_X ? nx : ny, wid = DIR == DIR_X ? ny : nx;
    const int na = DIR == DIR_X ? kXRows : kYCols;
    return (long long)((len + kSegOut - 1) / kSegOut) * ((wid + na - 1) / na);
}

__device__ __forceinline__ void copy8_async(double* dst, const double* src) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(src) : "memory");
}

// A sweep kernel's options: those of its arguments, or MUSCL with one limiter
// and one wave-speed estimate at compile time (the same operations: the bits
// do not depend on it).
constexpr int kAnyOption = -1;
constexpr int sweep_option(int limiter, int wavespeed) { return 2 * limiter + wavespeed; }

template <int MODEL, int DIR, int OPT>
__global__ void __launch_bounds__(sweep_threads<DIR>(), sweep_min_ctas<MODEL, DIR>())
    sweep_kernel(SweepArgs A) {
    using MT = ModelTraits<MODEL>;
    constexpr int NV = MT::NV;
    constexpr int NA = DIR == DIR_X ? kXRows : kYCols;
    constexpr int BUF = DIR == DIR_X ? NV * 32 * kXRows : NV * kYCols * kYStride;
    extern __shared__ __align__(16) double smem[];

    const DevState* st = A.st;
    if (!A.use_host_dt && st->done) return;
    const int cur = st->cur;
    const double* __restrict__ gin = A.bufs[cur ^ A.in_sel];
    double* __restrict__ gout = A.bufs[cur ^ A.in_sel ^ 1];
    const double dt_step = A.use_host_dt ? A.dt_host : st->dt;  // dt of the whole step
    const double dt = A.dt_scale * dt_step;                        // this sweep's dt
    const double s_half = 0.5 * (dt / A.h_flux);
    const double k_upd = dt / A.h_upd;
    const int len = (DIR == DIR_X) ? A.nx : A.ny;  // cells along the sweep
    const int wid = (DIR == DIR_X) ? A.ny : A.nx;  // lines
    // tiles in memory order: x fastest
    const int tiles_x = (A.nx + (DIR == DIR_X ? kSegOut : NA) - 1) / (DIR == DIR_X ? kSegOut : NA);
    const int tiles_y = (A.ny + (DIR == DIR_X ? NA : kSegOut) - 1) / (DIR == DIR_X ? NA : kSegOut);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    // Ghost cell g (g = -1, -2 or len, len+1) mirrors interior cell -g-1 or
    // 2*len-1-g; a reflective wall negates the normal momentum
    // (E/sourcecode/euler_ppsweep.cpp:16,27).  Staged cells beyond the last
    // ghost (partial tiles) are clamped into range.
    auto source = [&](int ga) {
        const int r = ga < 0 ? -ga - 1 : ga >= len ? 2 * len - 1 - ga : ga;
        return min(max(r, 0), len - 1);
    };
    // the thread's cell of a tile: in x its own lane's, in y one of the eight
    // cells of a staged row
    auto issue = [&](int tx, int ty, double* buf) {
        if (ty < tiles_y) {
            const int a0 = (DIR == DIR_X ? tx : ty) * kSegOut - 2, b0 = (DIR == DIR_X ? ty : tx) * NA;
            if constexpr (DIR == DIR_X) {
                const long long off = (long long)min(b0 + warp, wid - 1) * A.pitch + source(a0 + lane);
#pragma unroll
                for (int k = 0; k < NV; ++k)
                    copy8_async(buf + k * 32 * kXRows + threadIdx.x, gin + k * A.plane + off);
            } else {
                const int r = threadIdx.x / kYCols, c = threadIdx.x % kYCols;
                const long long off = (long long)source(a0 + r) * A.pitch + min(b0 + c, wid - 1);
#pragma unroll
                for (int k = 0; k < NV; ++k)
                    copy8_async(buf + (k * kYCols + c) * kYStride + r, gin + k * A.plane + off);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    const SegPar par{A.eos, OPT == kAnyOption ? A.limiter : OPT / 2,
                     OPT == kAnyOption ? A.wavespeed : OPT % 2, OPT == kAnyOption ? A.godunov : 0,
                     A.z_min};

    double r_mu = 0.0, r_mv = 0.0, r_m1 = 0.0, r_m2 = 0.0;
    // this tile and the next (tx across the grid, ty up), stepped by the grid
    const int step_x = (int)gridDim.x % tiles_x, step_y = (int)gridDim.x / tiles_x;
    int tx = (int)blockIdx.x % tiles_x, ty = (int)blockIdx.x / tiles_x;
    issue(tx, ty, smem);
    int which = 0;
    while (ty < tiles_y) {
        int nx_ = tx + step_x, ny_ = ty + step_y;
        if (nx_ >= tiles_x) {
            nx_ -= tiles_x;
            ++ny_;
        }
        double* buf = smem + which * BUF;
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        if (DIR == DIR_Y) __syncthreads();
        issue(nx_, ny_, smem + (which ^ 1) * BUF);
        const int a0 = (DIR == DIR_X ? tx : ty) * kSegOut - 2, b0 = (DIR == DIR_X ? ty : tx) * NA;
        const int ga = a0 + lane, gb = b0 + warp;
        const bool line = gb < wid;  // the same for the whole warp
        const bool cell = lane >= 2 && lane < 2 + kSegOut && ga < len;
        if (line) {
            const bool neg = (ga < 0 && A.bc_lo) || (ga >= len && A.bc_hi);
            double U[NV], N[NV];
            if constexpr (DIR == DIR_X) {
#pragma unroll
                for (int k = 0; k < NV; ++k) U[k] = buf[k * 32 * kXRows + threadIdx.x];
                if (neg) U[MT::IM] = -U[MT::IM];
            } else {
                // the rotated state (u,v) -> (v,-u) (E/sourcecode/euler_colsweep.cpp:22-29)
#pragma unroll
                for (int k = 0; k < NV; ++k) U[k] = buf[(k * kYCols + warp) * kYStride + lane];
                if (neg) U[MT::IT] = -U[MT::IT];
                const double t = U[MT::IM];
                U[MT::IM] = U[MT::IT];
                U[MT::IT] = -t;
            }
            bool ok = segment_update<MODEL>(par, U, s_half, k_upd, cell, N);
            double su = 0.0, sv = 0.0;  // symmetric in the rotation up to the order of the two
            if (A.reduce) ok &= wave_speeds_rn<MODEL>(par.q, N, su, sv) | !cell;
            if (!__all_sync(0xffffffffu, ok)) {  // rare
                const bool face = (lane >= 2 && lane < 2 + kSegOut && ga <= len) ||
                                  (lane == 2 + kSegOut && ga == len);
                const SegPar pc = par;
                double Uc[NV], Nc[NV];
                unsigned ec = 0;
#pragma unroll
                for (int k = 0; k < NV; ++k) Uc[k] = U[k];
                segment_update_plain<MODEL>(pc, Uc, s_half, k_upd, cell, face, Nc, ec);
#pragma unroll
                for (int k = 0; k < NV; ++k) N[k] = Nc[k];
                if (A.reduce && cell) plain_speeds<MODEL>(pc.q, Nc, su, sv);
                count_events(A.counters, ec);
            }
            if (A.reduce && cell) {
                r_mu = smax(r_mu, DIR == DIR_X ? su : sv);
                r_mv = smax(r_mv, DIR == DIR_X ? sv : su);
                r_m1 += N[0];
                if (MODEL == MODEL_ALLAIRE) r_m2 += N[1];
            }
            if (DIR == DIR_Y) {  // rotate back (E/sourcecode/euler_colsweep.cpp:66-73)
                const double t = N[MT::IM];
                N[MT::IM] = -N[MT::IT];
                N[MT::IT] = t;
            }
            if constexpr (DIR == DIR_X) {
                if (cell) {
                    const long long off = (long long)gb * A.pitch + ga;
#pragma unroll
                    for (int k = 0; k < NV; ++k) gout[k * A.plane + off] = N[k];
                }
            } else {
                // back through the staged column (read by this warp only)
#pragma unroll
                for (int k = 0; k < NV; ++k) buf[(k * kYCols + warp) * kYStride + lane] = N[k];
            }
        }
        if constexpr (DIR == DIR_Y) {
            __syncthreads();
            const int r = threadIdx.x / kYCols, c = threadIdx.x % kYCols;
            if (r >= 2 && r < 2 + kSegOut && a0 + r < len && b0 + c < wid) {
                const long long off = (long long)(a0 + r) * A.pitch + b0 + c;
#pragma unroll
                for (int k = 0; k < NV; ++k)
                    gout[k * A.plane + off] = buf[(k * kYCols + c) * kYStride + r];
            }
        }
        tx = nx_;
        ty = ny_;
        which ^= 1;
    }
    if (!A.reduce) return;

    // ---- block reduction, last-CTA finish ---------------------------------
    constexpr int NW = NA;
    __shared__ double red[4][NW];
    __shared__ bool is_last;
    for (int o = 16; o > 0; o >>= 1) {
        r_mu = smax(r_mu, __shfl_down_sync(0xffffffffu, r_mu, o));
        r_mv = smax(r_mv, __shfl_down_sync(0xffffffffu, r_mv, o));
        r_m1 += __shfl_down_sync(0xffffffffu, r_m1, o);
        r_m2 += __shfl_down_sync(0xffffffffu, r_m2, o);
    }
    if (lane == 0) {
        red[0][warp] = r_mu;
        red[1][warp] = r_mv;
        red[2][warp] = r_m1;
        red[3][warp] = r_m2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double mu = red[0][0], mv = red[1][0], m1 = red[2][0], m2 = red[3][0];
        for (int w = 1; w < NW; ++w) {
            mu = smax(mu, red[0][w]);
            mv = smax(mv, red[1][w]);
            m1 += red[2][w];
            m2 += red[3][w];
        }
        double* p = A.partials + 4 * blockIdx.x;
        p[0] = mu;
        p[1] = mv;
        p[2] = m1;
        p[3] = m2;
        __threadfence();
        unsigned t = atomicAdd(&A.st->ticket, 1u);
        is_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (is_last) {
        __threadfence();
        finish_reduction(A.st, A.partials, gridDim.x, A.advance_time, dt_step, A.flip_cur);
    }
}

}  // namespace cfd
