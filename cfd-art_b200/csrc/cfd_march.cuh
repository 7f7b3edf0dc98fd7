// Barrier-free warp forms of the mixed-precision sweeps.
//
// Marching strips (the y sweep): a warp owns a strip of 32 lines x A.rows
// cells along the sweep of one instance: lane = line, and every lane walks
// along its line one cell at a time, carrying the window the stencil needs
// from one row to the next in registers (primitive states, the face state,
// the flux).  The rows ahead of the one being computed are copied global ->
// shared with cp.async, three rows in flight, so no registers are held by
// the loads, and each row stays in shared memory until the update that
// starts from it.  The strip length is chosen per launch on the
// host (kMarchMinRows..kMarchMaxRows) so that the strips fill the resident
// warps.  No barrier is needed, and only the two halo cells at each end of
// a strip are re-read.  The lanes are 32 consecutive columns, so every step
// reads 32 consecutive cells (coalesced).  (Marching along x, with the lanes
// on 32 rows, measured 1.9x slower than the tiled x sweep.)  The arithmetic of every
// cell, face and update is the one of the tiled sweep (cfd_mixed.cuh): the
// same functions in the same order, so the two give the same results bit for
// bit and the autotuner may pick either.
//
// Both sweeps are compiled for the common options (limiter, PVRS speeds,
// stiffened gas) as well: a member's options come from memory, so the compiler
// cannot see that a branch on them is uniform and pays for reconvergence at
// every one.  A launch all of whose members have one such set of options runs
// its instantiation, any other the general one.
//
// Reduction: march_reduce, close_steps.
//
// Where a launch's tiles leave most warps idle (small grids, where the time of
// a sweep is that of one warp walking one tile), each tile is divided among
// several warps: A.split.
//
// Warp segments (the x sweep, further down): the lanes hold 32 consecutive
// cells of a row and exchange neighbour values by shuffles.
#pragma once

#include "cfd_mixed.cuh"

namespace cfd {
namespace mixed {

constexpr int kMarchMaxRows = 64, kMarchMinRows = 16;  // rows of a strip (its width is one warp)

template <bool B> struct Bool {
    static constexpr bool value = B;
};

// y-sweep frame: the boundary sign of a mirrored row, then (u, v) -> (v, -u).
template <int MODEL>
__device__ __forceinline__ void march_rotate_in(float* h, float* l, bool neg) {
    using MT = ModelTraits<MODEL>;
    if (neg) {
        h[MT::IT] = -h[MT::IT];
        l[MT::IT] = -l[MT::IT];
    }
    float t = h[MT::IM], tl = l[MT::IM];
    h[MT::IM] = h[MT::IT];
    l[MT::IM] = l[MT::IT];
    h[MT::IT] = -t;
    l[MT::IT] = -tl;
}

// The warp's four sums of a slot's lanes (speeds by maximum), fixed shuffle
// tree: reproducible sums, in lane 0.
__device__ __forceinline__ void warp_sums(double& mu, double& mv, double& m1, double& m2) {
    for (int o = 16; o > 0; o >>= 1) {
        mu = smax(mu, __shfl_down_sync(0xffffffffu, mu, o));
        mv = smax(mv, __shfl_down_sync(0xffffffffu, mv, o));
        m1 += __shfl_down_sync(0xffffffffu, m1, o);
        m2 += __shfl_down_sync(0xffffffffu, m2, o);
    }
}
__device__ __forceinline__ void put_slot(double* p, double mu, double mv, double m1, double m2) {
    reinterpret_cast<double2*>(p)[0] = make_double2(mu, mv);
    reinterpret_cast<double2*>(p)[1] = make_double2(m1, m2);
}
__device__ __forceinline__ void add_slot(const double* p, double& mu, double& mv, double& m1, double& m2) {
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
    const double2 b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
    mu = smax(mu, a.x);
    mv = smax(mv, a.y);
    m1 += b.x;
    m2 += b.y;
}

// Closes a member's step with the reduced wave speeds and masses of its new
// state: time, step count, dt of the next step.
__device__ __forceinline__ void close_step(DevState* st, double mu, double mv, double m1, double m2) {
    DevState s = *st;
    s.t = s.t + s.dt;
    s.n = s.n + 1;
    if (fabs(s.t - s.T) < 1e-12) s.t = s.T;
    s.maxu = mu;
    s.maxv = mv;
    s.mass1 = m1 * s.dx * s.dy;
    s.mass2 = m2 * s.dx * s.dy;
    s.dt = choose_dt(s, mu, mv);
    s.done = !(s.t < s.T);
    s.ticket = 0;
    *st = s;
    __threadfence();
}

// A part's wave speeds and masses (per lane) into its slot, by its warp.  The
// warp that completes the member's slots combines them in slot order
// (reproducible sums) and closes the step; a member of many slots is closed by
// close_steps instead, launched behind the y sweeps: the fence and the ticket
// of every part and one warp's walk over the slots took 10.5 us of the 63 us
// sweep of a 2048^2 Euler member (2,368 slots); sweep and close together take
// 57.6.  At 256^2 (1,024 slots) a step takes 14.1 us with the close and 16.2
// with the ticket; up to kTicketSlots, one per lane, the ticket is as fast
// (64^2: 10.3 and 10.4).  Batches of many uneven members that fit one round of
// the resident warps hide the ticket (24 members 69.9 us, 71.3 with the close),
// those of several rounds do not (100 members 363, 336).
__device__ __forceinline__ void march_reduce(const Inst& I, int slot, double mu, double mv, double m1,
                                             double m2) {
    const int lane = threadIdx.x & 31;
    DevState* st = I.st;
    warp_sums(mu, mv, m1, m2);
    if (lane == 0) put_slot(I.partials + 4 * slot, mu, mv, m1, m2);
    if (I.closed) return;
    unsigned t = 0;
    if (lane == 0) {
        __threadfence();
        t = atomicAdd(&st->ticket, 1u);
    }
    if (__shfl_sync(0xffffffffu, t, 0) + 1u != (unsigned)I.slots) return;
    __threadfence();
    mu = mv = m1 = m2 = 0.0;
    if (lane < I.slots) add_slot(I.partials + 4 * lane, mu, mv, m1, m2);
    warp_sums(mu, mv, m1, m2);
    if (lane == 0) close_step(st, mu, mv, m1, m2);
}

// Closes the steps of the members marked so, a CTA each, from the slots their
// y sweep has filled; members that sweep skipped are skipped.
constexpr int kCloseThreads = 256;
constexpr int kTicketSlots = 32;  // most slots of a member closed by its last warp, one per lane
__global__ void __launch_bounds__(kCloseThreads) close_steps(const Inst* insts, int which) {
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the last y sweep's completion
    const Inst& I = insts[blockIdx.x];
    DevState* st = I.st;
    if (I.closed != which || !I.active || st->done || st->n >= I.max_steps) return;
    double mu = 0.0, mv = 0.0, m1 = 0.0, m2 = 0.0;
    const int n = I.slots;
    const double* p = I.partials;
#pragma unroll 4
    for (int b = threadIdx.x; b < n; b += kCloseThreads) add_slot(p + 4 * b, mu, mv, m1, m2);
    warp_sums(mu, mv, m1, m2);
    __shared__ __align__(16) double red[4 * (kCloseThreads / 32)];
    if ((threadIdx.x & 31) == 0) put_slot(red + 4 * (threadIdx.x >> 5), mu, mv, m1, m2);
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < kCloseThreads / 32; ++w) {
        const double* q = red + 4 * w;
        mu = smax(mu, q[0]);
        mv = smax(mv, q[1]);
        m1 += q[2];
        m2 += q[3];
    }
    close_step(st, mu, mv, m1, m2);
}

// Parts of a tile: `rows` rows divided into A.split, a warp each.  Undivided,
// a 64^2 grid is 18 tiles of 12 rows in x and 8 strips of 16 (20 with the halo)
// in y, one warp walking each: 17.4 us a step of Euler, 10.2 divided; 256^2
// 19.9 -> 14.0 us (fast FP64 25.9 -> 16.9).
__device__ __forceinline__ int part_rows(const MixedArgs& A) { return (A.rows + A.split - 1) / A.split; }

// Rows staged through shared memory with cp.async (no registers held by the
// loads in flight): a ring of kMSlots slots per lane holding at least rows
// k-2 .. k+3 while row k is computed; kMAhead rows in flight; per slot MU
// 16-byte units per lane (value and compensation words of components 0-3; for
// Allaire E and z with their compensation words).  The raw cells of row
// k-2, which its update starts from, are therefore read again from the
// ring rather than carried in registers for two rows.  Six slots would do; with
// eight a slot's offset is a mask (4 instructions a row fewer).
//
// Element offsets within a plane are 32-bit: a plane has at most 2^31 cells
// and its row padding, and an address is then one multiply-add.
constexpr int kMAhead = 3, kMSlots = 8;
template <int MODEL>
__host__ __device__ constexpr int march_units() {
    return MODEL == MODEL_ALLAIRE ? 3 : 2;
}

// Dynamic shared memory of a 4-warp marching CTA: the staging rings.
template <int MODEL>
__host__ __device__ constexpr int march_smem_bytes() {
    return 4 * kMSlots * march_units<MODEL>() * 32 * 16;
}

// Starts copying the cell at element offset `off` of the planes `Q` (value
// and compensation words) into a slot of this lane's staging ring.
template <int MODEL>
__device__ __forceinline__ void mstage_issue(char* slot, const MPlanes& Q, unsigned off) {
    cp_async16(slot, Q.v4 + off);
    cp_async16(slot + 512, Q.c4 + off);
    if constexpr (MODEL == MODEL_ALLAIRE) {
        cp_async8(slot + 1024, Q.v2 + off);
        cp_async8(slot + 1024 + 8, Q.c2 + off);
    }
}

// The cell staged in a slot (as stored: no mirror, no rotation).
template <int MODEL>
__device__ __forceinline__ void mstage_read(const char* slot, float* h, float* l) {
    const float4 a = *reinterpret_cast<const float4*>(slot);
    const float4 b = *reinterpret_cast<const float4*>(slot + 512);
    h[0] = a.x; h[1] = a.y; h[2] = a.z; h[3] = a.w;
    l[0] = b.x; l[1] = b.y; l[2] = b.z; l[3] = b.w;
    if constexpr (MODEL == MODEL_ALLAIRE) {
        const float4 e = *reinterpret_cast<const float4*>(slot + 1024);
        h[4] = e.x; h[5] = e.y;
        l[4] = e.z; l[5] = e.w;
    }
}

// The options of a member as the sweeps branch on them: Inst::flags without
// the walls, and without the limiter in first order.
constexpr int MF_OPTIONS = 31;
constexpr int kOptGeneral = -1;
__host__ __device__ constexpr int sweep_options(int flags) {
    return flags & MF_GODUNOV ? flags & MF_OPTIONS & ~3 : flags & MF_OPTIONS;
}

// One part of a strip: rows [r0, r1) of the columns [b_org, b_org + 32) of
// instance g.inst (none where the strip is shorter than its parts).
template <int MODEL, int OPT>
__device__ __forceinline__ void march_strip(const MixedArgs& A, const TileGeom& g, int part) {
    using MT = ModelTraits<MODEL>;
    constexpr int NV = MT::NV;
    const int lane = threadIdx.x & 31;
    const Inst& I = A.insts[g.inst];
    MPar P = load_par(I);
    const bool wall_lo = (P.flags >> 7) & 1, wall_hi = (P.flags >> 8) & 1;  // bottom, top
    if (OPT != kOptGeneral) P.flags = OPT;
    DevState* st = I.st;
    const double dt = st->dt;
    const float s_half = (float)(0.5 * (dt / (I.fix_dy ? I.dy : I.dx)));
    const float k_upd = (float)(dt / I.dy);
    const int ny = g.len, nx = g.wid;
    const int col = g.b_org + lane;
    const bool live = col < nx;
    const int c = min(col, nx - 1);
    const int r0 = min(g.a_org + 2 + part * part_rows(A), ny);
    const int r1 = min(min(r0 + part_rows(A), g.a_org + 2 + A.rows), ny);
    // the y sweep reads the x sweep's output.  Euler holds the planes in
    // registers (2 % faster); Allaire, at its 128-register limit, spilled that
    // way and measured 3 % slower, so it reads them from the member descriptor
    // where it uses them
    const int bin = g.cur ^ 1, bout = g.cur;
    const MPlanes qin_r = mplanes<MODEL>(I, bin), qout_r = mplanes<MODEL>(I, bout);
    auto qin = [&] {
        if constexpr (MODEL == MODEL_EULER) return qin_r;
        else return mplanes<MODEL>(I, bin);
    };
    auto qout = [&] {
        if constexpr (MODEL == MODEL_EULER) return qout_r;
        else return mplanes<MODEL>(I, bout);
    };
    const unsigned pitch = I.pitch;
    const bool god = P.godunov();
    const int lim = P.limiter();

    // the mirrored source row of input row k and its sign
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

    float W1[NV], W2[NV];       // W(k-1), W(k-2)
    bool okp = false;           // whether Pp may be used
    float Pp[NV], Fl[NV];       // state at the high face of row k-2, flux at its low face
    float us_low = 0.f, zs_low = 0.f;
    float z3 = 0.f;             // z of row k-3 (first-order z update)
    float rmu = 0.f, rmv = 0.f;
    double rm1 = 0.0, rm2 = 0.0;
#pragma unroll
    for (int q = 0; q < NV; ++q) W1[q] = W2[q] = Pp[q] = Fl[q] = 0.f;

    extern __shared__ __align__(16) char march_stage[];
    constexpr int MU = march_units<MODEL>();
    constexpr int SB = MU * 32 * 16, RB = kMSlots * SB;  // bytes of a slot, of the ring
    char* stg = march_stage + (threadIdx.x >> 5) * RB + 16 * lane;
    bool ng;
#pragma unroll
    for (int j = 0; j < kMAhead; ++j) {
        if (r0 < r1)  // a part without rows copies none: nothing below would wait for them
            mstage_issue<MODEL>(stg + j * SB, qin(), (unsigned)src_row(r0 - 2 + j, ng) * pitch + c);
        cp_async_commit();
    }
    // the ring's slots are numbered by row: row r0 - 2 + j is in slot j mod
    // kMSlots; `at` is row k's
    int at = 0;
    auto slot_of = [&](int rows) {  // of row k + rows
        static_assert((kMSlots & (kMSlots - 1)) == 0, "a power of two");
        return stg + (unsigned)((at + rows) & (kMSlots - 1)) * SB;
    };

    // Row k arrives.  `steady`: k - 2 >= r0 and k + kMAhead < r1, so every
    // part of the step applies and no row in it is mirrored.
    auto row_step = [&](int k, auto steady_t) {
        constexpr bool steady = decltype(steady_t)::value;
        float h[NV], l[NV];
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kMAhead - 1) : "memory");
        mstage_read<MODEL>(slot_of(0), h, l);
        bool neg = false;
        if (steady) {
            mstage_issue<MODEL>(slot_of(kMAhead), qin(), (unsigned)(k + kMAhead) * pitch + c);
        } else {
            if (k + kMAhead <= r1 + 1)
                mstage_issue<MODEL>(slot_of(kMAhead), qin(),
                                    (unsigned)src_row(k + kMAhead, neg) * pitch + c);
            src_row(k, neg);
        }
        cp_async_commit();
        march_rotate_in<MODEL>(h, l, neg);
        float W0[NV];
        c2p_mixed<MODEL>(I, P, h, l, W0);

        // slopes and evolved face states of row k-1
        float Pn[NV], Mn[NV];
        bool okn = false, okm = false;
        if ((steady || k >= r0) && !god) {
            float d[NV];
            limit_all<NV>(lim, W2, W1, W0, d);
            face_states<MODEL>(P, W1, d, s_half, Pn, Mn, okn, okm);
        }

        // HLLC at the face between rows k-2 and k-1
        float Fh[NV + 2];
        if (steady || k >= r0 + 1) {
            const bool first = god || !(okp && okm);
            if (god || __any_sync(0xffffffffu, first)) {  // rare in second order
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    Pp[q] = first ? W2[q] : Pp[q];
                    Mn[q] = first ? W1[q] : Mn[q];
                }
            }
            hllc_prim<MODEL>(P, Pp, Mn, Fh);
        }

        // compensated update of row k-2
        if (steady || k >= r0 + 2) {
            const unsigned off = (unsigned)(k - 2) * pitch + c;  // inside [r0, r1): no mirror
            float hh[NV], ll[NV];
            mstage_read<MODEL>(slot_of(-2), hh, ll);
            march_rotate_in<MODEL>(hh, ll, false);
            comp_update<NV>(hh, ll, k_upd, Fl, Fh);
            if constexpr (MODEL == MODEL_ALLAIRE) {
                const float usL = us_low, usR = Fh[NV], zsL = zs_low, zsR = Fh[NV + 1];
                const float z = hh[5];
                float dz;
                if (god)
                    dz = -k_upd * ((W1[5] - z) * fminf_s(0.0f, usR) + (z - z3) * fmaxf_s(0.0f, usL));
                else
                    dz = -k_upd * ((usR * zsR - usL * zsL) - z * (usR - usL));
                comp_add(hh[5], ll[5], dz);
                clip_z(I, hh[5], ll[5]);
                if (hh[0] < 0.0f) { hh[0] = 0.0f; ll[0] = 0.0f; }
                if (hh[1] < 0.0f) { hh[1] = 0.0f; ll[1] = 0.0f; }
            }
            {  // rotate back
                float t = hh[MT::IM], tl = ll[MT::IM];
                hh[MT::IM] = -hh[MT::IT];
                ll[MT::IM] = -ll[MT::IT];
                hh[MT::IT] = t;
                ll[MT::IT] = tl;
            }
            float Wn[NV];
            c2p_mixed<MODEL>(I, P, hh, ll, Wn);
            if constexpr (MODEL == MODEL_EULER) {
                // density / energy restore as in the plain form (rare)
                if (!(hh[0] > 1e-12f) || !(P.plus_gp1(Wn[3]) > 0.0f)) {
                    float oh[NV], ol[NV], Wo[NV];  // the cell before the update
                    load_cell<MODEL>(qin(), off, oh, ol);
                    c2p_mixed<MODEL>(I, P, oh, ol, Wo);  // stored (unrotated) frame
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
            if (live) {
                store_cell<MODEL>(qout(), off, hh, ll);
                float cs = sound_f<MODEL>(P, Wn);
                rmu = fmaxf_s(rmu, fabsf(Wn[MT::IM]) + cs);
                rmv = fmaxf_s(rmv, fabsf(Wn[MT::IT]) + cs);
                rm1 += (double)hh[0] + (double)ll[0];
                if constexpr (MODEL == MODEL_ALLAIRE) rm2 += (double)hh[1] + (double)ll[1];
            }
        }

        // shift the window
        if constexpr (MODEL == MODEL_ALLAIRE) z3 = W2[5];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            W2[q] = W1[q];
            W1[q] = W0[q];
            Pp[q] = Pn[q];
        }
        okp = okn;
        ++at;
        if (steady || k >= r0 + 1) {
#pragma unroll
            for (int q = 0; q < NV; ++q) Fl[q] = Fh[q];
            us_low = Fh[NV];
            zs_low = MODEL == MODEL_ALLAIRE ? Fh[NV + 1] : 0.f;
        }
    };
    int k = r0 < r1 ? r0 - 2 : r1 + 2;
    while (k <= r1 + 1) {
        row_step(k, Bool<false>{});
        ++k;
        // Euler: the rows away from the strip's ends run a copy of the step
        // without its tests, unrolled by two so that half the window changes
        // roles instead of being copied (6 % faster in all); Allaire spills
        // with the two copies (5 % slower)
        if (MODEL == MODEL_EULER && k == r0 + 2)
#pragma unroll 2
            for (; k + kMAhead < r1; ++k) row_step(k, Bool<true>{});
    }

    march_reduce(I, g.ltile * A.split + part, (double)rmu, (double)rmv, rm1, rm2);
}

// Persistent sweep: warp w of the W warps of the grid walks the strips w,
// w + W, w + 2W, ... of the launch's strip list, so the strips of members
// that have finished (skipped) are spread over all warps instead of idling
// some of them.
template <int MODEL, int OPT>
__global__ void __launch_bounds__(128, 4) mixed_march_kernel(MixedArgs A) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // close_steps may be scheduled
    const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int w = gw; w < A.ntiles * A.split; w += nw) {
        const TileGeom g = tile_geom<DIR_Y, kMarchMaxRows, 32>(A, w / A.split);
        if (!g.skip) march_strip<MODEL, OPT>(A, g, w % A.split);
    }
}

// ---- x sweep by warp segments ------------------------------------------------
// A warp owns a tile of kSegCells columns x A.rows rows and walks its rows:
// the 32 lanes hold 32 consecutive cells of a row (kSegCells outputs plus a
// 2-cell halo at each end), so every load and store is coalesced, and the
// neighbours each stencil step needs (primitive states, face states, fluxes)
// come from the adjacent lanes by warp shuffles: no barrier, and shared
// memory only for the rows staged ahead.  The arithmetic is the tiled
// sweep's, in the same order.
// The rows are staged like the marching strips' (kMAhead in flight), in
// a ring of kSSlots slots per lane: the slot refilled at row r is the one
// read at row r - 1.
constexpr int kSSlots = kMAhead + 1;
template <int MODEL>
__host__ __device__ constexpr int seg_smem_bytes() {
    return 4 * kSSlots * march_units<MODEL>() * 32 * 16;  // 4 warps per CTA
}
constexpr int kSegCells = 28;  // outputs per row segment
// rows of a tile: chosen per launch on the host (kSegMinRows..kSegRows) so
// that the tiles fill the resident warps
constexpr int kSegRows = 32, kSegMinRows = 12;

template <int N>
__device__ __forceinline__ void shfl_up_n(const float* x, float* y) {
#pragma unroll
    for (int q = 0; q < N; ++q) y[q] = __shfl_up_sync(0xffffffffu, x[q], 1);
}
template <int N>
__device__ __forceinline__ void shfl_down_n(const float* x, float* y) {
#pragma unroll
    for (int q = 0; q < N; ++q) y[q] = __shfl_down_sync(0xffffffffu, x[q], 1);
}

template <int MODEL, int OPT>
__device__ __forceinline__ void segment_tile(const MixedArgs& A, const TileGeom& g, int row_begin, int row_end) {
    using MT = ModelTraits<MODEL>;
    constexpr int NV = MT::NV;
    const int lane = threadIdx.x & 31;
    const Inst& I = A.insts[g.inst];
    MPar P = load_par(I);
    const bool wall_lo = (P.flags >> 5) & 1, wall_hi = (P.flags >> 6) & 1;  // left, right
    if (OPT != kOptGeneral) P.flags = OPT;
    const double dt = I.st->dt;
    const float s_half = (float)(0.5 * (dt / I.dx));
    const float k_upd = (float)(dt / I.dx);
    const int nx = g.len, ny = g.wid;
    const int bin = g.cur, bout = g.cur ^ 1;
    const MPlanes qin = mplanes<MODEL>(I, bin), qout = mplanes<MODEL>(I, bout);
    const unsigned pitch = I.pitch;
    const bool god = P.godunov();
    const int lim = P.limiter();
    // this lane's column and its mirrored source (pre_sweep's fill)
    const int ga = g.a_org + lane;
    int src = ga;
    bool neg = false;
    if (ga < 0) {
        src = -ga - 1;
        neg = wall_lo;
    } else if (ga >= nx) {
        src = 2 * nx - 1 - ga;
        neg = wall_hi;
    }
    src = min(max(src, 0), nx - 1);
    const bool writer = lane >= 2 && lane < 2 + kSegCells && ga < nx;
    row_end = min(row_end, ny);

    extern __shared__ __align__(16) char seg_stage[];
    constexpr int MU = march_units<MODEL>();
    constexpr int SB = MU * 32 * 16;
    static_assert((kSSlots & (kSSlots - 1)) == 0, "a power of two");
    char* stg = seg_stage + (threadIdx.x >> 5) * (kSSlots * SB) + 16 * lane;
    unsigned off_in = (unsigned)row_begin * pitch + src;           // the next row to load
    unsigned off_out = (unsigned)row_begin * pitch + (unsigned)ga;  // this row's cell
#pragma unroll
    for (int j = 0; j < kMAhead; ++j) {
        if (row_begin + j < row_end) mstage_issue<MODEL>(stg + j * SB, qin, off_in);
        off_in += pitch;
        cp_async_commit();
    }
    int at = 0;
    for (int row = row_begin; row < row_end; ++row, off_in += pitch, off_out += pitch, ++at) {
        float h[NV], l[NV];
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kMAhead - 1) : "memory");
        mstage_read<MODEL>(stg + (unsigned)(at & (kSSlots - 1)) * SB, h, l);
        if (row + kMAhead < row_end)
            mstage_issue<MODEL>(stg + (unsigned)((at + kMAhead) & (kSSlots - 1)) * SB, qin, off_in);
        cp_async_commit();
        if (neg) {
            h[MT::IM] = -h[MT::IM];
            l[MT::IM] = -l[MT::IM];
        }
        float W[NV], Wl[NV], Wr[NV];
        c2p_mixed<MODEL>(I, P, h, l, W);
        shfl_up_n<NV>(W, Wl);
        if (!god || MODEL == MODEL_ALLAIRE) shfl_down_n<NV>(W, Wr);  // first order: Allaire's z only

        // slopes and evolved face states of this cell (used by lanes 1..30)
        float Pf[NV], Mf[NV];
        bool okp = false, okm = false;
        if (!god) {
            float d[NV];
            limit_all<NV>(lim, Wl, W, Wr, d);
            face_states<MODEL>(P, W, d, s_half, Pf, Mf, okp, okm);
        }

        // HLLC at this cell's low face (between the lane below and this one)
        float PL[NV];
        unsigned okL = 0;  // bit l: lane l - 1's high-face state may be used
        if (!god) {
            shfl_up_n<NV>(Pf, PL);
            okL = __ballot_sync(0xffffffffu, okp) << 1;
        }
        float F[NV + 2];
        {
            const bool first = god || (!(((okL >> lane) & 1u) && okm) && lane >= 2);
            // rare in second order (the vote measured 2 % faster than
            // selecting for Allaire, 3 % slower for Euler)
            if (MODEL == MODEL_EULER || god || __any_sync(0xffffffffu, first)) {
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    PL[q] = first ? Wl[q] : PL[q];
                    Mf[q] = first ? W[q] : Mf[q];
                }
            }
            hllc_prim<MODEL>(P, PL, Mf, F);
        }
        float FR[NV + 2];  // Euler's update needs only the NV fluxes, not u*
        shfl_down_n<MODEL == MODEL_EULER ? NV : NV + 2>(F, FR);

        // compensated update (lanes 2 .. 2 + kSegCells - 1)
        comp_update<NV>(h, l, k_upd, F, FR);
        if constexpr (MODEL == MODEL_ALLAIRE) {
            const float usL = F[NV], usR = FR[NV], zsL = F[NV + 1], zsR = FR[NV + 1];
            const float z = h[5];
            float dz;
            if (god)
                dz = -k_upd * ((Wr[5] - z) * fminf_s(0.0f, usR) + (z - Wl[5]) * fmaxf_s(0.0f, usL));
            else
                dz = -k_upd * ((usR * zsR - usL * zsL) - z * (usR - usL));
            comp_add(h[5], l[5], dz);
            clip_z(I, h[5], l[5]);
            if (h[0] < 0.0f) { h[0] = 0.0f; l[0] = 0.0f; }
            if (h[1] < 0.0f) { h[1] = 0.0f; l[1] = 0.0f; }
        }
        if constexpr (MODEL == MODEL_EULER) {
            // density / energy restore as in the plain form (rare)
            float Wn[NV];
            bool restore = writer && !euler_sure(h);
            if (restore) {
                c2p_mixed<MODEL>(I, P, h, l, Wn);
                restore = !(h[0] > 1e-12f) || !(P.plus_gp1(Wn[3]) > 0.0f);
            }
            if (restore) {
                float oh[NV], ol[NV], Wo[NV];  // the cell before the update
                load_cell<MODEL>(qin, (unsigned)row * pitch + src, oh, ol);
                c2p_mixed<MODEL>(I, P, oh, ol, Wo);
                float rho = h[0] > 1e-12f ? h[0] : oh[0];
                float u = Wn[1], v = Wn[2];
                float p = (P.plus_gp1(Wn[3]) > 0.0f) ? Wn[3] : Wo[3];
                h[0] = rho; l[0] = 0.f;
                h[1] = rho * u; l[1] = 0.f;
                h[2] = rho * v; l[2] = 0.f;
                h[3] = P.plus_gp1(p) * P.i1 + 0.5f * rho * (u * u + v * v); l[3] = 0.f;
            }
        }
        if (writer) store_cell<MODEL>(qout, off_out, h, l);
    }
}

// x sweep: a warp per part of a tile.  Bounded to 64 (Euler) and 96 (Allaire) registers for 8 and 5 CTAs per SM.
//
// Both sweeps are bound by instruction issue: at 2048^2 Euler the x sweep runs
// 263 thread instructions a cell (73 % of the issue slots, 5.3 TB/s of its
// 268 MB, 82 % of the measured copy) and the y sweep 267 (69 %, 4.6 TB/s with
// its close), against 384 and 390 before the slopes, face states and sums went through
// pairs of components, minmod took three instructions, one reciprocal served
// both star quotients, the physicality tests were made on the smallest values
// and the options were fixed at compile time: x 66.2 -> 49.8 us, y 80.4 ->
// 63.9 us a sweep, 57.9 since close_steps closes the steps.  Allaire at
// 2048x1024: x 62.7 -> 45.9 us, then 44.7, y 84.8 -> 68.1, then 60.9 us
// (x with its rows staged and 5 CTAs per SM instead of the next row in
// registers and 4: 49.1 -> 45.9).
template <int MODEL, int OPT>
__global__ void __launch_bounds__(128, MODEL == MODEL_EULER ? 8 : 5)
    mixed_segment_x_kernel(MixedArgs A) {
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (w >= A.ntiles * A.split) return;
    const TileGeom g = tile_geom<DIR_X, kSegCells, kSegRows>(A, w / A.split);
    if (g.skip) return;
    const int n = part_rows(A), r = g.b_org + (w % A.split) * n;  // this warp's rows
    segment_tile<MODEL, OPT>(A, g, r, min(r + n, g.b_org + A.rows));
}

}  // namespace mixed
}  // namespace cfd
