// Resident engine kernels: the arrested-Newton / RK4 step of
// core/integrator.py:284-410 as fused stage launches, whose last block runs the control,
// for a batch of lattice instances at once.
//
// With k1 = dt V, k2 = dt (V + l1/2), k3 = dt (V + l2/2), k4 = dt (V + l3) the
// stage inputs of the reference schedule are
//   X1 = F,  X2 = F + (dt/2) V,  X3 = F + (dt/2)(V + l1/2),  X4 = F + dt (V + l2/2)
// and the update is
//   F' = F + dt (V + (l1 + l2 + l3)/6),   V' = V + (l1 + 2 l2 + 2 l3 + l4)/6
// followed by the theory's normalisation of phi and projection of V'
// (core/integrator.py:163-175).  Stage s builds X_s for its haloed tile on the
// fly from F, V and the previous slope.
//
// F' needs no l4.  So stage 3 already writes the new field, into the other half of a
// ping-pong pair, and the sum l1 + 2 l2 + 2 l3 instead of l3; stage 4 adds l4, projects and leaves
// V'.  The work on the new field -- its energy and the next step's l1 (stage 1) -- then depends on
// stage 3 only and runs beside stage 4:
//   stage 2 -> stage 3 -> { stage 4 | [defect refresh,] [FP32 energy,] stage 1 } -> control.
// l1 alternates between two buffers, since stage 4 of an arrested step reads the old one (l2 = l1)
// while stage 1 writes the new one.
//
// Where one block fills an SM (FP64 stages of at most five components, the fused FP32 rho kernels)
// nothing runs beside stage 4, and the split update's array more would only cost: there stage 3
// writes l3 and stage 4 updates field and velocity (late_update); stage 1 follows it.
//
// The last block of stages 4 and 1 to finish runs every instance's control: it reduces the
// energy, baryon number and stage-4 gradient (compensated, fixed order), records the step's
// (energy, err) exactly as do_arrested_newton_flow returns them, takes the arrest decision for
// the next step (the velocity is treated as zero when killkinen is set and the energy rose,
// core/integrator.py:403-407) and flips the halves.
#pragma once

#include <string.h>

#include "sky_grad.cuh"
#include "sky_kernels.cuh"
#include "sky_rho.cuh"
#include "sky_rho_march.cuh"

namespace sky {

// Per-step statistics written by the control launch: record n describes the
// field after n steps (record 0: the admitted field).
struct StepStats {
    double energy;      // E after step n (FP64, compensated)
    double baryon;      // B after step n
    double err;         // signed max of step n's stage-4 gradient (reference `err`)
    double gabs;        // max |g| of step n's stage-4 gradient
    int arrested;       // velocity treated as zero in step n+1
    int step;           // n
    double kinetic;     // (1/2) h^3 sum |V'|^2 of the velocity step n produced (before any arrest)
    int status;         // the engine's error word when the record was written (0: no error)
    int reserved;
};

// Roles of an instance's TMA plane maps (InstDesc::tm): the haloed plane of a stage tile; the
// field's also of an energy tile (InstDesc::tme, kMapF and kMapFlo).
enum { kMapF = 0, kMapFlo = 2, kMapV = 4, kMapL = 6, kMapDlt = 9, kNumMaps = 10, kNumEnergyMaps = 4 };

// Default number of steps between refreshes of the defect correction of an FP32
// instance (sky_engine_set_defect_period changes it per instance).
constexpr int kDefectRefresh = 16;

// Sets of engine kernels: one per theory, and one for FP32 rho lattices of at most kFusedRhoSites
// sites (k_rho_fused).
constexpr int kFusedRho = 6, kNumKernelSets = 7;
constexpr int64_t kFusedRhoSites = 56 * 56 * 56;
inline int kernel_set(int theory, int prec, int64_t sites) {
    return theory == SKY_THEORY_RHO && prec == 0 && sites <= kFusedRhoSites ? kFusedRho : theory;
}
// Whether a kernel set has its own energy walk; else stage 1 sums the energy.
template <typename T>
constexpr bool energy_walk(int set) {
    return set != kFusedRho && (sizeof(T) == 4 || set == SKY_THEORY_RHO);
}

// Whether stage 4 updates the field (else stage 3 does).
template <typename T>
constexpr bool late_update(int set) {
    return set == kFusedRho || (sizeof(T) == 8 && set != SKY_THEORY_RHO);
}

// Device-resident state of one instance.
template <typename S>
struct InstDesc {
    TmaMap tm[kNumMaps];  // plane maps of F[0..1], Flo[0..1], V[0..1], L[0..2], Dlt (when tma is set)
    TmaMap tme[kNumEnergyMaps];  // energy-tile maps of F and Flo (FP32 instances with an energy walk; rho: the pions')
    TmaMap tmc[kNumEnergyMaps];  // FP32 rho: energy-tile maps of the rho components (as tmr)
    TmaMap tmr[kNumMaps];  // rho: maps of the rho components, 3 planes-long x axes of one isospin component each
    int tma;              // the stage kernels stage this instance's planes with TMA
    int* status;          // the engine's error word (bit 0: a wait for a TMA copy gave up)
    Params p;
    MarchCoef<S> coef;   // stencil scales of the lattice
    double r1d[3];       // ... of the FP64 energy's first derivatives
    S* F[2];           // ping-pong field
    S* Flo[2];         // ping-pong low parts of a compensated FP32 field (null otherwise)
    S* Dlt;            // defect correction g64 - g32 of a defect-corrected FP32 instance (null otherwise)
    S* V[2];           // ping-pong velocity (the next half holds l1 + 2 l2 + 2 l3 between stages 3 and 4)
    double* curl;      // FP32 rho: R^a_xy, R^a_xz, R^a_yz (at 3 a) of the field whose energy is being summed
    S* L[3];           // slopes: l2 in L[1]; l1 of this step and of the next in L[0] and L[2] (l1_slot), or with
                       // a late update l1 in L[0] and l3 in L[2]
    KSum* epart;       // energy partials, per energy tile (k_energy; FP32 rho: four each) or per stage tile (stage 1)
    KSum* bpart;       // per-tile baryon partials (stage 1)
    double* gpart;     // per-tile [signed max, abs max of stage-4 g, kinetic KSum (s, c)] (4 doubles / tile)
    StepStats* stats;  // ring of per-step records
    int stats_cap;
    int tile_begin;    // first global tile index of this instance
    int ntiles;
    int e_parts;       // entries of epart: e_ntiles, four times that for FP32 rho
    int gtiles;        // entries of gpart: ntiles, and for rho those of the rho components' epilogue
    int tiles_nz, tiles_ny, tiles_nx;
    int xc;            // x-chunk of the marching kernels
    int r_tile_begin;  // rho: tiles of the walk over the rho components (three items each)
    MarchGrid r_grid;
    int e_tile_begin, e_ntiles, e_nz, e_ny, e_nx, e_xc;  // energy tiles (e_ntiles = ntiles where stage 1 sums it)
    // control state (device-updated)
    double e_prev;     // energy entering the previous step
    int step;          // steps taken
    int arrested;      // arrest flag for the current step
    int active;        // 0 = skip (retired / paused)
    int cur;           // which half of the F / V ping-pong pairs is current
    int refresh;       // the current l1 comes from a defect refresh
    int refresh_period;  // steps between refreshes of the defect correction
};

// The field's update at one site: F' = F + dt (V + (l1 + l2 + l3)/6), then the theory's
// normalisation of the first nsky components; and sum = l1 + 2 l2 + 2 l3.
// With a compensated field (comp) F is the unevaluated sum hi + lo of two FP32
// values: the update and the normalisation run in FP64 and the result is
// split back into hi + lo, so increments far below one FP32 ulp of F still accumulate.
template <typename T, int C>
__device__ __forceinline__ void update_field(const T (&f0)[C], const T (&flo)[C], bool comp, const T (&v0)[C],
                                             const T (&l1)[C], const T (&l2)[C], const T (&l3)[C], T dtt, int nsky,
                                             int unit_length, T (&fo)[C], T (&lo)[C], T (&sum)[C]) {
    T inc[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        sum[c] = l1[c] + T(2) * l2[c] + T(2) * l3[c];
        inc[c] = dtt * (v0[c] + (l1[c] + l2[c] + l3[c]) * T(1.0 / 6.0));
        lo[c] = T(0);
    }
    if (!comp) {
#pragma unroll
        for (int c = 0; c < C; ++c) fo[c] = f0[c] + inc[c];
        if (unit_length) {
            // one reciprocal square root instead of a square root and nsky divisions
            // (within one unit in the last place of the quotients)
            T ss = T(0);
#pragma unroll
            for (int c = 0; c < C; ++c)
                if (c < nsky) ss += fo[c] * fo[c];
            if (ss != T(0)) {
                const T r = ss == T(1) ? T(1) : rsqrt(ss);  // unit fields (the vacuum shell) stay exact
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (c < nsky) fo[c] *= r;
            }
        }
    } else {
        // hi + lo + inc in FP64, with the two small terms summed in FP32 first: lo and the
        // increment are both far below hi, so their FP32 sum loses no more than the FP32
        // increment and the FP32 low part already do (about 2^-49 of the field).  One
        // reciprocal square root normalises.
        double fd[C];
#pragma unroll
        for (int c = 0; c < C; ++c) fd[c] = double(f0[c]) + double(flo[c] + inc[c]);
        if (unit_length) {
            double ss = 0.0;
#pragma unroll
            for (int c = 0; c < C; ++c)
                if (c < nsky) ss = fma(fd[c], fd[c], ss);
            if (ss != 0.0) {
                const double r = ss == 1.0 ? 1.0 : rsqrt(ss);  // unit fields (the vacuum shell) stay exact
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (c < nsky) fd[c] *= r;
            }
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            fo[c] = T(fd[c]);
            lo[c] = T(fd[c] - double(fo[c]));
        }
    }
}

// The velocity's update: V' = V + (l1 + 2 l2 + 2 l3 + l4)/6 -- the small terms are summed before
// the velocity, which is rounded once (kept as V + (l1 + 2 l2 + 2 l3)/6 between the stages it was
// rounded twice: up to one ulp from the exact sum instead of half of one) -- projected orthogonal to
// the first nsky components of the new field (a compensated field's high parts); returns |V'|^2.
template <typename T, int C>
__device__ __forceinline__ T update_velocity(const T (&v0)[C], const T (&sum)[C], const T (&g)[C], const T (&fo)[C],
                                             T dtt, int nsky, int unit_length, T (&vv)[C]) {
#pragma unroll
    for (int c = 0; c < C; ++c) vv[c] = v0[c] + (sum[c] + -dtt * g[c]) * T(1.0 / 6.0);
    if (unit_length) {
        T lm = T(0);
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (c < nsky) lm += vv[c] * fo[c];
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (c < nsky) vv[c] -= lm * fo[c];
    }
    T v2 = T(0);
#pragma unroll
    for (int c = 0; c < C; ++c) v2 += vv[c] * vv[c];
    return v2;
}

// Whether the work on the new field of the step in flight refreshes the defect correction.
template <typename S>
__device__ __forceinline__ bool refresh_due(const InstDesc<S>& in) {
    const int period = in.refresh_period > 0 ? in.refresh_period : kDefectRefresh;
    return in.Dlt != nullptr && (in.step + 1) % period == 0;
}
// The buffer of the current step's l1 (half 0) or of the next one's (half 1).
template <bool LATE, typename S>
__device__ __forceinline__ int l1_slot(const InstDesc<S>& in, int half) {
    return !LATE && (in.cur ^ half) ? 2 : 0;
}

// ---------------------------------------------------------------------------
// Control of one instance: reduces the partials of the step that ends -- energy and baryon
// number of its new field (stage 1 and the energy walk), its stage-4 gradient and kinetic sum --
// records StepStats and sets the arrest flag.
// ---------------------------------------------------------------------------
// mode 0: end of a step (advances the instance, arrest decision); 1: admission (step 0, no
// arrest); 2: resume after a precision change (keeps the pending arrest decision).
// The work is four warps' (the control kernel, or warps of the last block to finish a step's
// stage-4 and stage-1 launches): lane-strided compensated sums of the per-tile partials, a fixed
// shuffle tree per warp and the warps in order, so the order depends on the tile count only.  The
// partials are read through L2: in the stage kernel they were written by other blocks of the same
// launch.  A step ends with this, so it is laid out for latency: several turns of loads in flight
// (with one warp and one load after the other, 20 us for 1300 partials).
constexpr int kControlWarps = 4;
struct ControlSums {
    KSum e, b, kin;
    double gm, ga;
    __device__ __forceinline__ void merge(const ControlSums& o) {
        ksum_merge(e, o.e);
        ksum_merge(b, o.b);
        ksum_merge(kin, o.kin);
        gm = fmax(gm, o.gm);
        ga = fmax(ga, o.ga);
    }
};
// warp: the calling warp's number among the instance's four; sh: three entries of shared memory;
// bar: a barrier of the four warps.
template <typename S>
__device__ __forceinline__ void engine_control(InstDesc<S>& in, int mode, int warp, ControlSums* sh, int bar) {
    const int lane = (threadIdx.x + blockDim.x * threadIdx.y) & 31;
    ControlSums r{{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, -1.0e300, 0.0};
    constexpr int U = 2, T = 32 * kControlWarps;
    const int ne = in.e_parts, nb = in.ntiles, ng = in.gtiles, n = max(max(ne, nb), ng);
    const KSum *ep = in.epart, *bp = in.bpart;
    const double* gp = in.gpart;
    for (int t0 = 32 * warp + lane; t0 < n; t0 += T * U) {
        double le[U][2], lb[U][2], lg[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) {  // loads past an array's end read its last entry
            const int t = t0 + T * u;
            const int te = min(t, ne - 1), tb = min(t, nb - 1), tg = min(t, ng - 1);
            le[u][0] = __ldcg(&ep[te].s), le[u][1] = __ldcg(&ep[te].c);
            lb[u][0] = __ldcg(&bp[tb].s), lb[u][1] = __ldcg(&bp[tb].c);
#pragma unroll
            for (int k = 0; k < 4; ++k) lg[u][k] = __ldcg(&gp[4 * tg + k]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = t0 + T * u;
            if (t < ne) ksum_merge(r.e, KSum{le[u][0], le[u][1]});
            if (t < nb) ksum_merge(r.b, KSum{lb[u][0], lb[u][1]});
            if (t < ng) {
                r.gm = fmax(r.gm, lg[u][0]);
                r.ga = fmax(r.ga, lg[u][1]);
                ksum_merge(r.kin, KSum{lg[u][2], lg[u][3]});
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        ControlSums o;
        o.e = ksum_shfl_down(r.e, off), o.b = ksum_shfl_down(r.b, off), o.kin = ksum_shfl_down(r.kin, off);
        o.gm = __shfl_down_sync(0xffffffffu, r.gm, off), o.ga = __shfl_down_sync(0xffffffffu, r.ga, off);
        if (lane + off < 32) r.merge(o);
    }
    if (warp > 0 && lane == 0) sh[warp - 1] = r;
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(T) : "memory");
    if (warp == 0 && lane == 0) {
        for (int w = 1; w < kControlWarps; ++w) r.merge(sh[w - 1]);
        const double en = r.e.s + r.e.c;
        if (mode == 1) in.step = 0;
        if (mode == 0) {
            in.refresh = refresh_due(in) ? 1 : 0;
            in.step += 1;
            in.cur ^= 1;
        }
        const int step = in.step;
        // arrest (core/integrator.py:403-407): the energy after step n exceeds the one after step n-1
        int arrest = in.arrested;
        if (mode == 0) arrest = (step > 0 && in.p.killkinen && en > in.e_prev) ? 1 : 0;
        if (mode == 1) arrest = 0;
        StepStats& st = in.stats[step % in.stats_cap];
        st.energy = en;
        st.baryon = r.b.s + r.b.c;
        if (mode != 2) {  // a resume keeps the step's gradient statistics
            st.err = (step > 0) ? r.gm : 0.0;
            st.kinetic = (step > 0) ? r.kin.s + r.kin.c : 0.0;
            st.gabs = (step > 0) ? r.ga : 0.0;
        }
        st.arrested = arrest;
        st.step = step;
        st.status = in.status ? *in.status : 0;
        in.arrested = arrest;
        in.e_prev = en;
    }
    // (the next instance's sums wait for this one's to be read)
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(T) : "memory");
}

// Control of the instances [i_begin, i_end), one block each (admission, precision change; the
// steps themselves fold mode 0 into their last launches).
template <typename S>
__global__ void __launch_bounds__(32 * kControlWarps) k_engine_control(InstDesc<S>* __restrict__ insts, int i_begin, int i_end,
                                                       int mode) {
    const int ii = i_begin + blockIdx.x;
    if (ii >= i_end) return;
    InstDesc<S>& in = insts[ii];
    if (!in.active) return;
    __shared__ ControlSums sh[kControlWarps - 1];
    engine_control(in, mode, threadIdx.x >> 5, sh, 1);
}



// ---------------------------------------------------------------------------
// Stage kernels.  The stage input is built while the x-planes are staged; the epilogue
// writes l_s, or applies the RK4 update.  Every theory runs the gradient walk (sky_grad.cuh,
// k_grad_stage); rho's is over the pion components, between a walk over the rho components
// (sky_rho.cuh, k_rho_stage) and the rho components' epilogue (k_rho_finish).
// ---------------------------------------------------------------------------
// What a tile's stage reads and writes.  `half`: stage 1 works on the new field
// of the step in flight (1) or, at admission and after a precision change, on the current one (0).
template <typename T>
struct StageIo {
    const T* src[3];   // sources of the stage input
    T a, b;            // their weights
    const T *F, *Flo, *V, *l1, *l2;  // the update's operands (V null: zero; Flo null: not compensated)
    T* l3;                           // late update
    // stages 1, 2: l_s.  Stage 3: F', its low parts and the slopes' sum.  Stage 4: F' (read) and the
    // sum, which V' replaces.  Late update: stage 3 l3, stage 4 F', its low parts and V'.
    T *out, *out_lo, *pv;
    T* R;  // rho: where the stage's walk over the rho components leaves R (components 4 .. 12)
    T dtt;
    bool l2_is_l1;
};

// An arrested step treats the velocity as zero, so its stage-2 input F + (dt/2) V is
// the field itself: l2 = l1, and stage 2 has nothing to compute.  Stages 3 and 4 then
// read l1 where they read l2.  Not after a defect refresh: that stage 1 formed l1 from
// the FP64 gradient, and stage 2's FP32 gradient plus the new correction may differ
// from it in the last bit.
template <typename T>
__device__ __forceinline__ bool l2_is_l1(const InstDesc<T>& in) {
    return in.arrested && !in.refresh;
}

template <bool LATE, typename T, int STAGE>
__device__ __forceinline__ StageIo<T> stage_io(const InstDesc<T>& in, const Params& p, int half) {
    const int cur = STAGE == 1 ? in.cur ^ half : in.cur;
    StageIo<T> io;
    io.l2_is_l1 = l2_is_l1(in);
    io.F = in.F[cur];
    io.Flo = in.Flo[cur];
    io.V = in.arrested ? nullptr : in.V[cur];
    io.l1 = in.L[l1_slot<LATE>(in, 0)];
    io.l3 = in.L[2];
    io.l2 = io.l2_is_l1 ? io.l1 : in.L[1];  // the step's l2
    io.dtt = T(p.dt);
    const T hdt = T(0.5 * p.dt);
    io.src[0] = io.F;
    io.src[1] = io.V;
    io.src[2] = STAGE == 3 ? io.l1 : io.l2;
    io.a = STAGE == 4 ? io.dtt : hdt;
    io.b = STAGE == 3 ? T(0.25) * io.dtt : T(0.5) * io.dtt;
    io.out = STAGE == 1 ? in.L[l1_slot<LATE>(in, half)] : STAGE == 2 ? in.L[1] : LATE && STAGE == 3 ? io.l3 : in.F[cur ^ 1];
    io.out_lo = in.Flo[cur ^ 1];
    io.pv = in.V[cur ^ 1];
    // R lies where the stage's output will (stage 4: in the slope that it does not read)
    io.R = STAGE < 3 ? io.out : STAGE == 3 ? io.pv : io.l2_is_l1 ? in.L[1] : in.L[l1_slot<LATE>(in, 0)];
    return io;
}

// The maps of a tile's sources (null: the source reads as zero); tm: the instance's maps of the
// walk's components.
template <bool LATE, typename T, int STAGE>
__device__ __forceinline__ void stage_maps(const InstDesc<T>& in, const TmaMap* tm, const StageIo<T>& io, int half,
                                           TmaTile& tt) {
    const int cur = STAGE == 1 ? in.cur ^ half : in.cur;
    tt.map[0] = &tm[kMapF + cur];
    tt.map[1] = io.V != nullptr ? &tm[kMapV + cur] : nullptr;
    tt.map[2] = STAGE > 2 ? &tm[kMapL + (STAGE == 3 || io.l2_is_l1 ? l1_slot<LATE>(in, 0) : 1)] : nullptr;
    tt.status = in.status;
}

// The stage-4 statistics of a thread's sites.
template <typename T>
struct StageStats {
    T gmx, gab;   // signed and absolute maxima of the thread's stage-4 gradients (exact in T)
    // (1/2) h^3 sum |V'|^2 over the thread's sites: compensated FP64 for an FP64 instance; an
    // FP32 instance's per-site |V'|^2 is an FP32 value and its thread partial (at most one
    // x-chunk of sites) is summed in FP32, then merged per block in FP64
    KSum kin;
    T kin_t;
    T hvol;       // h^3 / 2
    __device__ __forceinline__ explicit StageStats(double vol)
        : gmx(T(-INFINITY)), gab(T(0)), kin{0.0, 0.0}, kin_t(T(0)), hvol(T(0.5 * vol)) {}
    __device__ __forceinline__ void gradient(T g) {
        if (g > gmx) gmx = g;  // (a NaN changes neither, as with fmax)
        if (fabs(g) > gab) gab = fabs(g);
    }
    __device__ __forceinline__ void velocity(T v2) {
        if constexpr (sizeof(T) == 8)
            ksum_add(kin, hvol * v2);
        else
            kin_t += hvol * v2;
    }
    __device__ __forceinline__ KSum kinetic() const { return sizeof(T) == 8 ? kin : KSum{double(kin_t), 0.0}; }
};

// Loads that stay where they are written (a plain load may be moved down to its use, where
// nothing is left to hide its latency).  ONCE: the array is not read again before the next stage
// streams past it, so the line is marked to leave L2 first (ld.cs), as are the stage's results
// (st.cs): the halo rows and the next planes' operands stay instead.  Step, with cg / cs: omega
// defect-corrected FP32 128^3 388 / 380 us, FP64 527 / 513; Coulomb FP64 128^3 805 / 786 (stage 3
// 274 / 253), compensated FP32 192^3 1321 / 1306; lattices that fit L2 the same.  (The drop-in
// stages keep cg: 128^3 omega would gain 1 %, but 64^3 nuclear loses 5 %.)
template <bool ONCE>
__device__ __forceinline__ double ld_early(const double* p) {
    double v;
    if constexpr (ONCE)
        asm volatile("ld.global.cs.f64 %0, [%1];" : "=d"(v) : "l"(p));
    else
        asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
template <bool ONCE>
__device__ __forceinline__ float2 ld_early2(const float* p) {
    float2 v;
    if constexpr (ONCE)
        asm volatile("ld.global.cs.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    else
        asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}

// Epilogue of the gradient walk's stages: a thread's pair of FP32 sites, or its FP64 site, at
// once.  The row pitch is a multiple of four, so a pair is one aligned 8-byte access; where Z is
// odd, the second lane of a row's last pair is padding, which nothing reads as a site.
// EARLY: the field update's operands are loaded before the point arithmetic (where 168 registers
// hold both: without mixed derivatives); of a stage 4 that updates the velocity only, F' and the
// slopes' sum always are, and the velocity, which the staged planes have brought into L2, is not.
template <typename T, int STAGE, int C, bool TMA, bool EARLY, bool LATE>
struct GradEpi {
    static constexpr bool UPDATE = STAGE == (LATE ? 4 : 3);  // the stage that updates the field
    static constexpr int NOP = UPDATE ? 5 : STAGE == 4 ? 3 : 1;
    using L = Lanes<T>;
    using V = typename L::V;
    static constexpr int NL = L::NL;
    StageIo<T> io;
    StageStats<T> st;
    int nsky, unit_length;
    T* dlt;       // defect correction (null unless defect-corrected)
    int refresh;  // stage 1 after the defect refresh: dlt holds g64 of the field; replace it by g64 - g32
    const T* ahead[4];  // operands that the stage reads at the site only (null: none), and their maps
    const TmaMap* ahead_map[4];
    V d[NL > 1 ? C : 1];  // the correction of the site's pair
    V op[NOP][NOP > 1 ? C : 1];  // the update's operands at the site

    template <bool ONCE = true>
    static __device__ __forceinline__ V get(const T* p) {
        if constexpr (NL == 1)
            return ld_early<ONCE>(p);
        else
            return P2(ld_early2<ONCE>(p));
    }
    static __device__ __forceinline__ void store(T* p, V v) {
        if constexpr (NL == 1)
            __stcs(p, v);
        else
            __stcs(reinterpret_cast<float2*>(p), v.v);
    }
    // The next plane of the operands into L2, so that the loads at the site do not wait for DRAM:
    // box prefetches by one thread, or 128-byte lines by each row.
    int z0, y0;
    __device__ __forceinline__ void prefetch(int64_t s0, int64_t N, int lane, int n, int x) {
        if constexpr (TMA) {
            if (threadIdx.x == 0 && threadIdx.y == 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (ahead_map[k]) tma_prefetch_plane(ahead_map[k], z0, y0, x, 0);
            }
        } else {
            constexpr int Q = sizeof(T) == 8 ? 3 : 2, PER = 128 / int(sizeof(T));  // lines a row can span
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (ahead[k] == nullptr) continue;
                for (int i = lane; i < Q * C; i += M_TZ) {
                    const int c = i / Q, q = i - Q * c;
                    prefetch_l2(ahead[k] + c * N + s0 + min(PER * q, n - 1));
                }
            }
        }
    }
    static constexpr int M_TZ = 32 / NL;
    __device__ __forceinline__ void begin_site(int64_t s, int64_t N, bool) {
        if constexpr (NL > 1) {
            if (dlt) {
#pragma unroll
                for (int c = 0; c < C; ++c) d[c] = get(dlt + at(c, N, s));
            }
        }
    }
    // element index of component c at site s (C N < 2^31)
    static __device__ __forceinline__ uint32_t at(int c, int64_t N, int64_t s) {
        return uint32_t(c) * uint32_t(N) + uint32_t(s);
    }
    __device__ __forceinline__ void load(int64_t s, int64_t N, bool) {
        if constexpr (EARLY || (STAGE == 4 && !UPDATE)) operands(s, N);
    }
    __device__ __forceinline__ void operands(int64_t s, int64_t N) {
        if constexpr (UPDATE) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const uint32_t j = at(c, N, s);
                op[0][c] = get(io.F + j);
                op[1][c] = LATE ? get(io.l3 + j) : io.Flo ? get(io.Flo + j) : V(0.0f);
                op[2][c] = io.V ? get(io.V + j) : V(0.0f);
                op[3][c] = get(io.l1 + j);
                op[4][c] = io.l2_is_l1 ? op[3][c] : get(io.l2 + j);
            }
        } else if constexpr (STAGE == 4) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                op[0][c] = get(io.out + at(c, N, s));
                op[1][c] = get(io.pv + at(c, N, s));
            }
        }
    }
    __device__ __forceinline__ void operator()(int64_t s, int64_t N, bool own1, const V (&)[C], const V (&g32)[C]) {
        V g[C];
#pragma unroll
        for (int c = 0; c < C; ++c) g[c] = g32[c];
        if constexpr (NL > 1) {
            if (dlt) {
                if (STAGE == 1 && refresh) {  // d = g64(F): the correction becomes g64 - g32(F)
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        store(dlt + at(c, N, s), d[c] - g32[c]);
                        g[c] = d[c];
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < C; ++c) g[c] = g32[c] + d[c];
                }
            }
        }
        if constexpr (STAGE < 3 || (LATE && STAGE == 3)) {
#pragma unroll
            for (int c = 0; c < C; ++c) store(io.out + at(c, N, s), V(-io.dtt) * g[c]);
        } else if constexpr (STAGE == 3) {
            if constexpr (!EARLY) operands(s, N);
            V fo[C], lo[C], sum[C];
#pragma unroll
            for (int c = 0; c < C; ++c) g[c] = V(-io.dtt) * g[c];  // l3
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                T F[C], Fl[C], v[C], b1[C], b2[C], b3[C], of[C], ol[C], sn[C];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    F[c] = L::get(op[0][c], l), Fl[c] = L::get(op[1][c], l), v[c] = L::get(op[2][c], l);
                    b1[c] = L::get(op[3][c], l), b2[c] = L::get(op[4][c], l), b3[c] = L::get(g[c], l);
                }
                update_field<T, C>(F, Fl, io.Flo != nullptr, v, b1, b2, b3, io.dtt, nsky, unit_length, of, ol, sn);
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    L::set(fo[c], l, of[c]);
                    L::set(lo[c], l, ol[c]);
                    L::set(sum[c], l, sn[c]);
                }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const uint32_t j = at(c, N, s);
                store(io.out + j, fo[c]);
                if (io.Flo) store(io.out_lo + j, lo[c]);
                store(io.pv + j, sum[c]);
            }
        } else if constexpr (LATE) {
            static_assert(NL == 1, "FP64 sites");
            if constexpr (!EARLY) operands(s, N);
            T zero[C], of[C], ol[C], sum[C], ov[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                zero[c] = T(0);
                st.gradient(g[c]);
            }
            update_field<T, C>(op[0], zero, false, op[2], op[3], op[4], op[1], io.dtt, nsky, unit_length, of, ol, sum);
            st.velocity(update_velocity<T, C>(op[2], sum, g, of, io.dtt, nsky, unit_length, ov));
#pragma unroll
            for (int c = 0; c < C; ++c) {
                store(io.out + at(c, N, s), of[c]);
                store(io.pv + at(c, N, s), ov[c]);
            }
        } else {
            V (&fo)[C] = op[0], (&sum)[C] = op[1], (&v0)[C] = op[2];
#pragma unroll
            for (int c = 0; c < C; ++c) v0[c] = io.V ? get(io.V + at(c, N, s)) : V(0.0f);
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                if (l == 1 && !own1) break;
                T F[C], v[C], sm[C], gg[C], ov[C];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    F[c] = L::get(fo[c], l), v[c] = L::get(v0[c], l), sm[c] = L::get(sum[c], l), gg[c] = L::get(g[c], l);
                    st.gradient(gg[c]);
                }
                st.velocity(update_velocity<T, C>(v, sm, gg, F, io.dtt, nsky, unit_length, ov));
#pragma unroll
                for (int c = 0; c < C; ++c) L::set(sum[c], l, ov[c]);
            }
#pragma unroll
            for (int c = 0; c < C; ++c) store(io.pv + at(c, N, s), sum[c]);
        }
    }
};

// Rho: the walk over the pion components takes R at the site and leaves H in its place
// (k_rho_finish applies it).
template <typename T, int STAGE, bool TMA>
struct RhoGradEpi : GradEpi<T, STAGE, 4, TMA, false, false> {
    using B = GradEpi<T, STAGE, 4, TMA, false, false>;
    using V = typename Lanes<T>::V;
    static constexpr bool kCoupled = true;
    __device__ __forceinline__ void coupling(int64_t s, int64_t N, bool, V (&R)[9]) {
#pragma unroll
        for (int m = 0; m < 9; ++m) R[m] = B::template get<false>(B::io.R + B::at(4 + m, N, s));
    }
    __device__ __forceinline__ void coupled(int64_t s, int64_t N, bool own1, const V (&J)[9], const Params& p) {
        V R[9];  // (read again, not held)
        coupling(s, N, own1, R);
#pragma unroll
        for (int m = 0; m < 9; ++m) B::store(B::io.R + B::at(4 + m, N, s), rho_rest(R[m], J[m], p));
    }
};
template <template <typename> class Th, typename T, int STAGE, class M, bool TMA>
using StageEpi = typename std::conditional<Th<T>::kId == SKY_THEORY_RHO, RhoGradEpi<T, STAGE, TMA>,
                                           GradEpi<T, STAGE, M::C, TMA, !Th<T>::kMixed, late_update<T>(Th<T>::kId)>>::type;

// A finished tile's partials: stage 1 the baryon number and (FP64) the energy, stage 4 the
// gradient maxima and the kinetic sum.
template <typename T, int STAGE>
__device__ __forceinline__ void tile_partials(const InstDesc<T>& in, int lt, const KSum& es, const KSum& bs,
                                              const StageStats<T>& st, bool energy, KSum* shk, double* shm) {
    const bool first = threadIdx.x == 0 && threadIdx.y == 0;
    if constexpr (STAGE == 1) {
        const KSum bb = block_ksum(bs, shk);
        if (first) in.bpart[lt] = bb;
        if (energy) {
            const KSum be = block_ksum(es, shk);
            if (first) in.epart[lt] = be;
        }
    }
    if constexpr (STAGE == 4) {
        // a thread without sites keeps -inf, which block_max maps below every gradient
        const double ga = block_max(fmax(double(st.gmx), -1.0e300), shm);
        const double gb = block_max(double(st.gab), shm);
        const KSum kk = block_ksum(st.kinetic(), shk);
        if (first) {
            in.gpart[4 * lt] = ga;
            in.gpart[4 * lt + 1] = gb;
            in.gpart[4 * lt + 2] = kk.s;
            in.gpart[4 * lt + 3] = kk.c;
        }
    }
}

// Tail of a step's stage-4 and stage-1 launches (total > 0: their blocks together): the last
// block of the two to finish runs the control of every active instance of the group, four warps
// per instance, so a step needs no separate launch for it.  Each block publishes its partials
// (fence) before it is counted; the counter returns to 0 for the next step.  The tail sits after
// the tile loop so that its registers do not add to the stencil loop's.
template <typename T, int STAGE>
__device__ __forceinline__ void stage_tail(InstDesc<T>* ctl, const int* tile_inst, int t_begin, int t_end, int* done,
                                           int total) {
    if constexpr (STAGE == 1 || STAGE == 4) {
        if (total > 0) {
            __shared__ int last_block;
            const int ltid = threadIdx.x + blockDim.x * threadIdx.y;
            __syncthreads();
            if (ltid == 0) {
                __threadfence();
                last_block = atomicAdd(done, 1) == total - 1 ? 1 : 0;
            }
            __syncthreads();
            if (last_block) {
                __threadfence();
                __shared__ ControlSums sh[4][kControlWarps - 1];
                const int ng = int(blockDim.x * blockDim.y) / (32 * kControlWarps);  // 1 to 4
                const int g = ltid / (32 * kControlWarps);
                const int i1 = __ldg(tile_inst + t_end - 1) + 1;
                if (g < ng)
                    for (int i = __ldg(tile_inst + t_begin) + g; i < i1; i += ng)
                        if (ctl[i].active)
                            engine_control(ctl[i], 0, (ltid >> 5) % kControlWarps, sh[g], 1 + g);
                if (ltid == 0) *done = 0;
            }
        }
    }
}

template <int STAGE>
constexpr int stage_nsrc() {
    return STAGE == 1 ? 1 : (STAGE == 2 ? 2 : 3);
}

// Shared memory of a walk's stage launch (TMA boxes land on 128-byte boundaries).
template <template <typename> class Th, class M, typename T, int STAGE, bool TMA>
constexpr size_t grad_stage_bytes() {
    return GradPipe<Th, M, T, T, stage_nsrc<STAGE>(), TMA>::bytes + (TMA ? 128 : 0);
}

template <template <typename> class Th, class M, typename T, int STAGE, int MINB, bool TMA>
__global__ void __launch_bounds__(GradBlock<M, T>::NT, MINB)
    k_grad_stage(const InstDesc<T>* __restrict__ insts, InstDesc<T>* ctl, const int* __restrict__ tile_inst,
                 int t_begin, int t_end, int half, int* done, int total) {
    constexpr int NSRC = stage_nsrc<STAGE>();
    constexpr int NW = GradBlock<M, T>::NT / 32;
    extern __shared__ __align__(128) unsigned char smraw[];
    T* sm = reinterpret_cast<T*>(smraw + (TMA ? ((128u - (smem_addr(smraw) & 127u)) & 127u) : 0u));
    __shared__ KSum shk[NW];
    __shared__ double shm[NW];
    __shared__ uint64_t tma_bar;
    __shared__ MarchCoef<T> coef;
    TmaTile tt{&tma_bar, 0u, {nullptr, nullptr, nullptr}, nullptr};
    const bool first = threadIdx.x == 0 && threadIdx.y == 0;
    if constexpr (TMA) {
        if (first) mbar_init(&tma_bar, 1);
        __syncthreads();
    }
    // the previous launch of the step (its tail writes the control state) must be complete
    grid_dep_wait();
    for (int t = t_begin + blockIdx.x; t < t_end; t += gridDim.x) {
        const InstDesc<T>& in = insts[__ldg(tile_inst + t)];
        if (!in.active) continue;  // uniform across the block
        if (STAGE == 2 && l2_is_l1(in)) continue;
        const Params p = in.p;
        const int lt = t - in.tile_begin;
        const MarchGrid mg{in.tiles_nz, in.tiles_ny, in.tiles_nx, in.xc};
        int xa, xe, y0, z0;
        march_origin(mg, lt, M::BY, xa, xe, y0, z0, p.X);
        using Epi = StageEpi<Th, T, STAGE, M, TMA>;
        constexpr bool LATE = late_update<T>(Th<T>::kId);
        Epi epi{GradEpi<T, STAGE, M::C, TMA, !Th<T>::kMixed, LATE>{
            stage_io<LATE, T, STAGE>(in, p, half), StageStats<T>(p.vol), p.nsky, p.unit_length, in.Dlt,
            STAGE == 1 && half && refresh_due(in), {nullptr, nullptr, nullptr, nullptr},
            {nullptr, nullptr, nullptr, nullptr}}};
        epi.z0 = z0;
        epi.y0 = y0;
        // what the staged sources have not brought into L2 already
        auto ahead = [&](int k, const T* a, int map) {
            epi.ahead[k] = a;
            epi.ahead_map[k] = a != nullptr ? &in.tm[map] : nullptr;
        };
        if constexpr (LATE && STAGE == 4) {
            ahead(0, epi.io.l3, kMapL + 2);
            ahead(1, epi.io.l2_is_l1 ? nullptr : epi.io.l1, kMapL);
        } else if constexpr (STAGE == 3 && !LATE) {
            ahead(0, epi.io.Flo, kMapFlo + in.cur);
            ahead(1, epi.io.l2_is_l1 ? nullptr : epi.io.l2, kMapL + 1);
        }
        if constexpr (STAGE == 4 && !LATE) {
            ahead(0, epi.io.out, kMapF + (in.cur ^ 1));
            ahead(1, epi.io.pv, kMapV + (in.cur ^ 1));
        }
        ahead(3, in.Dlt, kMapDlt);
        if constexpr (TMA) stage_maps<LATE, T, STAGE>(in, in.tm, epi.io, half, tt);
        __syncthreads();  // the previous tile's readers of coef are done
        if (first) coef = in.coef;
        __syncthreads();
        KSum es{0.0, 0.0}, bs{0.0, 0.0};
        constexpr bool own_energy = energy_walk<T>(Th<T>::kId);  // else stage 1 sums the energy
        const bool ok = grad_tile<Th, M, T, NSRC, STAGE == 1 ? (own_energy ? 2 : 1) : 0, Epi, T, TMA>(
            sm, p, coef, epi.io.src, epi.io.a, epi.io.b, xa, xe, y0, z0, epi, es, bs, &tt);
        if (!ok) break;  // a copy did not arrive; the error bit is set and the tile's partials stay stale
        tile_partials<T, STAGE>(in, lt, es, bs, epi.st, !own_energy, shk, shm);
    }
    grid_dep_launch();  // the next launch may be scheduled while the last blocks finish
    stage_tail<T, STAGE>(ctl, tile_inst, t_begin, t_end, done, total);
}

// ---------------------------------------------------------------------------
// Rho's first walk of a stage: R of the stage input (sky_rho.cuh), over tiles of its own, each of
// which gives three items, one per isospin component.
// ---------------------------------------------------------------------------
template <class M, typename T, int STAGE, bool TMA>
constexpr size_t rho_stage_bytes() {
    return RhoPipe<M, T, T, stage_nsrc<STAGE>(), TMA>::bytes + (TMA ? 128 : 0);
}

template <class M, typename T, int STAGE, int MINB, bool TMA>
__global__ void __launch_bounds__(GradBlock<M, T>::NT, MINB)
    k_rho_stage(const InstDesc<T>* __restrict__ insts, const int* __restrict__ tile_inst, int t_begin, int t_end,
                int half) {
    constexpr int NSRC = stage_nsrc<STAGE>();
    extern __shared__ __align__(128) unsigned char smraw[];
    T* sm = reinterpret_cast<T*>(smraw + (TMA ? ((128u - (smem_addr(smraw) & 127u)) & 127u) : 0u));
    __shared__ uint64_t tma_bar;
    __shared__ MarchCoef<T> coef;
    TmaTile tt{&tma_bar, 0u, {nullptr, nullptr, nullptr}, nullptr};
    const bool first = threadIdx.x == 0 && threadIdx.y == 0;
    if constexpr (TMA) {
        if (first) mbar_init(&tma_bar, 1);
        __syncthreads();
    }
    grid_dep_wait();
    for (int q = 3 * t_begin + blockIdx.x; q < 3 * t_end; q += gridDim.x) {
        const int t = q / 3, a = q - 3 * t;
        const InstDesc<T>& in = insts[__ldg(tile_inst + t)];
        if (!in.active) continue;  // uniform across the block
        if (STAGE == 2 && l2_is_l1(in)) continue;
        const Params p = in.p;
        int xa, xe, y0, z0;
        march_origin(in.r_grid, t - in.r_tile_begin, M::BY, xa, xe, y0, z0, p.X);
        const StageIo<T> io = stage_io<false, T, STAGE>(in, p, half);
        const int64_t N = n_sites(p), c0 = (4 + a) * N;
        const T* const src[3] = {io.src[0] + c0, io.src[1] ? io.src[1] + c0 : nullptr, io.src[2] + c0};
        if constexpr (TMA) {
            stage_maps<false, T, STAGE>(in, in.tmr, io, half, tt);
            tt.x0 = a * p.X;
        }
        __syncthreads();  // the previous tile's readers of coef are done
        if (first) coef = in.coef;
        __syncthreads();
        if (!rho_tile<M, T, NSRC, T, TMA>(sm, p, coef, src, io.a, io.b, xa, xe, y0, z0, io.R + c0, 3 * N, 3 * N,
                                              &tt))
            break;
    }
    grid_dep_launch();
}

// Rho's last kernel of a stage: the rho components' gradient 8 m_rho^2 X - H and what the
// epilogue of the gradient walk does with the pions' (the rho components are neither normalised
// nor projected).  Element by element over the nine components, 16 bytes per thread and array, an
// equal share of them per item.  In the epilogue of the pion walk the same work was a chain of
// dependent L2 round trips per plane and spilled: that walk 67 us at stage 3 of 64^3 FP32 sites
// and 82 of 57 x 50 x 45 FP64 ones.
template <typename T>
struct Vec16 {
    static constexpr int W = 16 / int(sizeof(T));
    using V4 = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
    T v[W];
    __device__ __forceinline__ void load(const T* p) {
        const V4 q = __ldcs(reinterpret_cast<const V4*>(p));
        memcpy(v, &q, 16);
    }
    __device__ __forceinline__ void store(T* p) const {
        V4 q;
        memcpy(&q, v, 16);
        __stcs(reinterpret_cast<V4*>(p), q);
    }
};
constexpr int kRhoFinishThreads = 256;
constexpr int kRhoFinishSplit = 2;  // items per tile of the walk over the rho components

template <typename T, int STAGE>
__global__ void __launch_bounds__(kRhoFinishThreads)
    k_rho_finish(const InstDesc<T>* __restrict__ insts, InstDesc<T>* ctl, const int* __restrict__ tile_inst,
                 int t_begin, int t_end, int half, int* done, int total) {
    using V = Vec16<T>;
    constexpr int W = V::W;
    __shared__ KSum shk[kRhoFinishThreads / 32];
    __shared__ double shm[kRhoFinishThreads / 32];
    grid_dep_wait();
    constexpr int K = kRhoFinishSplit;
    for (int u = K * t_begin + blockIdx.x; u < K * t_end; u += gridDim.x) {
        const int t = u / K;
        const InstDesc<T>& in = insts[__ldg(tile_inst + t)];
        if (!in.active) continue;  // uniform across the block
        if (STAGE == 2 && l2_is_l1(in)) continue;
        const Params p = in.p;
        const int lt = u - K * in.r_tile_begin, items = K * in.r_grid.count();
        const StageIo<T> io = stage_io<false, T, STAGE>(in, p, half);
        const bool refresh = STAGE == 1 && half && refresh_due(in);
        T* const dlt = in.Dlt;
        StageStats<T> st(p.vol);
        const int64_t N = n_sites(p), c0 = 4 * N, nv = 9 * N / W;  // (rows are whole vectors)
        const int64_t v0 = nv * lt / items, v1 = nv * (lt + 1) / items;
        for (int64_t q = v0 + threadIdx.x; q < v1; q += kRhoFinishThreads) {
            const int64_t j = c0 + q * W;
            // values that are sites (the others pad the row; they take no part in the statistics)
            const int n = STAGE < 4 || p.Zp == p.Z ? W : p.Z - int(uint32_t(j) % uint32_t(p.Zp));
            V x, v, l, l2, lo, d, h, pv;
            x.load(io.src[0] + j);
            h.load(io.R + j);
            if (STAGE > 1 && io.src[1]) v.load(io.src[1] + j);
            if (STAGE > 2) l.load(io.src[2] + j);
            if (STAGE == 3 && !io.l2_is_l1) l2.load(io.l2 + j);
            if (STAGE == 3 && io.Flo) lo.load(io.Flo + j);
            if (STAGE == 4) pv.load(io.pv + j);
            if (dlt) d.load(dlt + j);
            V o1, o2, o3;
#pragma unroll
            for (int i = 0; i < W; ++i) {
                T X = x.v[i];
                const T vi = STAGE > 1 && io.src[1] ? v.v[i] : T(0);
                if (STAGE > 1) X += io.a * vi;
                if (STAGE > 2) X += io.b * l.v[i];
                T g = rho_gradient(X, h.v[i], p);
                if (dlt) {
                    if (refresh) {  // d = g64(F): the correction becomes g64 - g32(F)
                        const T g64 = d.v[i];
                        d.v[i] = g64 - g;
                        g = g64;
                    } else {
                        g += d.v[i];
                    }
                }
                if constexpr (STAGE < 3) {
                    o1.v[i] = -io.dtt * g;
                } else if constexpr (STAGE == 3) {
                    const T F[1] = {x.v[i]}, Fl[1] = {io.Flo ? lo.v[i] : T(0)}, V0[1] = {vi};
                    const T b1[1] = {l.v[i]}, b2[1] = {io.l2_is_l1 ? l.v[i] : l2.v[i]}, b3[1] = {-io.dtt * g};
                    T of[1], ol[1], op[1];
                    update_field<T, 1>(F, Fl, io.Flo != nullptr, V0, b1, b2, b3, io.dtt, 0, 0, of, ol, op);
                    o1.v[i] = of[0], o2.v[i] = ol[0], o3.v[i] = op[0];
                } else {
                    const T V0[1] = {vi}, sum[1] = {pv.v[i]}, gg[1] = {g};
                    T o[1];
                    const T v2 = update_velocity<T, 1>(V0, sum, gg, V0, io.dtt, 0, 0, o);
                    if (i < n) {
                        st.gradient(g);
                        st.velocity(v2);
                    }
                    o1.v[i] = o[0];
                }
            }
            if (refresh && dlt) d.store(dlt + j);
            o1.store((STAGE == 4 ? io.pv : io.out) + j);
            if constexpr (STAGE == 3) {
                if (io.Flo) o2.store(io.out_lo + j);
                o3.store(io.pv + j);
            }
        }
        if constexpr (STAGE == 4) tile_partials<T, STAGE>(in, in.ntiles + lt, KSum{}, KSum{}, st, false, shk, shm);
    }
    grid_dep_launch();
    stage_tail<T, STAGE>(ctl, tile_inst, t_begin, t_end, done, total);
}

// ---------------------------------------------------------------------------
// Small FP32 rho lattices: all thirteen components in one walk, one site per thread.  The three
// kernels of a stage above are faster where they fill the GPU; up to kFusedRhoSites sites their
// launches, their smaller tiles' halos and the separate energy cost more than they give.  Step in
// us, fused / separate: FP32 48^3 148 / 171, 57 x 50 x 45 237 / 249, 64^3 252 / 243;
// defect-corrected 48^3 168 / 204, 64^3 306 / 295, 72^3 505 / 421, 96^3 786 / 700.
// ---------------------------------------------------------------------------
template <class M, int STAGE, bool TMA>
constexpr size_t rho_fused_bytes() {
    return rho_march_bytes<M>(stage_nsrc<STAGE>(), TMA) + (TMA ? 128 : 0);
}

template <int STAGE>
struct RhoFusedEpi {
    static constexpr int C = 13;
    StageIo<float> io;
    StageStats<float> st;
    int nsky, unit_length;
    float* dlt;
    bool refresh;  // stage 1 after the defect refresh: dlt holds g64 of the field; replace it by g64 - g32
    __device__ __forceinline__ void operator()(int64_t s, int64_t N, float (&g)[C]) {
        if (dlt) {
            // all loads before the refresh's stores, which the compiler does not move them across:
            // one latency and not thirteen (defect-corrected 56^3 sites: 244 -> 218 us per step)
            float d[C];
#pragma unroll
            for (int c = 0; c < C; ++c) d[c] = __ldcg(dlt + c * N + s);
            if (STAGE == 1 && refresh) {
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    __stcg(dlt + c * N + s, d[c] - g[c]);
                    g[c] = d[c];
                }
            } else {
#pragma unroll
                for (int c = 0; c < C; ++c) g[c] += d[c];
            }
        }
        if constexpr (STAGE < 4) {
#pragma unroll
            for (int c = 0; c < C; ++c) __stcg(io.out + c * N + s, -io.dtt * g[c]);
        } else {
            // the operands are read-only here: non-coherent loads
            float f0[C], fl[C], v0[C], a1[C], a2[C], a3[C], fo[C], lo[C], sum[C], vv[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                st.gmx = fmax(st.gmx, g[c]);
                st.gab = fmax(st.gab, fabs(g[c]));
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int64_t j = c * N + s;
                f0[c] = __ldg(io.F + j);
                fl[c] = io.Flo ? __ldg(io.Flo + j) : 0.0f;
                v0[c] = io.V ? __ldg(io.V + j) : 0.0f;
                a1[c] = __ldg(io.l1 + j);
                a2[c] = __ldg(io.l2 + j);
                a3[c] = __ldg(io.l3 + j);
            }
            update_field<float, C>(f0, fl, io.Flo != nullptr, v0, a1, a2, a3, io.dtt, nsky, unit_length, fo, lo, sum);
            st.velocity(update_velocity<float, C>(v0, sum, g, fo, io.dtt, nsky, unit_length, vv));
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int64_t j = c * N + s;
                __stcg(io.out + j, fo[c]);
                if (io.Flo) __stcg(io.out_lo + j, lo[c]);
                __stcg(io.pv + j, vv[c]);
            }
        }
    }
};

template <class M, int STAGE, bool TMA>
__global__ void __launch_bounds__(M::NTHREADS)
    k_rho_fused(const InstDesc<float>* __restrict__ insts, InstDesc<float>* ctl, const int* __restrict__ tile_inst,
                int t_begin, int t_end, int half, int* done, int total) {
    extern __shared__ __align__(128) unsigned char smraw[];
    float* sm = reinterpret_cast<float*>(smraw + (TMA ? ((128u - (smem_addr(smraw) & 127u)) & 127u) : 0u));
    __shared__ KSum shk[M::NTHREADS / 32];
    __shared__ double shm[M::NTHREADS / 32];
    __shared__ uint64_t tma_bar;
    TmaTile tt{&tma_bar, 0u, {nullptr, nullptr, nullptr}, nullptr};
    if constexpr (TMA) {
        if (threadIdx.x == 0 && threadIdx.y == 0) mbar_init(&tma_bar, 1);
        __syncthreads();
    }
    grid_dep_wait();
    for (int t = t_begin + blockIdx.x; t < t_end; t += gridDim.x) {
        const InstDesc<float>& in = insts[__ldg(tile_inst + t)];
        if (!in.active) continue;  // uniform across the block
        if (STAGE == 2 && l2_is_l1(in)) continue;
        const Params p = in.p;
        const int lt = t - in.tile_begin;
        const MarchGrid mg{in.tiles_nz, in.tiles_ny, in.tiles_nx, in.xc};
        int xa, xe, y0, z0;
        march_origin(mg, lt, M::BY, xa, xe, y0, z0, p.X);
        RhoFusedEpi<STAGE> epi{stage_io<true, float, STAGE>(in, p, half), StageStats<float>(p.vol), p.nsky, p.unit_length,
                               in.Dlt, STAGE == 1 && half && refresh_due(in)};
        if constexpr (TMA) stage_maps<true, float, STAGE>(in, in.tm, epi.io, half, tt);
        KSum es{0.0, 0.0}, bs{0.0, 0.0};
        const bool ok = rho_march_tile<M, stage_nsrc<STAGE>(), STAGE == 1, TMA>(
            sm, p, epi.io.src, epi.io.a, epi.io.b, xa, xe, y0, z0, epi, es, bs, TMA ? &tt : nullptr);
        if (!ok) break;  // a copy did not arrive; the error bit is set and the tile's partials stay stale
        tile_partials<float, STAGE>(in, lt, es, bs, epi.st, true, shk, shm);
    }
    grid_dep_launch();
    stage_tail<float, STAGE>(ctl, tile_inst, t_begin, t_end, done, total);
}

// ---------------------------------------------------------------------------
// Energy of FP32 instances, and of rho in both precisions: the FP64 density of the field (high
// plus low parts of a compensated one), evaluated in its own walk.  An FP32 value is converted
// once as it enters the FP64 ring.  (Inside stage 1 the 60 tap differences of a five-component site each needed an
// exact FP32 difference and two conversions: half of that stage's instructions.)
// ---------------------------------------------------------------------------

//
// FP32 rho: the thirteen components and their staged FP32 planes in one walk fill an SM with a
// block of 192 threads (60 us at 64^3 sites, and nothing beside it).  So a walk over the rho
// components, three at a time, sums their own part and leaves the curls, and one over the pions
// reads them.  (FP64, where 256 threads fit, keeps one walk: 35 us at 57 x 50 x 45 sites, and 41
// in two.)
template <template <typename> class Th>
struct EnergyOp {
    const Params& p;
    const double* curl;
    int64_t N;
    KSum sum;
    static constexpr int C = Th<double>::C;
    __device__ __forceinline__ void operator()(int64_t s, int, const double (&phi)[C], const double (&D)[3][C]) {
        if constexpr (std::is_same<Th<double>, RhoPion<double>>::value) {
            double R[9];
#pragma unroll
            for (int m = 0; m < 9; ++m) R[m] = __ldcg(curl + m * N + s);
            ksum_add(sum, Th<double>::energy(phi, D, R, p));
        } else {
            ksum_add(sum, Th<double>::energy(phi, D, p));
        }
    }
};
struct CurlOp {
    const Params& p;
    double* curl;  // of the isospin component
    int64_t N;
    KSum sum;
    __device__ __forceinline__ void operator()(int64_t s, int, const double (&r)[3], const double (&D)[3][3]) {
        const double R[3] = {D[0][1] - D[1][0], D[0][2] - D[2][0], D[1][2] - D[2][1]};
#pragma unroll
        for (int q = 0; q < 3; ++q) __stcg(curl + q * N + s, R[q]);
        ksum_add(sum, RhoPion<double>::rho_energy(r, R, p));
    }
};

// CURL: rho's walk over the rho components (M::C = 3, three items per tile).
template <template <typename> class Th, class M, typename S, bool TMA, bool CURL>
__global__ void __launch_bounds__(M::NTHREADS, M::C > 5 ? 1 : 2)
    k_energy(const InstDesc<S>* __restrict__ insts, const int* __restrict__ tile_inst, int t_begin, int t_end,
             int half) {
    extern __shared__ __align__(128) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw + (TMA ? ((128u - (smem_addr(smraw) & 127u)) & 127u) : 0u));
    __shared__ KSum shk[M::NTHREADS / 32];
    __shared__ uint64_t tma_bar;
    constexpr int NSRC = std::is_same<S, double>::value ? 1 : 2;
    constexpr bool SPLIT = std::is_same<Th<double>, RhoPion<double>>::value;
    constexpr int PER = CURL ? 3 : 1;
    TmaTile tt{&tma_bar, 0u, {nullptr, nullptr, nullptr}, nullptr};
    if constexpr (TMA) {
        if (threadIdx.x == 0 && threadIdx.y == 0) mbar_init(&tma_bar, 1);
        __syncthreads();
    }
    grid_dep_wait();
    for (int u = PER * t_begin + blockIdx.x; u < PER * t_end; u += gridDim.x) {
        const int t = u / PER, a = u - PER * t;
        const InstDesc<S>& in = insts[__ldg(tile_inst + t)];
        if (!in.active) continue;
        const Params p = in.p;
        const int lt = t - in.e_tile_begin, cur = in.cur ^ half;
        const MarchGrid mg{in.e_nz, in.e_ny, in.e_nx, in.e_xc};
        int xa, xe, y0, z0;
        march_origin(mg, lt, M::BY, xa, xe, y0, z0, p.X);
        const double r1[3] = {in.r1d[0], in.r1d[1], in.r1d[2]};
        const int64_t N = n_sites(p), c0 = CURL ? (4 + a) * N : 0;
        const S* const src[3] = {in.F[cur] + c0, in.Flo[cur] ? in.Flo[cur] + c0 : nullptr, nullptr};
        if constexpr (TMA) {
            const TmaMap* tm = CURL ? in.tmc : in.tme;
            tt.map[0] = &tm[kMapF + cur];
            tt.map[1] = in.Flo[cur] != nullptr ? &tm[kMapFlo + cur] : nullptr;
            tt.x0 = a * p.X;
            tt.status = in.status;
        }
        KSum sum;
        if constexpr (CURL) {
            CurlOp op{p, in.curl + 3 * a * N, N, KSum{0.0, 0.0}};
            if (!dens_tile<M, S, NSRC, TMA, true>(sm, p, r1, src, xa, xe, y0, z0, op, &tt, 3 * N)) break;
            sum = op.sum;
        } else {
            EnergyOp<Th> op{p, in.curl, N, KSum{0.0, 0.0}};
            if (!dens_tile<M, S, NSRC, TMA>(sm, p, r1, src, xa, xe, y0, z0, op, &tt)) break;
            sum = op.sum;
        }
        const KSum e = block_ksum(sum, shk);
        if (threadIdx.x == 0 && threadIdx.y == 0) in.epart[SPLIT ? 4 * lt + (CURL ? 1 + a : 0) : lt] = e;
    }
    grid_dep_launch();
}

// ---------------------------------------------------------------------------
// Defect refresh: for every defect-corrected FP32 instance whose refresh is due, the FP64
// gradient of the step's new compensated field hi + lo (staged from the FP32
// arrays into an FP64 ring) is written to Dlt; the following stage 1 turns it
// into the correction g64 - g32.
// ---------------------------------------------------------------------------
struct DefectEpi {
    float* dlt;
    template <int C>
    __device__ __forceinline__ void operator()(int64_t s, int64_t N, bool, const double (&)[C], const double (&g)[C]) {
#pragma unroll
        for (int c = 0; c < C; ++c) dlt[c * N + s] = float(g[c]);
    }
};
// Rho: R_j^a of the new field, in FP64, lies in slope buffer a (all three are free between
// stage 4 and the next stage 1).
struct RhoDefectEpi : DefectEpi {
    static constexpr bool kCoupled = true;
    const double* r[3];
    const float *F, *Flo;
    __device__ __forceinline__ void coupling(int64_t s, int64_t N, bool, double (&R)[9]) {
#pragma unroll
        for (int m = 0; m < 9; ++m) R[m] = __ldcg(r[m % 3] + (m / 3) * N + s);
    }
    __device__ __forceinline__ void coupled(int64_t s, int64_t N, bool, const double (&J)[9], const Params& p) {
#pragma unroll
        for (int m = 0; m < 9; ++m) {
            const int64_t j = (4 + m) * N + s;
            const double x = double(__ldcg(F + j)) + double(__ldcg(Flo + j));
            const double R = __ldcg(r[m % 3] + (m / 3) * N + s);
            dlt[j] = float(rho_gradient(x, rho_rest(R, J[m], p), p));
        }
    }
};

// TBY: rows of the engine's FP32 tiles; the FP64 ring walks each as TBY / M::BY sub-tiles.
// RHO: the walk over the rho components (three items per tile, M::C = 3), else the gradient walk.
template <template <typename> class Th, class M, int TBY, bool RHO>
__global__ void __launch_bounds__(M::NTHREADS, 1)
    k_defect(InstDesc<float>* __restrict__ insts, const int* __restrict__ tile_inst, int t_begin, int t_end) {
    static_assert(TBY % M::BY == 0, "sub-tiles of the engine tile's rows");
    extern __shared__ __align__(128) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw);
    constexpr int PER = RHO ? 3 : 1;
    grid_dep_wait();
    for (int q = PER * t_begin + blockIdx.x; q < PER * t_end; q += gridDim.x) {
        const int t = q / PER, a = q - PER * t;
        const InstDesc<float>& in = insts[__ldg(tile_inst + t)];
        if (!in.active || !refresh_due(in)) continue;  // uniform across the block
        const Params p = in.p;
        const MarchGrid mg{in.tiles_nz, in.tiles_ny, in.tiles_nx, in.xc};
        int xa, xe, y0, z0;
        march_origin(mg, t - in.tile_begin, TBY, xa, xe, y0, z0, p.X);
        const float *F = in.F[in.cur ^ 1], *Flo = in.Flo[in.cur ^ 1];  // the new field
        const int64_t N = n_sites(p);
        MarchCoef<double> k;
        k.init(p);
        for (int sy = 0; sy < TBY && y0 + sy < p.Y; sy += M::BY) {
            if constexpr (RHO) {
                const int64_t c0 = (4 + a) * N;
                const float* const src[3] = {F + c0, Flo + c0, nullptr};
                rho_tile<M, double, 2, float>(sm, p, k, src, 1.0, 0.0, xa, xe, y0 + sy, z0,
                                              reinterpret_cast<double*>(in.L[a]), N, 3 * N);
            } else {
                const float* const src[3] = {F, Flo, nullptr};
                KSum es{0.0, 0.0}, bs{0.0, 0.0};
                using Epi = typename std::conditional<Th<double>::kId == SKY_THEORY_RHO, RhoDefectEpi, DefectEpi>::type;
                Epi epi{DefectEpi{in.Dlt}};
                if constexpr (HasCoupling<Epi>::value) {
                    for (int i = 0; i < 3; ++i) epi.r[i] = reinterpret_cast<const double*>(in.L[i]);
                    epi.F = F;
                    epi.Flo = Flo;
                }
                grad_tile<Th, M, double, 2, 0, Epi, float>(sm, p, k, src, 1.0, 0.0, xa, xe, y0 + sy, z0, epi, es, bs);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Energy audit of one instance's current state (F, V), in FP64: the potential
// Phi of the RK4 dynamics (sky_theories.cuh, Dynamics) and the signed kinetic
// term (1/2) h^3 sum_c s_c |V_c|^2, whose sum H the dynamics conserves.  The
// field is staged into an FP64 ring (hi + lo for a compensated field); each
// block writes its two compensated partial sums to parts[4 * block].
// ---------------------------------------------------------------------------
template <template <typename> class Th, typename S>
struct AuditOp {
    const Params& p;
    const S* V;  // null: the velocity is zero (arrested)
    int64_t N;
    KSum pot, kin;
    __device__ __forceinline__ void operator()(int64_t s, int, const double (&phi)[Th<double>::C],
                                               const double (&D)[3][Th<double>::C]) {
        ksum_add(pot, Dynamics<Th>::potential(phi, D, p));
        if (!V) return;
        double k = 0.0;
#pragma unroll
        for (int c = 0; c < Th<double>::C; ++c) {
            const double v = double(V[c * N + s]);
            k += Dynamics<Th>::kinetic_sign(c) * v * v;
        }
        ksum_add(kin, 0.5 * p.vol * k);
    }
};

template <template <typename> class Th, class M, typename S>
__global__ void __launch_bounds__(M::NTHREADS, 1)
    k_engine_audit(const InstDesc<S>* __restrict__ d, MarchGrid mg, double* __restrict__ parts) {
    constexpr int NSRC = std::is_same<S, double>::value ? 1 : 2;
    extern __shared__ __align__(128) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw);
    __shared__ KSum shk[M::NTHREADS / 32];
    const Params p = d->p;
    const int cur = d->cur;
    const S* const src[3] = {d->F[cur], NSRC == 2 ? d->Flo[cur] : nullptr, nullptr};
    const double r1[3] = {d->r1d[0], d->r1d[1], d->r1d[2]};
    AuditOp<Th, S> op{p, d->arrested ? nullptr : d->V[cur], n_sites(p), KSum{0.0, 0.0}, KSum{0.0, 0.0}};
    for (int t = blockIdx.x; t < mg.count(); t += gridDim.x) {
        int xa, xe, y0, z0;
        march_origin(mg, t, M::BY, xa, xe, y0, z0, p.X);
        dens_tile<M, S, NSRC, false>(sm, p, r1, src, xa, xe, y0, z0, op);
    }
    const KSum pe = block_ksum(op.pot, shk);
    const KSum pk = block_ksum(op.kin, shk);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        parts[4 * blockIdx.x] = pe.s;
        parts[4 * blockIdx.x + 1] = pe.c;
        parts[4 * blockIdx.x + 2] = pk.s;
        parts[4 * blockIdx.x + 3] = pk.c;
    }
}

}  // namespace sky
