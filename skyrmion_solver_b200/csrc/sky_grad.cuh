// Gradient walk: one (y, z) tile of a lattice marched along x, for the theories with at
// most five components (and rho's pions, sky_rho.cuh).  It evaluates the energy gradient at every site of the stage
// input X = F + a V + b L and hands it to an epilogue; stage 1 also sums the FP64 energy
// and baryon densities.
//
// Haloed x-planes live in a ring of six shared-memory slots: planes x-2 .. x+2 of the
// site plane being finished, and plane x+3 on its way in.  When the input is one array
// (or the hi / lo pair of a compensated field) the planes are copied straight into the
// ring; further sources land in staging slots and are added in.
//
// Mixed derivatives.  The reference's 5x5 outer-product stencil (core/derivatives.py:121-173)
// is the first-difference sum u(f) = (f[-2] - f[2]) + 8 (f[1] - f[-1]) taken along one axis of
// the same sum along the other.  Per plane the block writes
//   G = u_x(f)  (own sites, a y-halo of two rows and a z-halo of two columns) and
//   H = u_z(f)  (own sites and a y-halo)
// of the four pion components to shared memory; after a barrier each thread takes
//   d_x d_y = u_y(G),  d_x d_z = u_z(G),  d_y d_z = u_y(H),   four taps each.
// G and H at the thread's own site are its first derivatives along x and z anyway.  The
// earlier form kept u_y and u_z of five planes in registers (16 C values a thread, 64
// registers in FP64) and read 16 taps for d_y d_z: 37 shared-memory reads per component
// against about 30 here, 57 against 41 arithmetic operations, and the freed registers let
// FP64 run 16 warps per SM where it ran 8.
//
// Point arithmetic is streamed over the components (Th::Stream) after the first
// derivatives are known, so the 24 second derivatives of the pion field are never all live.
//
// FP32 threads compute two adjacent z-sites each with packed FP32x2 instructions
// (sky_pair.cuh): every tap is one 8-byte shared-memory read and every operation of the
// stencils and the point arithmetic issues once for both sites.
#pragma once

#include "sky_march.cuh"
#include "sky_pair.cuh"

namespace sky {

// Stencil scales of a lattice: first, second and mixed derivatives are integer tap sums
//   8 (f1 - f-1) - (f2 - f-2),   16 (f1 + f-1 - 2 f0) - (f2 + f-2 - 2 f0),   u(u(f))
// times r1 = 1 / (12 h), r2 = 1 / (12 h^2), mix = 1 / (144 h h').
template <typename T>
struct MarchCoef {
    T r1[3], r2[3], mix[3];
    __host__ __device__ __forceinline__ void init(const Params& p) {
        const double h[3] = {p.hx, p.hy, p.hz};
        for (int i = 0; i < 3; ++i) {
            r1[i] = T(1.0 / (12.0 * h[i]));
            r2[i] = T(1.0 / (12.0 * h[i] * h[i]));
        }
        mix[0] = T(1.0 / (144.0 * p.hx * p.hy));
        mix[1] = T(1.0 / (144.0 * p.hx * p.hz));
        mix[2] = T(1.0 / (144.0 * p.hy * p.hz));
    }
};

// Optional hook of a gradient walk's epilogue: prefetch(s, N, lane, n, x) is called by every
// thread of a row with the row's first site on the next plane, its number of sites and that plane.
template <class E, class = void>
struct HasPrefetch : std::false_type {};
template <class E>
struct HasPrefetch<E, std::void_t<decltype(std::declval<E&>().prefetch(int64_t(0), int64_t(0), 0, 0, 0))>>
    : std::true_type {};
// load(s, N, own1): at the site, between the plane's pure derivatives and its point arithmetic
// (before the barrier in between, where there is one): operands loaded here arrive while the
// point arithmetic runs.
template <class E, class = void>
struct HasLoad : std::false_type {};
template <class E>
struct HasLoad<E, std::void_t<decltype(std::declval<E&>().load(int64_t(0), int64_t(0), true))>> : std::true_type {};

// begin_site(s, N, own1): at the site, before its plane is computed.
template <class E, class = void>
struct HasGradBegin : std::false_type {};
template <class E>
struct HasGradBegin<E, std::void_t<decltype(std::declval<E&>().begin_site(int64_t(0), int64_t(0), true))>>
    : std::true_type {};

// coupling(s, N, own1, R) and coupled(s, N, own1, J, p): what a walk over the pion components
// (RhoPion) takes from and leaves for the other fields at the site.
template <class E, class = void>
struct HasCoupling : std::false_type {};
template <class E>
struct HasCoupling<E, std::void_t<decltype(E::kCoupled)>> : std::true_type {};

__device__ __forceinline__ void prefetch_l2(const void* a) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a)); }

// Lanes of a thread: one FP64 site, or a packed pair of FP32 sites (z, z + 1).
template <typename T>
struct Lanes {
    static constexpr int NL = 1;
    using V = T;
    static __device__ __forceinline__ V load(const T* f) { return *f; }
    static __device__ __forceinline__ void store(T* f, V v) { *f = v; }
    // values at z - 1 and z + 1 (and at z - 2, z + 2), given the pointer to z
    static __device__ __forceinline__ void ztaps(const T* f, V& m2, V& m1, V& p1, V& p2) {
        m2 = f[-2], m1 = f[-1], p1 = f[1], p2 = f[2];
    }
    static __device__ __forceinline__ V mask(V v, bool m0, bool) { return m0 ? v : V(0); }
    static __device__ __forceinline__ T get(V v, int) { return v; }
    static __device__ __forceinline__ void set(V& v, int, T a) { v = a; }
};
template <>
struct Lanes<float> {
    static constexpr int NL = 2;
    using V = P2;
    static __device__ __forceinline__ V load(const float* f) { return p2_load(f); }
    static __device__ __forceinline__ void store(float* f, V v) { *reinterpret_cast<float2*>(f) = v.v; }
    static __device__ __forceinline__ void ztaps(const float* f, V& m2, V& m1, V& p1, V& p2) {
        const P2 o = p2_load(f);
        m2 = p2_load(f - 2);
        p2 = p2_load(f + 2);
        m1 = P2(m2.v.y, o.v.x);
        p1 = P2(o.v.y, p2.v.x);
    }
    static __device__ __forceinline__ V mask(V v, bool m0, bool m1) { return p2_mask(v, m0, m1); }
    static __device__ __forceinline__ float get(V v, int l) { return l ? v.v.y : v.v.x; }
    static __device__ __forceinline__ void set(V& v, int l, float a) { (l ? v.v.y : v.v.x) = a; }
};

// The stencils' integer tap sums (MarchCoef).  The second one is negated and formed from second
// differences at both distances: -(16 (f1 + f-1 - 2 f0) - (f2 + f-2 - 2 f0)).  Differences of
// neighbours are nearly exact, where 16 (f1 + f-1) - 30 f0 rounds numbers thirty times as large as the
// field: a constant field has exactly no second derivative, and the FP32 gradient's error, which the
// other form left 5 % above that of one scale per tap, is below both (root mean square of eight steps'
// velocity error of compensated Coulomb 48^3 fields, scale per tap / other form / this: 5.2e-7, 5.5e-7,
// 5.05e-7), in as many operations.
template <typename V>
__device__ __forceinline__ V tap_first(V m2, V m1, V p1, V p2) {
    return V(8.0f) * (p1 - m1) + (m2 - p2);
}
template <typename V>
__device__ __forceinline__ V tap_second_neg(V m2, V m1, V o, V p1, V p2) {
    const V a = V(-2.0f) * o + (p1 + m1), b = V(-2.0f) * o + (p2 + m2);
    return V(-16.0f) * a + b;
}

// Threads of a gradient walk's block: (32 / NL) x BY.
template <class M, typename T>
struct GradBlock {
    static constexpr int TZ = M::BZ / Lanes<T>::NL;
    static constexpr int NT = TZ * M::BY;
};

// v += a u over 16 bytes of values.
__device__ __forceinline__ void axpy16(float4& v, float a, const float4& u) {
    const float2 av = make_float2(a, a);
    const float2 lo = __ffma2_rn(av, make_float2(u.x, u.y), make_float2(v.x, v.y));
    const float2 hi = __ffma2_rn(av, make_float2(u.z, u.w), make_float2(v.z, v.w));
    v = make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void axpy16(double2& v, double a, const double2& u) {
    v.x += a * u.x;
    v.y += a * u.y;
}

// ---------------------------------------------------------------------------
// The plane pipeline of a walk: a ring of six haloed planes and its copies.
//
// S = T: the first source is copied straight into the ring.  Further sources pass through a
// staging slot each and are added in (X = F + a V + b L).  The ring has six slots, so that a
// plane travels while the whole previous one is computed.  The late ring (LATE, three sources by
// TMA) has five, and a plane travels during the point arithmetic only: for tiles of which 7 slots
// leave two blocks on an SM and 8 do not.  The density walks, whose threads keep their own
// column in registers, have four.
// S != T (float arrays, FP64 ring): every source is staged and converted; X = F + a V.
// Planes outside the lattice and points outside it in y and z read as zero.
// ---------------------------------------------------------------------------
// STRIDED: the walk's components are not consecutive (every third of the rho field's nine): the
// caller gives their stride, and TMA reads one map of 3 X planes per component (TmaTile::x0).
template <class M, typename T, typename S, int NSRC, bool TMA, int NT, int R_ = 6, bool STRIDED = false>
struct PlanePipe {
    static constexpr bool SAME = std::is_same<S, T>::value;
    static constexpr bool DIRECT = SAME && NSRC == 1;
    static constexpr int R = R_;
    static constexpr bool LATE = R == 5;
    static constexpr int FIRST = R < 5 ? R : 5;  // planes the prologue fills
    static constexpr int SLOT = M::SLOT;
    static constexpr int NSTG = SAME ? NSRC - 1 : NSRC;
    static constexpr size_t ring_bytes = size_t(R) * SLOT * sizeof(T);
    static constexpr size_t stage_bytes = size_t(NSTG) * SLOT * sizeof(S);
    static constexpr size_t bytes = ring_bytes + stage_bytes;
    static_assert(!TMA || M::WIDE, "TMA staging: wide rows");
    static_assert(!TMA || (SLOT * sizeof(S) % 128 == 0 && SLOT * sizeof(T) % 128 == 0),
                  "TMA boxes land on 128-byte boundaries");
    static_assert(!LATE || (TMA && SAME && NSRC == 3), "the late ring is the staged TMA pipeline's");
    static_assert(R >= 5 || DIRECT || !SAME, "the density walks' ring");
    static_assert(SAME || NSRC <= 2, "converted sources: a field and its low parts");

    T* ring;
    S* stage;
    const S* const (&src)[3];
    T w[3];       // weights of the sources (w[0] unused)
    TmaTile* tma;
    int tid, y0, z0, X;
    int64_t YZ;
    int ns;       // extra sources present (TMA: V may be absent, then L takes the first staging slot)
    int e0;       // the first of them
    static constexpr bool ROWS = !M::WIDE && M::C > 5 && DIRECT;
    using PO = typename std::conditional<M::WIDE, PlaneChunks<M, S, NT>,
                                         typename std::conditional<ROWS, PlaneRows<M, NT>, PlaneOffsets<M, NT>>::type>::type;
    PO po;

    __device__ __forceinline__ PlanePipe(T* sm, const Params& p, const S* const (&src_)[3], T a, T b, int tid_, int y0_,
                                         int z0_, TmaTile* tma_, int64_t cstride = 0)
        : ring(sm), stage(reinterpret_cast<S*>(reinterpret_cast<char*>(sm) + ring_bytes)), src(src_), w{T(1), a, b},
          tma(tma_), tid(tid_), y0(y0_), z0(z0_), X(p.X), YZ((int64_t)p.Y * p.Zp), ns(0), e0(1) {
        if constexpr (!TMA) po.init(p, STRIDED ? cstride : n_sites(p), y0, z0, tid);
#pragma unroll
        for (int s = 1; s < NSRC; ++s)
            if (TMA ? tma->map[s] != nullptr : src[s] != nullptr) {
                if (ns == 0) e0 = s;
                ++ns;
            }
    }
    // the x coordinate of plane q in the maps (planes outside the lattice: outside the map)
    __device__ __forceinline__ int plane(int q) const {
        if constexpr (STRIDED) return unsigned(q) < unsigned(X) ? tma->x0 + q : 3 * X;
        return q;
    }
    __device__ __forceinline__ void box(void* dst, int s, int q) {
        tma_load_plane(dst, tma->map[s], z0 - M::ZOFF, y0 - 2, plane(q), 0, tma->bar);
    }
    static constexpr uint32_t kBox = uint32_t(SLOT * sizeof(S));

    // Plane q of every source into L2.
    __device__ __forceinline__ void ahead(int q) {
        if constexpr (TMA) {
            if (q >= X) return;
            tma_prefetch_plane(tma->map[0], z0 - M::ZOFF, y0 - 2, plane(q), 0);
            if (NSRC > 1 && ns > 0) tma_prefetch_plane(tma->map[e0], z0 - M::ZOFF, y0 - 2, plane(q), 0);
            if (NSRC > 2 && ns > 1) tma_prefetch_plane(tma->map[2], z0 - M::ZOFF, y0 - 2, plane(q), 0);
        }
    }
    // Start the copies of plane q into `slot`.
    __device__ __forceinline__ void issue(int q, int slot) {
        if constexpr (TMA) {
            if (tid == 0) {
                fence_proxy_async_smem();
                mbar_arrive_expect_tx(tma->bar, uint32_t(1 + (NSRC > 1 ? ns : 0)) * kBox);
                box(SAME ? (void*)(ring + slot * SLOT) : (void*)stage, 0, q);
                S* d = SAME ? stage : stage + SLOT;
                if (NSRC > 1 && ns > 0) box(d, e0, q);
                if (NSRC > 2 && ns > 1) box(d + SLOT, 2, q);
                ahead(q + 2);
            }
        } else {
            const bool xok = q >= 0 && q < X;
            const int64_t base = (int64_t)q * YZ;
            const S* const f[3] = {src[0], nullptr, nullptr};
            const S* const g[3] = {src[1], src[2], nullptr};
            S* d0 = SAME ? reinterpret_cast<S*>(ring + slot * SLOT) : stage;
            S* d1 = SAME ? stage : stage + SLOT;
            if constexpr (ROWS) {
                plane_issue_rows<M, S, NT>(d0, po, src[0], base, xok);
            } else if constexpr (M::WIDE) {
                plane_issue_wide<M, 1, S, SLOT, NT>(d0, po, f, base, xok, tid, src[0]);
                if constexpr (NSRC > 1) plane_issue_wide<M, NSRC - 1, S, SLOT, NT>(d1, po, g, base, xok, tid, src[0]);
            } else {
                plane_issue<M, 1, S, SLOT, NT>(d0, po, f, base, xok, tid, src[0]);
                if constexpr (NSRC > 1) plane_issue<M, NSRC - 1, S, SLOT, NT>(d1, po, g, base, xok, tid, src[0]);
            }
        }
    }
    // ring[slot] += w buf, over the thread's own elements
    __device__ __forceinline__ void add(int slot, const S* buf, T wt) {
        static_assert(SAME || sizeof(T) == 8, "");
        if constexpr (SAME) {
            if constexpr (M::WIDE) {
                using V4 = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
                constexpr int NV = SLOT * int(sizeof(T)) / 16;
                static_assert(SLOT * sizeof(T) % 16 == 0, "slot of whole 16-byte vectors");
                V4* d = reinterpret_cast<V4*>(ring + slot * SLOT);
                const V4* u = reinterpret_cast<const V4*>(buf);
#pragma unroll 2
                for (int i = tid; i < NV; i += NT) {
                    V4 v = d[i];
                    axpy16(v, wt, u[i]);
                    d[i] = v;
                }
            } else {
                T* d = ring + slot * SLOT;
#pragma unroll 2
                for (int i = tid; i < SLOT; i += NT) d[i] += wt * buf[i];
            }
        }
    }
    // ring[slot] = buf0 + w1 buf1, converted (S != T): pairs of consecutive values per lane, or,
    // with cp.async, the chunks the thread copied itself
    __device__ __forceinline__ void convert(int slot) {
        if constexpr (!SAME) {
            static_assert(sizeof(S) == 4 && sizeof(T) == 8 && SLOT % 4 == 0, "FP32 sources of an FP64 ring");
            double* d = reinterpret_cast<double*>(ring + slot * SLOT);
            const float* u = reinterpret_cast<const float*>(stage);
            const bool two = NSRC > 1 && ns > 0;
            const double wt = w[1];
            if constexpr (TMA) {
                for (int i = tid; i < SLOT / 2; i += NT) {
                    const float2 a = reinterpret_cast<const float2*>(u)[i];
                    double2 v = make_double2(a.x, a.y);
                    if (two) {
                        const float2 b = reinterpret_cast<const float2*>(u + SLOT)[i];
                        v.x += wt * double(b.x);
                        v.y += wt * double(b.y);
                    }
                    reinterpret_cast<double2*>(d)[i] = v;
                }
            } else {
                constexpr int VW = M::WIDE ? 4 : 1;
                for (int i = tid; i < SLOT / VW; i += NT) {
#pragma unroll
                    for (int j = 0; j < VW; ++j) {
                        double v = double(u[i * VW + j]);
                        if (two) v += wt * double(u[SLOT + i * VW + j]);
                        d[i * VW + j] = v;
                    }
                }
            }
        }
    }
    __device__ __forceinline__ bool wait() {
        bool ok = true;
        if constexpr (TMA) {
            ok = mbar_wait_bounded(tma->bar, tma->phase & 1u);
            tma->phase ^= 1u;
        } else {
            cp_async_wait_all();
        }
        return ok;
    }
    // The copies of issue() have landed and are in the ring (for the thread's own elements).
    __device__ __forceinline__ bool land(int slot) {
        const bool ok = wait();
        if constexpr (!SAME) {
            convert(slot);
        } else if constexpr (NSRC > 1) {
            if constexpr (TMA) {
                if (ns > 0) add(slot, stage, e0 == 1 ? w[1] : w[2]);
                if (NSRC > 2 && ns > 1) add(slot, stage + SLOT, w[2]);
            } else {
                if (src[1] != nullptr) add(slot, stage, w[1]);
                if (NSRC > 2 && src[2] != nullptr) add(slot, stage + SLOT, w[2]);
            }
        }
        return ok;
    }
    // Block barrier; true when some thread's wait gave up.  Every thread first orders its own
    // shared-memory accesses before the copies that thread 0 issues after the barrier.
    __device__ __forceinline__ bool meet(bool ok) {
        if constexpr (TMA) {
            fence_proxy_async_smem();
            return __syncthreads_or(ok ? 0 : 1) != 0;
        } else {
            __syncthreads();
            return false;
        }
    }
    __device__ __forceinline__ void give_up() {
        if constexpr (TMA) {
            if (tid == 0) {
                atomicOr(tma->status, 1);
                mbar_wait_bounded(tma->bar, tma->phase & 1u);  // let late copies land before the block exits
            }
        }
    }
    // Planes q0 .. q0 + FIRST - 1 into slots 0, 1, .., complete and visible to the block.  `spare` is
    // shared memory of at least `nspare` slots that the walk does not use yet, so that several
    // staged planes travel at once.
    __device__ __forceinline__ bool prologue(int q0, S* spare, int nspare) {
        meet(true);  // the previous tile's readers are done
        bool ok = true;
        if constexpr (TMA && SAME) {
            // staged planes travel through the staging slots, a sixth ring slot and the spare ones
            constexpr int own = NSTG + (R > 5 ? 1 : 0);
            const int nb = DIRECT ? 0 : own + nspare;
            const int items = NSRC > 1 ? FIRST * ns : 0;
            auto buf = [&](int k) -> S* {
                return k < NSTG ? stage + k * SLOT
                                : k < own ? reinterpret_cast<S*>(ring + 5 * SLOT) : spare + (k - own) * SLOT;
            };
            auto which = [&](int i) { return ns == 1 ? e0 : 1 + i % 2; };
            for (int it = 0; it == 0 || it < items;) {
                const int n = min(nb, items - it);
                if (tid == 0) {
                    fence_proxy_async_smem();
                    mbar_arrive_expect_tx(tma->bar, uint32_t((it == 0 ? FIRST : 0) + n) * kBox);
                    if (it == 0)
                        for (int j = 0; j < FIRST; ++j) box(ring + j * SLOT, 0, q0 + j);
                    for (int k = 0; k < n; ++k) box(buf(k), which(it + k), q0 + (it + k) / ns);
                }
                ok = wait();
                for (int k = 0; k < n; ++k) add((it + k) / ns, buf(k), which(it + k) == 1 ? w[1] : w[2]);
                it += n > 0 ? n : 1;
                if (meet(ok)) {
                    give_up();
                    return false;
                }
            }
        } else if constexpr (DIRECT) {
            for (int j = 0; j < FIRST; ++j) issue(q0 + j, j);
            wait();
            meet(true);
        } else {
            for (int j = 0; j < FIRST; ++j) {
                issue(q0 + j, j);
                ok = land(j);
                if (meet(ok)) {
                    give_up();
                    return false;
                }
            }
        }
        return true;
    }
};

// Rows of an FP64 gradient walk's tiles (32 threads each).  The drop-in kernels, whose scales and
// couplings are kernel parameters, take 16 where they fit 128 registers (gradient of 128^3
// sites: nuclear 110 us with 16 rows, 134 with 12; omega 89 and 89), else 12 at 168 registers
// (Coulomb 147 with 12 and 230 with 16, where it spills; Berger 140).  8-row tiles with the
// register queues of the earlier form: 154, 119, 200 and 173 us.  Every engine stage spills with
// 16 (omega stage 1: 143 us against 114, stage 3: 222 against 173): 12; so does rho's pion walk,
// which also holds the nine sums of its couplings.
template <template <typename> class Th>
constexpr int grad_rows64(bool engine) {
    constexpr int id = Th<double>::kId;
    return engine || id == SKY_THEORY_COULOMB || id == SKY_THEORY_BERGER || id == SKY_THEORY_RHO ? 12 : 16;
}

// Shared memory of a gradient walk.
template <template <typename> class Th, class M, typename T, typename S, int NSRC, bool TMA>
struct GradPipe {
    static constexpr bool GH = Th<T>::kMixed;
    static constexpr int CM = 4;  // components with mixed derivatives: the pion field
    static constexpr size_t gh_bytes = GH ? size_t(CM) * (M::PLANE + M::HY * M::BZ) * sizeof(T) : 0;
    // the late ring where the full one would leave one FP32 block fewer on an SM than its stages run
    // with: two, or three of eight-row tiles (228 KB, less 1 KB and the static variables of each)
    static constexpr bool LATE = TMA && NSRC == 3 && sizeof(T) == 4 && sizeof(S) == 4 &&
                                 size_t(8) * M::SLOT * sizeof(T) + gh_bytes > (M::BY == 8 ? 76000 : 114000);
    using Pipe = PlanePipe<M, T, S, NSRC, TMA, GradBlock<M, T>::NT, LATE ? 5 : 6>;
    static constexpr size_t bytes = Pipe::bytes + gh_bytes;
    // staging slots that G and H can stand in for during the prologue
    static constexpr int nspare = int(gh_bytes / (size_t(M::SLOT) * sizeof(S)));
};

// One tile: sites x in [xa, xe), rows y0 .., columns z0 .. of lattice p.  Sources, weights and
// TMA as march_tile's (sky_march.cuh); the epilogue gets the pair (or the site) at once:
// epi(s, N, own1, phi, g) with s the first site and own1 whether the second is in the lattice.
// DENS: the baryon density of the input is summed into bsum (per site in T), and for FP64 its
// energy density into esum (DENS = 2: the baryon density only).  Returns false (every thread of the block) when a wait for a TMA
// copy gave up.
template <template <typename> class Th, class M, typename T, int NSRC, int DENS, class Epi, typename S = T,
          bool TMA = false>
__device__ __forceinline__ bool grad_tile(T* __restrict__ sm, const Params& p, const MarchCoef<T>& k,
                                          const S* const (&src)[3], T a, T b, int xa, int xe, int y0, int z0, Epi& epi,
                                          KSum& esum, KSum& bsum, TmaTile* tma = nullptr) {
    using P = GradPipe<Th, M, T, S, NSRC, TMA>;
    using Pipe = typename P::Pipe;
    using L = Lanes<T>;
    using V = typename L::V;
    constexpr int NL = L::NL;
    constexpr int C = M::C, R = Pipe::R, SLOT = M::SLOT, PLANE = M::PLANE, HZ = M::HZ;
    constexpr bool GH = P::GH;
    // two barriers per plane: between writing and reading G and H, and for the late ring
    constexpr bool LATE = Pipe::LATE, PHASED = GH || LATE;
    static_assert(Th<T>::C == C && C <= 5, "component count");
    T* ring = sm;
    T* Gs = reinterpret_cast<T*>(reinterpret_cast<char*>(sm) + Pipe::bytes);
    T* Hs = Gs + P::CM * PLANE;

    const int64_t N = n_sites(p);
    const int64_t YZ = (int64_t)p.Y * p.Zp;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int y = y0 + ty, z = z0 + NL * tx;
    const bool own = (y < p.Y) && (z < p.Z);
    const bool own1 = NL > 1 && (y < p.Y) && (z + 1 < p.Z);
    const int hl = p.halo;
    const bool py = y >= hl && y < p.Y - hl, my = py && y > hl;
    const bool pz0 = z >= hl && z < p.Z - hl, mz0 = pz0 && z > hl;
    const bool pz1 = z + 1 >= hl && z + 1 < p.Z - hl, mz1 = pz1 && z + 1 > hl;
    const int q0 = xa - 2, q1 = xe + 1;
    const int lofs = (ty + 2) * HZ + (NL * tx + M::ZOFF);
    const int hofs = (ty + 2) * M::BZ + NL * tx;

    Pipe pipe(sm, p, src, a, b, tx + GradBlock<M, T>::TZ * ty, y0, z0, tma);
    if (!pipe.prologue(q0, reinterpret_cast<S*>(Gs), P::nspare)) return false;
    if (!LATE && q0 + 5 <= q1) pipe.issue(q0 + 5, 5);

    // ring offsets of planes x-2 .. x+2 (and, with six slots, x+3)
    int o0 = 0, o1 = SLOT, o2 = 2 * SLOT, o3 = 3 * SLOT, o4 = 4 * SLOT, o5 = 5 * SLOT;
    int nslot = 0;  // slot of plane x - 2
    int64_t s = (int64_t)xa * YZ + (int64_t)y * p.Zp + z;
    // the second derivatives have the opposite sign, as the streamed point arithmetic wants them (no
    // negations to issue)
    const V r1x = V(k.r1[0]), r1y = V(k.r1[1]), r1z = V(k.r1[2]);
    const V r2x = V(k.r2[0]), r2y = V(k.r2[1]), r2z = V(k.r2[2]);
    for (int x = xa; x < xe; ++x, s += YZ) {
        const int pslot = nslot == 0 ? R - 1 : nslot - 1;  // slot of plane x + 3, or of x + 2 in the late ring
        if constexpr (PHASED) {
            // plane x - 1 is finished: G and H may be overwritten; in the late ring plane x + 2 is in
            if (x > xa) {
                const bool ok = LATE ? pipe.land(pslot) : true;
                if (pipe.meet(ok)) {
                    pipe.give_up();
                    return false;
                }
            }
        }
        if constexpr (HasGradBegin<Epi>::value) {
            if (own) epi.begin_site(s, N, own1);
        }
        if constexpr (HasPrefetch<Epi>::value) {
            // the row's operands of plane x + 1, while this plane is computed
            if (y < p.Y && x + 1 < xe) epi.prefetch(s - NL * tx + YZ, N, tx, min(M::BZ, p.Z - z0), x + 1);
        }
        const bool px = x >= hl && x < p.X - hl;
        // ---- pure derivatives; G and H ----
        V phi[C], D[3][C], Sp[3][C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int co = lofs + c * PLANE;
            const T* f = ring + o2 + co;
            const V f0 = L::load(f);
            phi[c] = f0;
            {
                const V m2 = L::load(ring + o0 + co), m1 = L::load(ring + o1 + co);
                const V p1 = L::load(ring + o3 + co), p2 = L::load(ring + o4 + co);
                const V u = tap_first(m2, m1, p1, p2);
                if constexpr (GH) {
                    if (c < P::CM) L::store(Gs + co, u);
                }
                D[0][c] = L::mask(r1x * u, px, px);
                Sp[0][c] = L::mask(r2x * tap_second_neg(m2, m1, f0, p1, p2), px, px);
            }
            {
                const V m2 = L::load(f - 2 * HZ), m1 = L::load(f - HZ), p1 = L::load(f + HZ), p2 = L::load(f + 2 * HZ);
                D[1][c] = L::mask(r1y * tap_first(m2, m1, p1, p2), py, py);
                Sp[1][c] = L::mask(r2y * tap_second_neg(m2, m1, f0, p1, p2), py, py);
            }
            {
                V m2, m1, p1, p2;
                L::ztaps(f, m2, m1, p1, p2);
                const V u = tap_first(m2, m1, p1, p2);
                if constexpr (GH) {
                    if (c < P::CM) L::store(Hs + c * M::HY * M::BZ + hofs, u);
                }
                D[2][c] = L::mask(r1z * u, pz0, pz1);
                Sp[2][c] = L::mask(r2z * tap_second_neg(m2, m1, f0, p1, p2), pz0, pz1);
            }
        }
        if constexpr (GH) {
            auto put_g = [&](int o) {
                L::store(Gs + o, tap_first(L::load(ring + o0 + o), L::load(ring + o1 + o), L::load(ring + o3 + o),
                                           L::load(ring + o4 + o)));
            };
            // the y-halo rows of G and H, one (component, row) per thread row and turn
            for (int it = ty; it < 4 * P::CM; it += M::BY) {
                const int c = it >> 2, hr = it & 3;
                const int row = hr < 2 ? hr : M::BY + hr;
                const int o = c * PLANE + row * HZ + NL * tx + M::ZOFF;
                put_g(o);
                V m2, m1, p1, p2;
                L::ztaps(ring + o2 + o, m2, m1, p1, p2);
                L::store(Hs + (c * M::HY + row) * M::BZ + NL * tx, tap_first(m2, m1, p1, p2));
            }
            // the z-halo columns of G in the thread row's own row
            constexpr int HC = 4 / NL;  // column groups: z0-2, z0-1, z0+32, z0+33
            if (tx < HC * P::CM) {
                const int c = tx / HC, hc = NL * (tx % HC);
                put_g(c * PLANE + (ty + 2) * HZ + M::ZOFF + (hc < 2 ? hc - 2 : M::BZ + hc - 2));
            }
        }
        if constexpr (DENS != 0) {
            if (own) {
                const V bd = Th<V>::baryon(phi, D, p);
                ksum_add(bsum, double(L::get(bd, 0)));
                if constexpr (NL > 1) {
                    if (own1) ksum_add(bsum, double(L::get(bd, 1)));
                }
                if constexpr (sizeof(T) == 8 && DENS == 1) ksum_add(esum, Th<double>::energy(phi, D, p));
            }
        }
        if constexpr (HasLoad<Epi>::value) {
            if (own) epi.load(s, N, own1);
        }
        auto point = [&]() {
            const bool mx = px && x > hl;
            V g[C];
            typename Th<V>::Stream st;
            st.begin(phi, D, p);
            if constexpr (HasCoupling<Epi>::value) {
                V R[9];
                epi.coupling(s, N, own1, R);
                st.couple(R, D, p);
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                V s6[6] = {Sp[0][c], Sp[1][c], Sp[2][c], V(0.0f), V(0.0f), V(0.0f)};
                if constexpr (GH) {
                    if (c < P::CM) {
                        const T* G = Gs + lofs + c * PLANE;
                        const T* H = Hs + c * M::HY * M::BZ + hofs;
                        V m2, m1, p1, p2;
                        L::ztaps(G, m2, m1, p1, p2);
                        const V sxy = tap_first(L::load(G - 2 * HZ), L::load(G - HZ), L::load(G + HZ),
                                                L::load(G + 2 * HZ));
                        const V syz = tap_first(L::load(H - 2 * M::BZ), L::load(H - M::BZ), L::load(H + M::BZ),
                                                L::load(H + 2 * M::BZ));
                        s6[3] = L::mask(V(k.mix[0]) * sxy, mx && my, mx && my);
                        s6[4] = L::mask(V(k.mix[1]) * tap_first(m2, m1, p1, p2), mx && mz0, mx && mz1);
                        s6[5] = L::mask(V(k.mix[2]) * syz, my && mz0, my && mz1);
                    }
                }
                st.add(c, s6, phi, D, g);
            }
            if constexpr (HasCoupling<Epi>::value) {
                epi.coupled(s, N, own1, st.J, p);
                // the values are read again, not held
#pragma unroll
                for (int c = 0; c < C; ++c) phi[c] = L::load(ring + o2 + lofs + c * PLANE);
            }
            st.end(phi, D, p, g);
            epi(s, N, own1, phi, g);
        };
        if constexpr (!PHASED) {
            if (own) point();
        }
        // ---- plane x + 3 is in; the slot of plane x - 2 takes the next plane ----
        const bool ok = !LATE && x + 3 <= q1 ? pipe.land(pslot) : true;
        if (pipe.meet(ok)) {
            pipe.give_up();
            return false;
        }
        constexpr int next = LATE ? 3 : 4;
        if (x + next <= q1) pipe.issue(x + next, nslot);
        if constexpr (PHASED) {
            if (own) point();
        }
        const int t0 = o0;
        o0 = o1, o1 = o2, o2 = o3, o3 = o4, o4 = LATE ? t0 : o5, o5 = t0;
        nslot = nslot + 1 == R ? 0 : nslot + 1;
    }
    return true;
}

// Density walk: the FP64 value and first derivatives of the first M::C components at every
// site of a tile, handed to op(s, x, phi, D).  Sources: an FP64 array, or an FP32 one with
// optional low parts (S = float, NSRC = 2, weight 1), converted once as they enter the FP64
// ring.  The walk is bound by shared-memory reads and their latency: a thread keeps its own
// column (x-2 .. x+1) in registers, which leaves nine reads per component and a ring of four
// planes (x, whose y and z taps are read, x+1, x+2 and the one on its way), so that several
// blocks share an SM.
template <class M, typename S, int NSRC, bool TMA, bool STRIDED = false>
using DensPipe = PlanePipe<M, double, S, NSRC, TMA, M::NTHREADS, 4, STRIDED>;

template <class M, typename S, int NSRC, bool TMA, bool STRIDED = false, class Op>
__device__ __forceinline__ bool dens_tile(double* __restrict__ sm, const Params& p, const double (&r1)[3],
                                          const S* const (&src)[3], int xa, int xe, int y0, int z0, Op& op,
                                          TmaTile* tma = nullptr, int64_t cstride = 0) {
    using Pipe = DensPipe<M, S, NSRC, TMA, STRIDED>;
    constexpr int C = M::C, SLOT = M::SLOT, PLANE = M::PLANE, HZ = M::HZ;
    const int64_t YZ = (int64_t)p.Y * p.Zp;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int y = y0 + ty, z = z0 + tx;
    const bool own = (y < p.Y) && (z < p.Z);
    const int hl = p.halo;
    const bool py = y >= hl && y < p.Y - hl, pz = z >= hl && z < p.Z - hl;
    const int q1 = xe + 1;
    const int lofs = (ty + 2) * HZ + (tx + M::ZOFF);
    Pipe pipe(sm, p, src, 1.0, 1.0, tx + M::BZ * ty, y0, z0, tma, cstride);
    if (!pipe.prologue(xa - 2, nullptr, 0)) return false;
    double qm2[C], qm1[C], qc[C], qp1[C];  // planes x-2 .. x+1 of the thread's column
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const int co = lofs + c * PLANE;
        qm2[c] = sm[co], qm1[c] = sm[SLOT + co], qc[c] = sm[2 * SLOT + co], qp1[c] = sm[3 * SLOT + co];
    }
    pipe.meet(true);  // planes xa - 2 and xa - 1 have been read
    pipe.issue(xa + 2, 0);
    if (pipe.meet(pipe.land(0))) {
        pipe.give_up();
        return false;
    }
    if (xa + 3 <= q1) pipe.issue(xa + 3, 1);
    int k = 2;  // slot of plane x
    int64_t s = (int64_t)xa * YZ + (int64_t)y * p.Zp + z;
    for (int x = xa; x < xe; ++x, s += YZ) {
        const double* P0 = sm + k * SLOT + lofs;
        const double* P2 = sm + ((k + 2) & 3) * SLOT + lofs;
        if (own) {
            const bool px = x >= hl && x < p.X - hl;
            double phi[C], D[3][C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const double* f = P0 + c * PLANE;
                const double p2 = P2[c * PLANE];
                phi[c] = qc[c];
                D[0][c] = px ? r1[0] * tap_first(qm2[c], qm1[c], qp1[c], p2) : 0.0;
                D[1][c] = py ? r1[1] * tap_first(f[-2 * HZ], f[-HZ], f[HZ], f[2 * HZ]) : 0.0;
                D[2][c] = pz ? r1[2] * tap_first(f[-2], f[-1], f[1], f[2]) : 0.0;
                qm2[c] = qm1[c], qm1[c] = qc[c], qc[c] = qp1[c], qp1[c] = p2;
            }
            op(s, x, phi, D);
        }
        const bool ok = x + 3 <= q1 ? pipe.land((k + 3) & 3) : true;
        if (pipe.meet(ok)) {
            pipe.give_up();
            return false;
        }
        if (x + 4 <= q1) pipe.issue(x + 4, k);
        k = (k + 1) & 3;
    }
    return true;
}

// ---------------------------------------------------------------------------
// Reference-layout FP64 kernels built on the walks.
// ---------------------------------------------------------------------------
// do_gradient_step_kernel: EG = projected gradient of `field`, l = -dt EG.
struct PlainGradEpi {
    double* eg;
    double* l;
    double mdt;
    template <int C>
    __device__ __forceinline__ void operator()(int64_t s, int64_t N, bool, const double (&)[C], const double (&g)[C]) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            eg[c * N + s] = g[c];
            l[c * N + s] = mdt * g[c];
        }
    }
};

template <template <typename> class Th, class M>
__global__ void __launch_bounds__(M::NTHREADS)
    k_grad_plain(Params p, const __grid_constant__ MarchCoef<double> k, MarchGrid mg, const double* __restrict__ field,
                 double* __restrict__ eg, double* __restrict__ l) {
    extern __shared__ __align__(128) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw);
    PlainGradEpi epi{eg, l, -p.dt};
    const double* const src[3] = {field, nullptr, nullptr};
    KSum es{0.0, 0.0}, bs{0.0, 0.0};
    for (int t = blockIdx.x; t < mg.count(); t += gridDim.x) {
        int xa, xe, y0, z0;
        march_origin(mg, t, M::BY, xa, xe, y0, z0, p.X);
        grad_tile<Th, M, double, 1, 0>(sm, p, k, src, 0.0, 0.0, xa, xe, y0, z0, epi, es, bs);
    }
}

// One RK4 stage of the drop-in step as one kernel (core/integrator.py:382-398): the slope
// k_s = dt (V + f_s l_{s-1}) (do_rk4_step_kernel, :50-92), the gradient step l_s at the stage
// field, and the next stage's field F + f_{s+1} k_s, all at the site whose gradient the walk has
// just formed; stage 4 also writes EG and applies do_rk4_kernel (:143-177) in place.  The stage
// fields alternate between two buffers, so every stage reads one haloed array.
// A step then moves 31 arrays of C N values, the energy's read included, where the separate kernels
// moved 49, in five launches instead of thirteen: 1.12 -> 0.70 ms for omega at 128^3.
struct StageArrays {
    double *V, *F;
    const double *l1, *l2, *l3;  // slopes of the earlier stages
    double *k, *l;               // this stage's
    double* next;                // the next stage's field (stages 1-3); EG (stage 4)
};

template <int STAGE, int C>
struct PlainStageEpi {
    static constexpr int NA = STAGE == 1 ? 1 : (STAGE == 4 ? 5 : 3);  // operand arrays read at the site
    StageArrays a;
    double dt, gmx;
    int nsky, constrain;
    // V; F; l1 | V; F; l2 | V; F; l1; l2; l3
    __device__ __forceinline__ const double* operand(int k) const {
        return k == 0 ? a.V : k == 1 ? a.F : STAGE == 3 ? a.l2 : k == 2 ? a.l1 : k == 3 ? a.l2 : a.l3;
    }
    // 128-byte lines of the row's operands into L2 (a row of 32 values spans three at most) a
    // plane ahead: the loads at the site then wait for L2 and not for DRAM (omega 128^3,
    // stage 4: 280 -> 206 us, stage 2: 135 -> 129; loading the operands into registers before
    // the point arithmetic gained nothing, 12 rows of them 229 us)
    __device__ __forceinline__ void prefetch(int64_t s0, int64_t N, int lane, int n, int) {
        for (int i = lane; i < 3 * NA * C; i += 32) {
            const int k = i / (3 * C), r = i - k * 3 * C, c = r / 3, q = r - 3 * c;
            prefetch_l2(operand(k) + c * N + s0 + min(16 * q, n - 1));
        }
    }
    __device__ __forceinline__ void operator()(int64_t s, int64_t N, bool, const double (&phi)[C],
                                               const double (&g)[C]) {
        const double mdt = -dt;
        double o[NA][C];
#pragma unroll
        for (int k = 0; k < NA; ++k)
#pragma unroll
            for (int c = 0; c < C; ++c) o[k][c] = __ldcg(operand(k) + c * N + s);
        if constexpr (STAGE < 4) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int64_t j = c * N + s;
                const double v = o[0][c];
                const double kk = STAGE == 1 ? rk4_slope(dt, v, 0.0, v) : rk4_slope(dt, v, 0.5, o[NA - 1][c]);
                a.k[j] = kk;
                a.l[j] = __dmul_rn(mdt, g[c]);
                a.next[j] = rk4_field(STAGE == 1 ? phi[c] : o[NA - 2][c], STAGE == 3 ? 1.0 : 0.5, kk);
            }
        } else {
            double fv[C], vv[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int64_t j = c * N + s;
                const double v = o[0][c], s1 = o[2][c], s2 = o[3][c], s3 = o[NA - 1][c];
                const double k1 = rk4_slope(dt, v, 0.0, v), k2 = rk4_slope(dt, v, 0.5, s1);
                const double k3 = rk4_slope(dt, v, 0.5, s2), k4 = rk4_slope(dt, v, 1.0, s3);
                const double s4 = __dmul_rn(mdt, g[c]);
                a.k[j] = k4;
                a.l[j] = s4;
                a.next[j] = g[c];
                gmx = fmax(gmx, g[c]);
                vv[c] = rk4_sum(v, s1, s2, s3, s4);
                fv[c] = rk4_sum(o[1][c], k1, k2, k3, k4);
            }
            rk4_constrain<C>(fv, vv, nsky, constrain);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                a.V[c * N + s] = vv[c];
                a.F[c * N + s] = fv[c];
            }
        }
    }
};
// counters: the completion counters of the step's two reductions, cleared by stage 1.
template <template <typename> class Th, class M, int STAGE>
__global__ void __launch_bounds__(M::NTHREADS)
    k_plain_stage(Params p, const __grid_constant__ MarchCoef<double> k, MarchGrid mg, const double* __restrict__ in,
                  StageArrays a, double* __restrict__ counter_e, double* __restrict__ scratch_m,
                  double* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw);
    __shared__ double shm[M::NTHREADS / 32];
    if (STAGE == 1 && blockIdx.x == 0 && threadIdx.x == 0 && threadIdx.y == 0) {
        *counter_e = 0.0;
        scratch_m[2 * kMaxRedBlocks + 1] = 0.0;
    }
    PlainStageEpi<STAGE, M::C> epi{a, p.dt, -1.0e300, p.nsky, p.unit_length};
    const double* const src[3] = {in, nullptr, nullptr};
    KSum es{0.0, 0.0}, bs{0.0, 0.0};
    for (int t = blockIdx.x; t < mg.count(); t += gridDim.x) {
        int xa, xe, y0, z0;
        march_origin(mg, t, M::BY, xa, xe, y0, z0, p.X);
        grad_tile<Th, M, double, 1, 0>(sm, p, k, src, 0.0, 0.0, xa, xe, y0, z0, epi, es, bs);
    }
    if constexpr (STAGE == 4) finish_max(epi.gmx, scratch_m, err, shm);
}

// Reference-layout FP64 density (drop-in for compute_energy_kernel /
// compute_skyrmion_number_kernel): per-site e h^3 or b h^3 (optional) and its
// compensated sum finished by the last block (deterministic for a given grid).
// MODE 0: energy (all components), 1: baryon (phi_0..3; M::C = 4).
template <template <typename> class Th, int MODE>
struct DensOp {
    const Params& p;
    double* dens;
    KSum sum;
    template <int C>
    __device__ __forceinline__ void operator()(int64_t s, int, const double (&phi)[C], const double (&D)[3][C]) {
        constexpr int CT = Th<double>::C;
        double ph[CT], d[3][CT];
#pragma unroll
        for (int c = 0; c < CT; ++c) {
            ph[c] = c < C ? phi[c] : 0.0;
#pragma unroll
            for (int i = 0; i < 3; ++i) d[i][c] = c < C ? D[i][c] : 0.0;
        }
        const double v = MODE == 0 ? Th<double>::energy(ph, d, p) : Th<double>::baryon(ph, d, p);
        if (dens) dens[s] = v;
        ksum_add(sum, v);
    }
};

// Rows of a density walk's tiles.  Two 8-row blocks per SM: 46 us for the nuclear energy of 128^3
// sites and 55 for omega's (16 rows, one block: 50 and 56; a ring of six planes read at every
// tap: 56 and 62).  Rho's 13 components: 8 rows, one block, 36 us at 64^3 (4 rows: 58).
constexpr int kDensRows = 8;

template <template <typename> class Th, class M, int MODE>
__global__ void __launch_bounds__(M::NTHREADS, M::C > 5 ? 1 : 2)
    k_dens_plain(Params p, const __grid_constant__ MarchCoef<double> k, MarchGrid mg, const double* __restrict__ field,
                 double* __restrict__ dens, double* __restrict__ scratch, double* __restrict__ out_dev) {
    extern __shared__ __align__(128) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw);
    __shared__ KSum shk[32];
    DensOp<Th, MODE> op{p, dens, KSum{0.0, 0.0}};
    const double* const src[3] = {field, nullptr, nullptr};
    for (int t = blockIdx.x; t < mg.count(); t += gridDim.x) {
        int xa, xe, y0, z0;
        march_origin(mg, t, M::BY, xa, xe, y0, z0, p.X);
        dens_tile<M, double, 1, false>(sm, p, k.r1, src, xa, xe, y0, z0, op);
    }
    if (scratch) finish_ksum(op.sum, scratch, out_dev, shk);
}

}  // namespace sky
