// The rho field's walk: R_j^a = sum_i (S_ii rho_j^a - S_ij rho_i^a) of one isospin component a,
// whose three spatial components 4 + a, 7 + a and 10 + a march along x as in the gradient walk
// (sky_grad.cuh).
//
// The thirteen components' gradient used to be one walk: in FP64 a ring of four-row planes filled
// an SM's shared memory with 128 threads, each at 255 registers and spilling (16 % of the issue
// slots used).  R is all that the gradient takes from the rho field's derivatives, so the rho
// components run three at a time here, and the pions in a gradient walk of their own (RhoPion),
// which finishes the rho components at the site (or leaves what they still need, k_rho_finish).
// Step of the engine: FP64 630 -> 316 us at 57 x 50 x 45 sites and 1608 -> 621 at 72^3,
// defect-corrected FP32 505 -> 418 at 72^3.  What bounds the walks is latency: at 57 x 50 x 45 the
// rho walk takes 25 to 42 us a stage (one or three sources) at 16 warps per SM, where reading and
// writing its arrays once from L2 takes 4; 12 rows and one block per SM took 34 to 59.
//
// Mixed derivatives.  R_x takes d_x d_y rho_y + d_x d_z rho_z, R_y takes d_y (d_x rho_x + d_z
// rho_z) and R_z takes d_z (d_x rho_x + d_y rho_y).  Per plane the block writes u_x(rho_y) (with a
// y-halo), u_x(rho_z) (with a z-halo) and the two sums in brackets (with a y- and a z-halo) to
// shared memory; after a barrier each thread takes the outer difference, four taps each.  The
// sums' terms are masked by the axes that their taps share with the site, so that the mixed
// derivatives vanish where the reference's do.
#pragma once

#include "sky_grad.cuh"

namespace sky {

template <class M, typename T, typename S, int NSRC, bool TMA>
struct RhoPipe {
    static_assert(M::C == 3 && M::BY >= 8, "three components; the halo rows' work is spread over eight");
    using Pipe = PlanePipe<M, T, S, NSRC, TMA, GradBlock<M, T>::NT, 6, true>;
    // planes with a y-halo hold HY x BZ values, planes with a z-halo BY x HZ
    static constexpr int YP = M::HY * M::BZ, ZP = M::BY * M::HZ;
    static constexpr size_t bytes = Pipe::bytes + size_t(2) * (YP + ZP) * sizeof(T);
    static constexpr int nspare = int(size_t(2) * (YP + ZP) * sizeof(T) / (size_t(M::SLOT) * sizeof(S)));
};

// One tile of isospin component a: src are the arrays' component 4 + a (or null), whose spatial
// components are cstride apart, and out the destination of R_x^a, with components ostride apart.
// Returns false (every thread of
// the block) when a wait for a TMA copy gave up.
template <class M, typename T, int NSRC, typename S = T, bool TMA = false>
__device__ __forceinline__ bool rho_tile(T* __restrict__ sm, const Params& p, const MarchCoef<T>& k,
                                         const S* const (&src)[3], T wa, T wb, int xa, int xe, int y0, int z0,
                                         T* __restrict__ out, int64_t ostride, int64_t cstride, TmaTile* tma = nullptr) {
    using P = RhoPipe<M, T, S, NSRC, TMA>;
    using Pipe = typename P::Pipe;
    using L = Lanes<T>;
    using V = typename L::V;
    constexpr int NL = L::NL, R = 6, SLOT = M::SLOT, PLANE = M::PLANE, HZ = M::HZ, BZ = M::BZ;
    T* ring = sm;
    T* Ay = reinterpret_cast<T*>(reinterpret_cast<char*>(sm) + Pipe::bytes);  // u_x(rho_y), y-halo
    T* Wy = Ay + P::YP;                                                       // d_x rho_x + d_z rho_z, y-halo
    T* Az = Wy + P::YP;                                                       // u_x(rho_z), z-halo
    T* Wz = Az + P::ZP;                                                       // d_x rho_x + d_y rho_y, z-halo

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
    const int yofs = (ty + 2) * BZ + NL * tx, zofs = ty * HZ + NL * tx + M::ZOFF;

    Pipe pipe(sm, p, src, wa, wb, tx + GradBlock<M, T>::TZ * ty, y0, z0, tma, cstride);
    if (!pipe.prologue(q0, reinterpret_cast<S*>(Ay), P::nspare)) return false;
    if (q0 + 5 <= q1) pipe.issue(q0 + 5, 5);

    int o0 = 0, o1 = SLOT, o2 = 2 * SLOT, o3 = 3 * SLOT, o4 = 4 * SLOT, o5 = 5 * SLOT;
    int nslot = 0;
    int64_t s = (int64_t)xa * YZ + (int64_t)y * p.Zp + z;
    const V r1x = V(k.r1[0]), r1y = V(k.r1[1]), r1z = V(k.r1[2]);
    const V r2x = V(-k.r2[0]), r2y = V(-k.r2[1]), r2z = V(-k.r2[2]);  // (of negated tap sums)
    for (int x = xa; x < xe; ++x, s += YZ) {
        const int pslot = nslot == 0 ? R - 1 : nslot - 1;
        if (x > xa && pipe.meet(true)) {  // plane x - 1 is finished: its sums may be overwritten
            pipe.give_up();
            return false;
        }
        const bool px = x >= hl && x < p.X - hl, mx = px && x > hl;
        // first differences at an offset into the planes
        auto ux = [&](int o) {
            return tap_first(L::load(ring + o0 + o), L::load(ring + o1 + o), L::load(ring + o3 + o),
                             L::load(ring + o4 + o));
        };
        auto uy = [&](int o) {
            const T* f = ring + o2 + o;
            return tap_first(L::load(f - 2 * HZ), L::load(f - HZ), L::load(f + HZ), L::load(f + 2 * HZ));
        };
        auto uz = [&](int o) {
            V m2, m1, p1, p2;
            L::ztaps(ring + o2 + o, m2, m1, p1, p2);
            return tap_first(m2, m1, p1, p2);
        };
        auto wy = [&](V dx, V dz) { return L::mask(r1x * dx, mx, mx) + L::mask(r1z * dz, mz0, mz1); };
        auto wz = [&](V dx, V dy) { return L::mask(r1x * dx, mx, mx) + L::mask(r1y * dy, my, my); };
        // ---- the site: pure second derivatives, and the planes of first differences ----
        V rx, ry, rz;
        {
            const int ox = lofs, oy = lofs + PLANE, oz = lofs + 2 * PLANE;
            const T *fx = ring + o2 + ox, *fy = ring + o2 + oy, *fz = ring + o2 + oz;
            const V x0 = L::load(fx), y0v = L::load(fy), z0v = L::load(fz);
            const V dxx = ux(ox);  // u_x(rho_x)
            {
                V m2, m1, p1, p2;
                L::ztaps(fx, m2, m1, p1, p2);
                rx = L::mask(r2z * tap_second_neg(m2, m1, x0, p1, p2), pz0, pz1);
                rx += L::mask(r2y * tap_second_neg(L::load(fx - 2 * HZ), L::load(fx - HZ), x0, L::load(fx + HZ),
                                               L::load(fx + 2 * HZ)), py, py);
            }
            {
                const V m2 = L::load(ring + o0 + oy), m1 = L::load(ring + o1 + oy);
                const V p1 = L::load(ring + o3 + oy), p2 = L::load(ring + o4 + oy);
                L::store(Ay + yofs, tap_first(m2, m1, p1, p2));
                ry = L::mask(r2x * tap_second_neg(m2, m1, y0v, p1, p2), px, px);
                V a2, a1, b1, b2;
                L::ztaps(fy, a2, a1, b1, b2);
                ry += L::mask(r2z * tap_second_neg(a2, a1, y0v, b1, b2), pz0, pz1);
                L::store(Wz + zofs, wz(dxx, uy(oy)));
            }
            {
                const V m2 = L::load(ring + o0 + oz), m1 = L::load(ring + o1 + oz);
                const V p1 = L::load(ring + o3 + oz), p2 = L::load(ring + o4 + oz);
                L::store(Az + zofs, tap_first(m2, m1, p1, p2));
                rz = L::mask(r2x * tap_second_neg(m2, m1, z0v, p1, p2), px, px);
                rz += L::mask(r2y * tap_second_neg(L::load(fz - 2 * HZ), L::load(fz - HZ), z0v, L::load(fz + HZ),
                                               L::load(fz + 2 * HZ)), py, py);
                L::store(Wy + yofs, wy(dxx, uz(oz)));
            }
        }
        // the y-halo rows, one (plane, row) per thread row
        if (ty < 8) {
            const int hr = ty & 3, row = hr < 2 ? hr : M::BY + hr;
            const int o = row * HZ + NL * tx + M::ZOFF, w = row * BZ + NL * tx;
            if (ty < 4)
                L::store(Ay + w, ux(o + PLANE));
            else
                L::store(Wy + w, wy(ux(o), uz(o + 2 * PLANE)));
        }
        // the z-halo columns z0-2, z0-1, z0+32, z0+33 of the thread row's own row
        constexpr int HC = 4 / NL;
        if (tx < 2 * HC) {
            const int hc = NL * (tx % HC);
            const int c = M::ZOFF + (hc < 2 ? hc - 2 : BZ + hc - 2);
            const int o = (ty + 2) * HZ + c;
            if (tx < HC)
                L::store(Az + ty * HZ + c, ux(o + 2 * PLANE));
            else
                L::store(Wz + ty * HZ + c, wz(ux(o), uy(o + PLANE)));
        }
        // ---- plane x + 3 is in; the slot of plane x - 2 takes the next plane ----
        const bool ok = x + 3 <= q1 ? pipe.land(pslot) : true;
        if (pipe.meet(ok)) {
            pipe.give_up();
            return false;
        }
        if (x + 4 <= q1) pipe.issue(x + 4, nslot);
        if (own) {
            auto dy = [&](const T* f) {
                return tap_first(L::load(f - 2 * BZ), L::load(f - BZ), L::load(f + BZ), L::load(f + 2 * BZ));
            };
            auto dz = [&](const T* f) {
                V m2, m1, p1, p2;
                L::ztaps(f, m2, m1, p1, p2);
                return tap_first(m2, m1, p1, p2);
            };
            rx -= L::mask(V(k.mix[0]) * dy(Ay + yofs), mx && my, mx && my);
            rx -= L::mask(V(k.mix[1]) * dz(Az + zofs), mx && mz0, mx && mz1);
            ry -= L::mask(r1y * dy(Wy + yofs), my, my);
            rz -= L::mask(r1z * dz(Wz + zofs), mz0, mz1);
            const V r[3] = {rx, ry, rz};
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                T* d = out + j * ostride + s;
                __stcg(d, L::get(r[j], 0));
                if constexpr (NL > 1) {
                    if (own1) __stcg(d + 1, L::get(r[j], 1));
                }
            }
        }
        const int t0 = o0;
        o0 = o1, o1 = o2, o2 = o3, o3 = o4, o4 = o5, o5 = t0;
        nslot = nslot + 1 == R ? 0 : nslot + 1;
    }
    return true;
}

// ---------------------------------------------------------------------------
// Reference-layout FP64 gradient of the thirteen components (do_gradient_step_kernel): the rho
// walk leaves R in EG's rho components, which the pion walk replaces by the gradient.
// ---------------------------------------------------------------------------
template <class M>
__global__ void __launch_bounds__(M::NTHREADS)
    k_rho_plain(Params p, const __grid_constant__ MarchCoef<double> k, MarchGrid mg, const double* __restrict__ field,
                double* __restrict__ eg) {
    extern __shared__ __align__(128) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw);
    const int64_t N = n_sites(p);
    for (int t = blockIdx.x; t < 3 * mg.count(); t += gridDim.x) {
        int xa, xe, y0, z0;
        march_origin(mg, t / 3, M::BY, xa, xe, y0, z0, p.X);
        const int64_t c0 = (4 + t % 3) * N;
        const double* const src[3] = {field + c0, nullptr, nullptr};
        rho_tile<M, double, 1>(sm, p, k, src, 0.0, 0.0, xa, xe, y0, z0, eg + c0, 3 * N, 3 * N);
    }
}

struct RhoPlainEpi : PlainGradEpi {
    static constexpr bool kCoupled = true;
    const double* field;
    __device__ __forceinline__ void coupling(int64_t s, int64_t N, bool, double (&R)[9]) {
#pragma unroll
        for (int m = 0; m < 9; ++m) R[m] = __ldcg(eg + (4 + m) * N + s);
    }
    __device__ __forceinline__ void coupled(int64_t s, int64_t N, bool, const double (&J)[9], const Params& p) {
#pragma unroll
        for (int m = 0; m < 9; ++m) {
            const int64_t j = (4 + m) * N + s;
            const double g = rho_gradient(__ldcg(field + j), rho_rest(__ldcg(eg + j), J[m], p), p);
            eg[j] = g;
            l[j] = mdt * g;
        }
    }
};

template <class M>
__global__ void __launch_bounds__(M::NTHREADS)
    k_rho_pion_plain(Params p, const __grid_constant__ MarchCoef<double> k, MarchGrid mg,
                     const double* __restrict__ field, double* eg, double* __restrict__ l) {
    extern __shared__ __align__(128) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw);
    RhoPlainEpi epi;
    epi.eg = eg;
    epi.l = l;
    epi.mdt = -p.dt;
    epi.field = field;
    const double* const src[3] = {field, nullptr, nullptr};
    KSum es{0.0, 0.0}, bs{0.0, 0.0};
    for (int t = blockIdx.x; t < mg.count(); t += gridDim.x) {
        int xa, xe, y0, z0;
        march_origin(mg, t, M::BY, xa, xe, y0, z0, p.X);
        grad_tile<RhoPion, M, double, 1, 0>(sm, p, k, src, 0.0, 0.0, xa, xe, y0, z0, epi, es, bs);
    }
}

}  // namespace sky
