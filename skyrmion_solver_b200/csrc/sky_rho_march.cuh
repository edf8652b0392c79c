// The thirteen FP32 components of a small rho lattice in one marching walk (k_rho_fused): a ring of
// five planes and a staging slot per source (six planes and one slot less with a source that goes
// straight into the ring), one site per thread.  The mixed derivatives take 16 taps across the ring.
#pragma once

#include "sky_march.cuh"

namespace sky {

// Shared-memory slots of one plane: the ring and the staged sources.
constexpr int rho_march_slots(int nsrc, bool tma) {
    return nsrc == 1 ? 6 : tma ? 6 + nsrc - 1 : 5 + nsrc;
}
template <class M>
constexpr size_t rho_march_bytes(int nsrc, bool tma) {
    return size_t(rho_march_slots(nsrc, tma)) * M::SLOT * sizeof(float);
}

// Combine the thread's own staged chunks (source type S) into a ring slot of
// type T: X = F + a V + b L.
template <class M, int NSRC, typename T, typename S = T, int NT = M::NTHREADS>
__device__ __forceinline__ void plane_combine_wide(T* __restrict__ slot, const S* __restrict__ stage, T a, T b,
                                                   int tid) {
    using PC = PlaneChunks<M, S, NT>;
#pragma unroll
    for (int k = 0; k < PC::NCH; ++k) {
        const int ci = tid + k * NT;
        if (PC::NCHS % NT == 0 || ci < PC::NCHS) {
            T v[PC::VW];
#pragma unroll
            for (int e = 0; e < PC::VW; ++e) v[e] = T(stage[ci * PC::VW + e]);
            if (NSRC > 1) {
#pragma unroll
                for (int e = 0; e < PC::VW; ++e) v[e] += a * T(stage[M::SLOT + ci * PC::VW + e]);
            }
            if (NSRC > 2) {
#pragma unroll
                for (int e = 0; e < PC::VW; ++e) v[e] += b * T(stage[2 * M::SLOT + ci * PC::VW + e]);
            }
#pragma unroll
            for (int e = 0; e < PC::VW; ++e) slot[ci * PC::VW + e] = v[e];
        }
    }
}

// Raw first-difference sum c_m f[m*st], c = (1, -8, 0, 8, -1) for m = -2..2.
template <typename T>
__device__ __forceinline__ T diff5(const T* f, int st) {
    return (f[-2 * st] - f[2 * st]) + T(8) * (f[st] - f[-st]);
}

// One tile: planes xa-2 .. xe+1 of lattice p through the ring; the gradient of X = F + a V + b L
// and the epilogue epi(s, N, g) run at every in-lattice site with x in [xa, xe).  DENS adds the FP64
// energy and baryon densities of the stage input to esum / bsum.  A plane outside the lattice reads
// as zero.  Returns false (every thread of the block) when a wait for a TMA copy gave up (the error
// word is then set).
template <class M, int NSRC, bool DENS, bool TMA, class Epi>
__device__ __forceinline__ bool rho_march_tile(float* __restrict__ sm, const Params& p, const float* const (&src)[3],
                                               float a, float b, int xa, int xe, int y0, int z0, Epi& epi, KSum& esum,
                                               KSum& bsum, TmaTile* tma) {
    using T = float;
    constexpr int C = M::C;
    static_assert(M::WIDE, "the engine's rows are padded to whole 16-byte chunks");
    constexpr bool DIRECT = NSRC == 1;
    constexpr int R = rho_march_slots(NSRC, TMA) - (DIRECT ? 0 : (TMA ? NSRC - 1 : NSRC));  // ring slots
    constexpr int DST = DIRECT ? R * M::SLOT : M::SLOT;  // distance between the sources' copies
    T* ring = sm;
    T* stage = sm + R * M::SLOT;

    const int64_t N = n_sites(p);
    const int64_t YZ = (int64_t)p.Y * p.Zp;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int y = y0 + ty, z = z0 + tx;
    const bool own = (y < p.Y) && (z < p.Z);
    StencilCoef<T> k;
    k.init(p);
    PlaneChunks<M, T> po;  // 16-byte chunks of the haloed plane
    po.init(p, N, y0, z0, tx + M::BZ * ty);
    const int q0 = xa - 2, q1 = xe + 1;
    const int lofs = (ty + 2) * M::HZ + (tx + M::ZOFF);  // thread's site within a component plane
    auto issue = [&](int64_t base, bool xok, int dslot) {
        T* dst = DIRECT ? ring + dslot * M::SLOT : stage;
        plane_issue_wide<M, NSRC, T, DST>(dst, po, src, base, xok, tx + M::BZ * ty, src[0]);
    };
    // TMA: thread 0 copies plane qq of every present source (a plane outside the lattice arrives as
    // zeros); source 0 into ring slot dslot, further sources into the staging slots
    const int tid0 = threadIdx.x + M::BZ * threadIdx.y;
    auto issue_tma = [&](int qq, int dslot) {
        if (tid0 != 0) return;
        constexpr uint32_t box = uint32_t(M::SLOT * sizeof(T));
        uint32_t n = 1;
#pragma unroll
        for (int k = 1; k < NSRC; ++k) n += tma->map[k] != nullptr ? 1u : 0u;
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(tma->bar, n * box);
        const int zc = z0 - M::ZOFF, yc = y0 - 2;
        tma_load_plane(ring + dslot * M::SLOT, tma->map[0], zc, yc, qq, 0, tma->bar);
#pragma unroll
        for (int k = 1; k < NSRC; ++k)
            if (tma->map[k] != nullptr)
                tma_load_plane(stage + (k - 1) * M::SLOT, tma->map[k], zc, yc, qq, 0, tma->bar);
    };
    __syncthreads();
    if constexpr (TMA) {
        issue_tma(q0, 0);
    } else {
        issue((int64_t)q0 * YZ, q0 >= 0 && q0 < p.X, 0);
    }
    int slot = 0;  // ring slot of plane q
    for (int q = q0; q <= q1; ++q) {
        if constexpr (TMA) {
            // plane q has landed; for further sources, add a V + b L into the ring slot
            const bool ok = mbar_wait_bounded(tma->bar, tma->phase & 1u);
            tma->phase ^= 1u;
            if constexpr (!DIRECT) {
                using V4 = float4;
                constexpr int VW = 4;
                constexpr int NV = M::SLOT / VW;
                static_assert(M::SLOT % VW == 0, "slot of whole 16-byte vectors");
                V4* dstv = reinterpret_cast<V4*>(ring + slot * M::SLOT);
                const V4* s1 = reinterpret_cast<const V4*>(stage);
                const V4* s2 = s1 + NV;
                const bool h1 = tma->map[1] != nullptr;
                const bool h2 = NSRC > 2 && tma->map[2] != nullptr;
                if (h1 || h2) {
                    for (int i = tid0; i < NV; i += M::NTHREADS) {
                        V4 v = dstv[i];
                        T* e = reinterpret_cast<T*>(&v);
                        if (h1) {
                            const V4 u = s1[i];
                            const T* f = reinterpret_cast<const T*>(&u);
#pragma unroll
                            for (int j = 0; j < VW; ++j) e[j] += a * f[j];
                        }
                        if (h2) {
                            const V4 u = s2[i];
                            const T* f = reinterpret_cast<const T*>(&u);
#pragma unroll
                            for (int j = 0; j < VW; ++j) e[j] += b * f[j];
                        }
                        dstv[i] = v;
                    }
                }
            }
            // the ring slots are written by ordinary stores (the combine above) and read by
            // ordinary loads, and later overwritten by the copy engine: every thread orders
            // its own generic accesses before those async-proxy writes, and the barrier
            // then orders all threads' accesses before the next copy is issued
            fence_proxy_async_smem();
            // every thread has its plane q (and finished the centre of plane q - 1): the
            // ring slot of plane q - 5 and the staging slots are free for plane q + 1
            if (__syncthreads_or(ok ? 0 : 1)) {
                if (tid0 == 0) {
                    atomicOr(tma->status, 1);
                    // let late copies land before the block exits
                    mbar_wait_bounded(tma->bar, tma->phase & 1u);
                }
                return false;
            }
            if (q < q1) issue_tma(q + 1, slot + 1 == R ? 0 : slot + 1);
        } else if constexpr (DIRECT) {
            cp_async_wait_all();
            // (A) plane q has landed for every thread, and every thread finished the
            // previous centre: the slot of plane q - 5 (staging: the staging area) is free
            __syncthreads();
            if (q < q1) issue((int64_t)(q + 1) * YZ, q + 1 >= 0 && q + 1 < p.X, slot + 1 == R ? 0 : slot + 1);
        } else {
            cp_async_wait_all();
            __syncthreads();  // (A), as above
            plane_combine_wide<M, NSRC, T>(ring + slot * M::SLOT, stage, a, b, tx + M::BZ * ty);
            if (q < q1) issue((int64_t)(q + 1) * YZ, q + 1 >= 0 && q + 1 < p.X, 0);
            __syncthreads();  // (B) slot complete
        }
        const int x = q - 2;
        if (x >= xa && own) {
            // plane q-j sits in slot (slot + R - j) % R: x-2 = q-4, ..., x+2 = q
            const T* Pm2 = ring + ((slot + R - 4) % R) * M::SLOT + lofs;
            const T* Pm1 = ring + ((slot + R - 3) % R) * M::SLOT + lofs;
            const T* P0 = ring + ((slot + R - 2) % R) * M::SLOT + lofs;
            const T* Pp1 = ring + ((slot + R - 1) % R) * M::SLOT + lofs;
            const T* Pp2 = ring + slot * M::SLOT + lofs;
            const Mask mk = site_mask(p, x, y, z);
            const int64_t s = (int64_t)x * YZ + (int64_t)y * p.Zp + z;
            // baryon density of an FP32 stage input, from the FP32 derivatives the gradient uses
            // (its FP64 sum needs no more than FP32 per-site accuracy; only the energy, which
            // decides the arrest, is evaluated in FP64)
            T phi[C], D[3][C], Sd[6][C], g[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int co = c * M::PLANE;
                const T* f = P0 + co;
                const T f0 = f[0];
                phi[c] = f0;
                {
                    const T fm2 = Pm2[co], fm1 = Pm1[co], fp1 = Pp1[co], fp2 = Pp2[co];
                    D[0][c] = mk.px ? k.d1a[0] * (fp1 - fm1) - k.d1b[0] * (fp2 - fm2) : T(0);
                    Sd[0][c] = mk.px ? k.d2a[0] * (fp1 + fm1) - k.d2b[0] * (fp2 + fm2) - k.d2c[0] * f0 : T(0);
                }
                {
                    const T fm2 = f[-2 * M::HZ], fm1 = f[-M::HZ], fp1 = f[M::HZ], fp2 = f[2 * M::HZ];
                    D[1][c] = mk.py ? k.d1a[1] * (fp1 - fm1) - k.d1b[1] * (fp2 - fm2) : T(0);
                    Sd[1][c] = mk.py ? k.d2a[1] * (fp1 + fm1) - k.d2b[1] * (fp2 + fm2) - k.d2c[1] * f0 : T(0);
                }
                {
                    const T fm2 = f[-2], fm1 = f[-1], fp1 = f[1], fp2 = f[2];
                    D[2][c] = mk.pz ? k.d1a[2] * (fp1 - fm1) - k.d1b[2] * (fp2 - fm2) : T(0);
                    Sd[2][c] = mk.pz ? k.d2a[2] * (fp1 + fm1) - k.d2b[2] * (fp2 + fm2) - k.d2c[2] * f0 : T(0);
                }
                T sxy, sxz;
                {
                    sxy = (diff5<T>(Pm2 + co, M::HZ) - diff5<T>(Pp2 + co, M::HZ)) +
                          T(8) * (diff5<T>(Pp1 + co, M::HZ) - diff5<T>(Pm1 + co, M::HZ));
                    sxz = (diff5<T>(Pm2 + co, 1) - diff5<T>(Pp2 + co, 1)) +
                          T(8) * (diff5<T>(Pp1 + co, 1) - diff5<T>(Pm1 + co, 1));
                }
                Sd[3][c] = (mk.mx && mk.my) ? k.mix[0] * sxy : T(0);
                Sd[4][c] = (mk.mx && mk.mz) ? k.mix[1] * sxz : T(0);
                Sd[5][c] = (mk.my && mk.mz) ? k.mix[2] * mixed16<T>(f, M::HZ, 1) : T(0);
            }
            Rho<T>::gradient(phi, D, Sd, p, g);
            [[maybe_unused]] double b32 = 0.0;
            if constexpr (DENS) b32 = double(Rho<T>::baryon(phi, D, p));
            epi(s, N, g);
            if constexpr (DENS) {
                // FP64 energy and baryon densities of the stage input (stage 1: the field itself),
                // evaluated after the gradient so their registers do not overlap
                StencilCoef<double> kd;
                kd.init(p);
                double phd[C], Dd[3][C];
                // (differences of two tap values are exact in FP64)
                auto dif = [](const T* u, const T* v) { return double(u[0]) - double(v[0]); };
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int co = c * M::PLANE;
                    const T* f = P0 + co;
                    phd[c] = double(f[0]);
                    const double xd = dif(Pp1 + co, Pm1 + co), xd2 = dif(Pp2 + co, Pm2 + co);
                    const double yd = dif(f + M::HZ, f - M::HZ), yd2 = dif(f + 2 * M::HZ, f - 2 * M::HZ);
                    const double zd = dif(f + 1, f - 1), zd2 = dif(f + 2, f - 2);
                    Dd[0][c] = mk.px ? kd.d1a[0] * xd - kd.d1b[0] * xd2 : 0.0;
                    Dd[1][c] = mk.py ? kd.d1a[1] * yd - kd.d1b[1] * yd2 : 0.0;
                    Dd[2][c] = mk.pz ? kd.d1a[2] * zd - kd.d1b[2] * zd2 : 0.0;
                }
                ksum_add(esum, Rho<double>::energy(phd, Dd, p));
                ksum_add(bsum, b32);
            }
        }
        slot = (slot + 1) % R;
    }
    return true;
}

}  // namespace sky
