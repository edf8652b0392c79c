// Diagnostic walks of a reference-layout FP64 field: the baryon moments behind the centre of mass
// and the RMS radius, and the nuclear model's inertia and shape sums.  One density walk
// (sky_grad.cuh) per kernel; a cluster of eight blocks reduces its sums through distributed
// shared memory to one partial, and the last cluster to finish reduces the partials, so that a
// full grid of blocks fits the standard reduction scratch and the host reads the sums alone.
// 128^3 sites: moments 100 -> 76 us; the 28 sums took 587 us on the 42 blocks whose partials the
// scratch held, one group of them takes 57 (Q) to 91 us (W).
#pragma once

#include <cooperative_groups.h>

#include "sky_grad.cuh"

namespace sky {

constexpr int kDiagCluster = 8;
// Clusters whose partials (two doubles for each of n sums) fit the scratch below the result and the
// completion counter at 2 kMaxRedBlocks.
constexpr int diag_clusters(int n) { return 2 * kMaxRedBlocks / (2 * n); }
constexpr bool diag_fits(int n) { return diag_clusters(n) >= 1 && 2 * n * diag_clusters(n) <= 2 * kMaxRedBlocks; }

// Reduce the block's NS sums over the grid in a fixed order.  Partial c of cluster c sits at
// scratch[2 NS c]; the results replace the partials' first NS values.
template <int NS, int NT>
__device__ __forceinline__ void finish_sums(const KSum (&v)[NS], double* __restrict__ scratch) {
    static_assert(diag_fits(NS) && 2 * kMaxRedBlocks + 1 < kScratchDoubles, "partials below the counter");
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ KSum part[NS][NT / 32];
    __shared__ KSum sums[NS];
    __shared__ bool am_last;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    // every sum's warps side by side, one barrier for all of them (block_ksum's order; a barrier pair
    // per sum made the moments of a small lattice slower than one block's worth of partials each:
    // 32^3 sites 61 us a call, 52 before the cluster reduction)
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        KSum a = v[q];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const KSum o = ksum_shfl_down(a, off);
            if ((tid & 31) + off < 32) ksum_merge(a, o);
        }
        if ((tid & 31) == 0) part[q][tid >> 5] = a;
    }
    __syncthreads();
    if (tid < NS) {
        KSum a{0.0, 0.0};
        for (int w = 0; w < NT / 32; ++w) ksum_merge(a, part[tid][w]);
        sums[tid] = a;
    }
    cluster.sync();
    const int nc = int(gridDim.x) / kDiagCluster;
    if (cluster.block_rank() == 0) {
        if (tid < NS) {
            KSum a = sums[tid];
            for (int r = 1; r < kDiagCluster; ++r) ksum_merge(a, *cluster.map_shared_rank(&sums[tid], r));
            double* p = scratch + 2 * NS * (blockIdx.x / kDiagCluster) + 2 * tid;
            __stcg(p, a.s);
            __stcg(p + 1, a.c);
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            unsigned int* counter = reinterpret_cast<unsigned int*>(scratch + 2 * kMaxRedBlocks + 1);
            am_last = atomicAdd(counter, 1u) == unsigned(nc - 1);
        }
        __syncthreads();
        if (am_last) {
            __threadfence();
            // one warp per sum: lane-strided partials, then a fixed shuffle tree
            const int lane = tid & 31;
            for (int q = tid >> 5; q < NS; q += NT / 32) {
                KSum a{0.0, 0.0};
                for (int c = lane; c < nc; c += 32)
                    ksum_merge(a, KSum{__ldcg(scratch + 2 * (NS * c + q)), __ldcg(scratch + 2 * (NS * c + q) + 1)});
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) {
                    const KSum o = ksum_shfl_down(a, off);
                    if (lane + off < 32) ksum_merge(a, o);
                }
                if (lane == 0) sums[q] = a;
            }
            __syncthreads();
            if (tid < NS) scratch[tid] = sums[tid].s + sums[tid].c;
        }
    }
    cluster.sync();  // a block's sums stay until rank 0 has read them
}

// ---------------------------------------------------------------------------
// Baryon moments (compute_center_of_mass_kernel / compute_rms_radius_kernel,
// th/nuclear_skyrme/kernels.py:678-758, and their host sums,
// th/nuclear_skyrme/observables.py:182-270): with b the baryon density of a
// site (h^3 included) and r = (h_x i, h_y j, h_z k) its grid point
// (create_grid_kernel), the nine sums of b, b r, |b|, |b| r and |b| |r|^2.
// y and z are constant along a thread's column, so only five sums run per site.
// ---------------------------------------------------------------------------
constexpr int kMoments = 9;

template <template <typename> class Th>
struct MomentOp {
    const Params& p;
    KSum b, bx, a, ax, axx;  // of the column: b, b x, |b|, |b| x, |b| x^2
    __device__ __forceinline__ void operator()(int64_t, int ix, const double (&phi)[4], const double (&D)[3][4]) {
        constexpr int CT = Th<double>::C;
        double ph[CT], d[3][CT];
#pragma unroll
        for (int c = 0; c < CT; ++c) {
            ph[c] = c < 4 ? phi[c] : 0.0;
#pragma unroll
            for (int i = 0; i < 3; ++i) d[i][c] = c < 4 ? D[i][c] : 0.0;
        }
        const double v = Th<double>::baryon(ph, d, p), w = fabs(v), x = p.hx * ix;
        ksum_add(b, v);
        ksum_add(bx, v * x);
        ksum_add(a, w);
        ksum_add(ax, w * x);
        ksum_add(axx, w * (x * x));
    }
};

template <template <typename> class Th, class M>
__global__ void __cluster_dims__(kDiagCluster, 1, 1) __launch_bounds__(M::NTHREADS, 2)
    k_moments(Params p, const __grid_constant__ MarchCoef<double> k, MarchGrid mg, const double* __restrict__ field,
              double* __restrict__ scratch) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw);
    KSum m[kMoments];
#pragma unroll
    for (int q = 0; q < kMoments; ++q) m[q] = KSum{0.0, 0.0};
    const double* const src[3] = {field, nullptr, nullptr};
    for (int t = blockIdx.x; t < mg.count(); t += gridDim.x) {
        int xa, xe, y0, z0;
        march_origin(mg, t, M::BY, xa, xe, y0, z0, p.X);
        const KSum zero{0.0, 0.0};
        MomentOp<Th> op{p, zero, zero, zero, zero, zero};
        dens_tile<M, double, 1, false>(sm, p, k.r1, src, xa, xe, y0, z0, op);
        const double y = p.hy * (y0 + int(threadIdx.y)), z = p.hz * (z0 + int(threadIdx.x));
        auto times = [](const KSum& s, double f) { return KSum{s.s * f, s.c * f}; };
        ksum_merge(m[0], op.b);
        ksum_merge(m[1], op.bx);
        ksum_merge(m[2], times(op.b, y));
        ksum_merge(m[3], times(op.b, z));
        ksum_merge(m[4], op.a);
        ksum_merge(m[5], op.ax);
        ksum_merge(m[6], times(op.a, y));
        ksum_merge(m[7], times(op.a, z));
        ksum_merge(m[8], op.axx);
        ksum_merge(m[8], times(op.a, y * y + z * z));
    }
    finish_sums<kMoments, M::NTHREADS>(m, scratch);
}

// ---------------------------------------------------------------------------
// Nuclear-model diagnostics in one FP64 pass (th/nuclear_skyrme/kernels.py:
// 484-1033 and observables.py:273-487): per site the left currents L_k and
// isorotation currents T_i, their Gram matrices LL, TT, LT, and with
// r = grid point - centre of mass (grid point = (h_x i, h_y j, h_z k)):
//   U  += 2 h^3 U0,  U0 = TT + kappa^2 (TT tr LL - LT LT^T)          (symmetric)
//   V  += 2 h^3 r x (r x A),  A = LL + kappa^2 (LL tr LL - LL LL)   (symmetric)
//   W  += 2 h^3 r x B_i,      B = LT + kappa^2 (LT tr LL - LT LL)
//   Q  += (3 r r^T - r^2) b / 2                                      (symmetric)
//   D  += h^3 (r^T S r - r^2 tr S / 3),  S the stress tensor
// (V_ij = eps_ilm eps_jnp r_l r_n A_mp and W_ij = eps_jlm r_l B_im, written as
// cross products).  28 sums in five groups; WHICH selects the groups a walk evaluates (bit 0: U,
// 1: V, 2: W, 3: Q, 4: D), since an observable needs one of them.
// ---------------------------------------------------------------------------
constexpr int kDiag = 28;  // U(6) V(6) W(9) Q(6) D(1)
constexpr int kDiagSize[5] = {6, 6, 9, 6, 1}, kDiagStart[5] = {0, 6, 12, 21, 27};
__host__ __device__ constexpr int diag_count(int which) {
    return (which & 1 ? 6 : 0) + (which & 2 ? 6 : 0) + (which & 4 ? 9 : 0) + (which & 8 ? 6 : 0) + (which & 16 ? 1 : 0);
}

template <int WHICH>
struct DiagOp {
    const Params& p;
    double com[3];
    double gy, gz;  // the column's y and z
    double acc[diag_count(WHICH)];
    // first sum of group g
    static constexpr int at(int g) { return diag_count(WHICH & ((1 << g) - 1)); }
    __device__ __forceinline__ static void cross3(const double* a, const double* b, double* o) {
        o[0] = a[1] * b[2] - a[2] * b[1];
        o[1] = a[2] * b[0] - a[0] * b[2];
        o[2] = a[0] * b[1] - a[1] * b[0];
    }
    __device__ __forceinline__ void operator()(int64_t, int ix, const double (&phi)[4], const double (&D)[3][4]) {
        const double k2 = p.c1 * p.c1, m2 = p.c0 * p.c0, vol = p.vol;
        const double sg = phi[0];
        const double pi[3] = {phi[1], phi[2], phi[3]};
        double L[3][3], T[3][3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double ds = D[k][0];
            const double dp[3] = {D[k][1], D[k][2], D[k][3]};
            double cr[3];
            cross3(pi, dp, cr);
#pragma unroll
            for (int a = 0; a < 3; ++a) L[k][a] = sg * dp[a] - pi[a] * ds + cr[a];
        }
        const double pi2 = pi[0] * pi[0] + pi[1] * pi[1] + pi[2] * pi[2];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                double e = 0.0;
#pragma unroll
                for (int b = 0; b < 3; ++b) e += double(eps3(i, a, b)) * pi[b];
                T[i][a] = pi[i] * pi[a] - (i == a ? pi2 : 0.0) + sg * e;
            }
        double LL[3][3], TT[3][3], LT[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                LL[i][j] = L[i][0] * L[j][0] + L[i][1] * L[j][1] + L[i][2] * L[j][2];
                TT[i][j] = T[i][0] * T[j][0] + T[i][1] * T[j][1] + T[i][2] * T[j][2];
                LT[i][j] = T[i][0] * L[j][0] + T[i][1] * L[j][1] + T[i][2] * L[j][2];
            }
        const double tr = LL[0][0] + LL[1][1] + LL[2][2];
        // grid point relative to the centre of mass
        const double r[3] = {p.hx * ix - com[0], gy - com[1], gz - com[2]};
        const double r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
        const int si[6] = {0, 0, 0, 1, 1, 2}, sj[6] = {0, 1, 2, 1, 2, 2};
        if constexpr ((WHICH & 1) != 0) {  // U
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const int i = si[q], j = sj[q];
            const double u = TT[i][j] + k2 * (TT[i][j] * tr - (LT[i][0] * LT[j][0] + LT[i][1] * LT[j][1] +
                                                                 LT[i][2] * LT[j][2]));
            acc[at(0) + q] += 2.0 * vol * u;
        }
        }
        if constexpr ((WHICH & 2) != 0) {  // V = r x (r x A): X[:, p] = r x A[:, p], then V[i, :] = r x X[i, :]
        double A[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                A[i][j] = LL[i][j] + k2 * (LL[i][j] * tr - (LL[i][0] * LL[j][0] + LL[i][1] * LL[j][1] +
                                                             LL[i][2] * LL[j][2]));
        double X[3][3];
#pragma unroll
        for (int pp = 0; pp < 3; ++pp) {
            const double col[3] = {A[0][pp], A[1][pp], A[2][pp]};
            double o[3];
            cross3(r, col, o);
#pragma unroll
            for (int i = 0; i < 3; ++i) X[i][pp] = o[i];
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const int i = si[q], j = sj[q];
            double o[3];
            cross3(r, X[i], o);
            acc[at(1) + q] += 2.0 * vol * o[j];
        }
        }
        if constexpr ((WHICH & 4) != 0) {  // W[i, :] = r x B[i, :]
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            double Bi[3];
#pragma unroll
            for (int m = 0; m < 3; ++m)
                Bi[m] = LT[i][m] + k2 * (LT[i][m] * tr - (LT[i][0] * LL[m][0] + LT[i][1] * LL[m][1] +
                                                           LT[i][2] * LL[m][2]));
            double o[3];
            cross3(r, Bi, o);
#pragma unroll
            for (int j = 0; j < 3; ++j) acc[at(2) + 3 * i + j] += 2.0 * vol * o[j];
        }
        }
        if constexpr ((WHICH & 8) != 0) {  // Q
        const double rho = 0.5 * Nuclear<double>::baryon(phi, D, p);
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const int i = si[q], j = sj[q];
            acc[at(3) + q] += (3.0 * r[i] * r[j] - (i == j ? r2 : 0.0)) * rho;
        }
        }
        if constexpr ((WHICH & 16) != 0) {  // D-term integrand: S = LL + kappa^2 (tr LL - LL LL) - e 1
        double quartic = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = i + 1; j < 3; ++j) quartic += LL[i][i] * LL[j][j] - LL[i][j] * LL[i][j];
        const double e = 0.5 * tr + 0.5 * k2 * quartic + m2 * (1.0 - sg);
        double rSr = 0.0, trS = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const double d2 = LL[i][0] * LL[0][j] + LL[i][1] * LL[1][j] + LL[i][2] * LL[2][j];
                const double Sij = LL[i][j] + k2 * (tr * LL[i][j] - d2) - (i == j ? e : 0.0);
                rSr += r[i] * r[j] * Sij;
                if (i == j) trS += Sij;
            }
        acc[at(4)] += (rSr - r2 * trS / 3.0) * vol;
        }
    }
};


// 128^3: U 75 us, V 69, W 91, Q 57, D 72.
template <class M, int WHICH>
__global__ void __cluster_dims__(kDiagCluster, 1, 1) __launch_bounds__(M::NTHREADS, WHICH == 31 ? 1 : 2)
    k_diag(Params p, const __grid_constant__ MarchCoef<double> k, MarchGrid mg, const double* __restrict__ field,
           double* __restrict__ scratch, double cx, double cy, double cz) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sm = reinterpret_cast<double*>(smraw);
    constexpr int NS = diag_count(WHICH);
    DiagOp<WHICH> op{p, {cx, cy, cz}, 0.0, 0.0, {}};
#pragma unroll
    for (int q = 0; q < NS; ++q) op.acc[q] = 0.0;
    const double* const src[3] = {field, nullptr, nullptr};
    for (int t = blockIdx.x; t < mg.count(); t += gridDim.x) {
        int xa, xe, y0, z0;
        march_origin(mg, t, M::BY, xa, xe, y0, z0, p.X);
        op.gy = p.hy * (y0 + int(threadIdx.y));
        op.gz = p.hz * (z0 + int(threadIdx.x));
        dens_tile<M, double, 1, false>(sm, p, k.r1, src, xa, xe, y0, z0, op);
    }
    KSum v[NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) v[q] = KSum{op.acc[q], 0.0};
    finish_sums<NS, M::NTHREADS>(v, scratch);
}

}  // namespace sky
