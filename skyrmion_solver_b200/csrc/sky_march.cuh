// Marching ("2.5-D" x-march): tile shapes, the copies of a haloed plane and the tiling of a lattice.
//
// A thread block owns a BY x 32 (y, z) tile of one lattice and walks along x over a chunk
// [xa, xe).  The haloed input planes of the walk's components pass through a ring of
// shared-memory slots; the next plane travels (cp.async or TMA) while the current one is computed.
// The walks are in sky_grad.cuh and sky_rho.cuh.
#pragma once

#include <type_traits>

#include "sky_kernels.cuh"
#include "sky_tma.cuh"

namespace sky {

// A row of a staged plane holds z = z0 - ZOFF .. z0 - ZOFF + HZ - 1.  Narrow rows
// (36 values: z0-2 .. z0+33) are filled element by element; wide rows (40 values:
// z0-4 .. z0+35) are filled with 16-byte copies, which needs the row pitch Zp to be a multiple
// of 16 / sizeof(T) so that every 16-byte chunk of a row starts on a 16-byte boundary
// and lies wholly inside or (as the first chunk at z0 = 0) wholly outside the lattice
// in z; a chunk crossing z = Z copies its in-lattice part and zero-fills the rest.
//
// ZP: columns staged on each side of a wide row's 32 (4, or 2 for 8-byte values, whose
// 16-byte chunks start at z0 - 2).
template <int C_, int BY_, bool WIDE_ = false, int ZP = 4>
struct MarchShape {
    static constexpr int C = C_, BY = BY_, BZ = 32;
    static constexpr bool WIDE = WIDE_;
    static constexpr int ZOFF = WIDE ? ZP : 2;
    static constexpr int HY = BY + 4, HZ = BZ + 2 * ZOFF;
    static constexpr int PLANE = HY * HZ;  // one component of one plane, with halo
    static constexpr int SLOT = C * PLANE;  // all components of one plane
    static constexpr int NTHREADS = BZ * BY;
};

// Per-tile TMA state of a walk: the kernel's mbarrier (initialised once per launch), the
// parity of the phase it completes next, the maps of the tile's sources (null: the source reads as zero) and the launch-wide error word
// that a timed-out wait sets.
struct TmaTile {
    uint64_t* bar;
    uint32_t phase;
    const TmaMap* map[3];
    int* status;
    int x0 = 0;  // first plane of the walk's components in the maps (strided components)
};

// ---------------------------------------------------------------------------
// cp.async (sm_80+ asynchronous global -> shared copies; zero-fill when the
// source size is 0, so out-of-lattice halo points read as 0 without a load).
// ---------------------------------------------------------------------------
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem, bool valid) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    const int n = valid ? BYTES : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(gmem), "n"(BYTES), "r"(n)
                 : "memory");
}
// 16-byte copy of `nbytes` (0..16) bytes, zero-filling the rest of the 16.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int nbytes) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(nbytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Per-thread element offsets of the haloed plane: element k of thread tid is
// idx = tid + k*NTHREADS of the slot, i.e. (c, yy, zz) = decompose(idx); its
// global offset within the x-plane is c*N + gy*Zp + gz (32 bits), or all ones when the
// point lies outside the lattice in y or z (or idx is past the slot).  The
// host guarantees C*N < 2^32 - 1 for marching launches.
template <class M, int NT = M::NTHREADS>
struct PlaneOffsets {
    static constexpr int NPER = (M::SLOT + NT - 1) / NT;
    static constexpr uint32_t kNone = 0xffffffffu;
    uint32_t off[NPER];
    __device__ __forceinline__ void init(const Params& p, int64_t N, int y0, int z0, int tid) {
#pragma unroll
        for (int k = 0; k < NPER; ++k) {
            const int idx = tid + k * NT;
            const int row = idx / M::HZ;
            const int zz = idx - row * M::HZ;
            const int c = row / M::HY;
            const int yy = row - c * M::HY;
            const int gy = y0 - 2 + yy, gz = z0 - M::ZOFF + zz;
            const bool ok = idx < M::SLOT && gy >= 0 && gy < p.Y && gz >= 0 && gz < p.Z;
            off[k] = ok ? static_cast<uint32_t>(c * N + (int64_t)gy * p.Zp + gz) : kNone;
        }
    }
};

// Narrow rows of many components: a thread keeps its column of the slot's rows and walks down them,
// NT / HZ rows at a time, so that no offsets sit in registers: 22 of them with 13 components and 256
// threads, where the density walk spilled.  A call for rho's energy density at 101 x 99 x 97 sites
// takes 159 us, with offsets 191 (175 before the density walk).
template <class M, int NT = M::NTHREADS>
struct PlaneRows {
    static constexpr int STEP = NT / M::HZ, ROWS = M::C * M::HY;
    static_assert(STEP >= 1 && STEP < M::HY, "a step stays within the next component");
    int64_t N;
    int col, row0, gz, gy0, Y, Zp;  // column of the slot (or -1), first row, lattice column, and row of the slot's first
    bool zok;
    __device__ __forceinline__ void init(const Params& p, int64_t N_, int y0, int z0, int tid) {
        N = N_;
        row0 = tid / M::HZ;
        col = row0 < STEP ? tid - row0 * M::HZ : -1;
        gz = z0 - M::ZOFF + col;
        zok = gz >= 0 && gz < p.Z;
        gy0 = y0 - 2;
        Y = p.Y;
        Zp = p.Zp;
    }
};
template <class M, typename T, int NT>
__device__ __forceinline__ void plane_issue_rows(T* __restrict__ slot, const PlaneRows<M, NT>& pr, const T* src,
                                                 int64_t plane_base, bool xok) {
    if (pr.col >= 0) {
        int yy = pr.row0;
        const T* g = src + plane_base + pr.gz;  // component c's plane
#pragma unroll 4
        for (int row = pr.row0; row < PlaneRows<M, NT>::ROWS; row += PlaneRows<M, NT>::STEP) {
            const int gy = pr.gy0 + yy;
            const bool ok = xok && pr.zok && gy >= 0 && gy < pr.Y;
            cp_async<sizeof(T)>(slot + row * M::HZ + pr.col, ok ? (const void*)(g + (int64_t)gy * pr.Zp) : (const void*)src,
                                ok);
            yy += PlaneRows<M, NT>::STEP;
            if (yy >= M::HY) {
                yy -= M::HY;
                g += pr.N;
            }
        }
    }
    cp_async_commit();
}

// Wide rows: per-thread 16-byte chunks of the haloed plane.  Chunk k of thread tid
// is ci = tid + k*NTHREADS; its global element offset within the x-plane and the
// number of its bytes inside the lattice (0 when outside or past the slot).
template <class M, typename T, int NT = M::NTHREADS>
struct PlaneChunks {
    static constexpr int VW = 16 / int(sizeof(T));
    static constexpr int CPR = M::HZ / VW;
    static constexpr int NCHS = M::C * M::HY * CPR;
    static constexpr int NCH = (NCHS + NT - 1) / NT;
    uint32_t off[NCH];
    int nb[NCH];
    __device__ __forceinline__ void init(const Params& p, int64_t N, int y0, int z0, int tid) {
        static_assert(M::WIDE && M::HZ % VW == 0, "16-byte chunks need the wide row layout");
#pragma unroll
        for (int k = 0; k < NCH; ++k) {
            const int ci = tid + k * NT;
            const int row = ci / CPR;
            const int cz = ci - row * CPR;
            const int c = row / M::HY;
            const int yy = row - c * M::HY;
            const int gy = y0 - 2 + yy, gz0 = z0 - M::ZOFF + cz * VW;
            const bool ok = ci < NCHS && gy >= 0 && gy < p.Y && gz0 >= 0 && gz0 < p.Z;
            off[k] = ok ? static_cast<uint32_t>(c * N + (int64_t)gy * p.Zp + gz0) : 0;
            nb[k] = ok ? int(sizeof(T)) * min(VW, p.Z - gz0) : 0;
        }
    }
};

// `any`: a readable address for copies that only zero-fill.  Source s of a plane lands at stage + s * DST (DST = M::SLOT: consecutive staging
// slots; a ring of R slots per source when the plane goes straight into the ring).
template <class M, int NSRC, typename T, int DST = M::SLOT, int NT = M::NTHREADS>
__device__ __forceinline__ void plane_issue_wide(T* __restrict__ stage, const PlaneChunks<M, T, NT>& pc,
                                                 const T* const (&src)[3], int64_t plane_base, bool xok, int tid,
                                                 const T* any) {
    using PC = PlaneChunks<M, T, NT>;
#pragma unroll
    for (int k = 0; k < PC::NCH; ++k) {
        const int ci = tid + k * NT;
        if (PC::NCHS % NT == 0 || ci < PC::NCHS) {
#pragma unroll
            for (int s = 0; s < NSRC; ++s) {
                const T* g = src[s];
                const int n = (xok && g != nullptr) ? pc.nb[k] : 0;
                cp_async16(stage + s * DST + ci * PC::VW, n ? (const void*)(g + plane_base + pc.off[k])
                                                                : (const void*)any, n);
            }
        }
    }
    cp_async_commit();
}

// Issue the cp.async copies of one x-plane (element offset plane_base) of the
// NSRC source arrays into the staging slots; a null source reads as zero.
template <class M, int NSRC, typename T, int DST = M::SLOT, int NT = M::NTHREADS>
__device__ __forceinline__ void plane_issue(T* __restrict__ stage, const PlaneOffsets<M, NT>& po,
                                            const T* const (&src)[3], int64_t plane_base, bool xok, int tid,
                                            const T* any) {
    // T here is the source (staging) type
#pragma unroll
    for (int k = 0; k < PlaneOffsets<M, NT>::NPER; ++k) {
        const int idx = tid + k * NT;
        if (M::SLOT % NT == 0 || idx < M::SLOT) {
            const bool ok = xok && po.off[k] != PlaneOffsets<M, NT>::kNone;
#pragma unroll
            for (int s = 0; s < NSRC; ++s) {
                const T* g = src[s];
                const bool v = ok && g != nullptr;
                cp_async<sizeof(T)>(stage + s * DST + idx,
                                    v ? (const void*)(g + plane_base + po.off[k]) : (const void*)any, v);
            }
        }
    }
    cp_async_commit();
}

// ---------------------------------------------------------------------------
// Tiling of one lattice into (x-chunk, 8-row y, 32-column z) tiles.
// ---------------------------------------------------------------------------
struct MarchGrid {
    int nz, ny, nx, xc;
    __host__ __device__ int count() const { return nz * ny * nx; }
};

template <class M>
__host__ __device__ inline MarchGrid march_grid(const Params& p, int xc) {
    MarchGrid g;
    g.xc = xc;
    g.nz = (p.Z + M::BZ - 1) / M::BZ;
    g.ny = (p.Y + M::BY - 1) / M::BY;
    g.nx = (p.X + xc - 1) / xc;
    return g;
}

__device__ __forceinline__ void march_origin(const MarchGrid& g, int t, int by, int& xa, int& xe, int& y0, int& z0,
                                             int X) {
    const int iz = t % g.nz;
    const int r = t / g.nz;
    const int iy = r % g.ny;
    const int ix = r / g.ny;
    z0 = iz * 32;
    y0 = iy * by;
    xa = ix * g.xc;
    xe = min(xa + g.xc, X);
}

}  // namespace sky
