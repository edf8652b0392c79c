// Resident batched engine (host side): owns device memory for a set of lattice
// instances, groups them by (theory, precision), launches the fused stage
// kernels of sky_engine.cuh over every instance of a group at once and replays
// the per-step launch sequence from CUDA graphs.
#include <stdio.h>
#include <string.h>

#include <cmath>
#include <map>
#include <vector>

#include "sky_engine.cuh"
#include "sky_engine_host.h"
#include "sky_host.h"

namespace sky {

constexpr int kStatsCap = 8192;
constexpr int kGraphSteps = 8;  // steps captured per graph replay
// Steps launched kernel by kernel after a change of the instance set before they are captured: a
// server that admits or retires a request every chunk would capture every chunk.  A served request,
// launched / captured, in ms: nuclear FP64 32^3, 8 steps 1.55 / 1.85, 64 steps 5.57 / 5.80; 64^3, 64
// steps 13.7 / 13.6; defect-corrected 32^3, 64 steps 4.2 / 6.1, 64^3 9.9 / 11.4 (two patterns of
// refreshes to capture, and to destroy with the next change).  Beyond 64 steps the replays' smaller
// gaps between kernels pay for the capture.
constexpr int kDirectSteps = 64;

// A captured run of steps.  Bit k of `refresh`: its step k refreshes defect corrections (it may do so
// where none is due: the kernels look at each instance).
struct StepGraph {
    int nsteps;
    unsigned refresh;
    cudaGraphExec_t exec;
};
// An engine keeps this many patterns of refreshes; beyond them every captured step has one.
constexpr size_t kMaxGraphs = 8;

struct Engine {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr;  // stage 4 of a captured step, beside the work on the new field
    cudaEvent_t forked = nullptr, joined = nullptr;
    std::map<int, HostInst> insts;
    int next_id = 0;
    Group groups[kNumKernelSets][2];
    std::vector<StepGraph> graphs;     // of the current instance set
    int graph_pdl = -1;                // option 4 when the graphs were captured
    int direct_steps = 0;              // steps launched kernel by kernel since the instance set changed
    int64_t bytes = 0;
    int* d_status = nullptr;  // device error word the stage kernels set (bit 0: a TMA wait gave up)
};

const TheoryOps& kernel_ops(int set) {
    switch (set) {
        case SKY_THEORY_NUCLEAR: return kNuclearOps;
        case SKY_THEORY_OMEGA: return kOmegaOps;
        case SKY_THEORY_COULOMB: return kCoulombOps;
        case SKY_THEORY_RHO: return kRhoOps;
        case SKY_THEORY_BERGER: return kBergerOps;
        case kFusedRho: return kFusedRhoOps;
        default: return kLightlyBoundOps;
    }
}
static int launch_stage_group(int stage, const Group& g, const StageArgs& a, cudaStream_t st) {
    return kernel_ops(g.set).stage(g.prec, stage, g, a, st);
}
static int launch_energy(const Group& g, const StageArgs& a, cudaStream_t st) {
    return energy_walk(g.set, g.prec) ? kernel_ops(g.set).energy(g, a, st) : SKY_OK;
}
// Defect refresh of the group's defect-corrected FP32 instances (those whose refresh is due;
// the others' tiles are skipped).
static int launch_defect(const Group& g, cudaStream_t st) {
    return g.prec || !g.any_defect ? SKY_OK : kernel_ops(g.set).defect(g, st);
}
static int setup_group(const Group& g) { return kernel_ops(g.set).setup(g); }

// Row pitch of an instance's arrays: Z rounded up to four values, so that the rows of every
// lattice start on 16-byte boundaries and are staged by TMA or in 16-byte chunks.  With the
// caller's pitch an odd Z could only be copied value by value, and with two or three sources that
// took the stages longer than before they were gradient walks.  Step in us with the caller's pitch /
// padded: Coulomb FP64 63^3 208 / 149, omega FP64 49^3 102 / 83, nuclear FP32 75 x 83 x 61 169 / 115,
// rho defect-corrected 63^3 358 / 286.
static int row_pitch(int Z) { return (Z + 3) / 4 * 4; }
// Whether the caller's rows have such a pitch: the staging of those instances can be chosen.
static bool rows_aligned(int prec, int Z) { return Z % (prec ? 2 : 4) == 0; }

// Stage tiles of an instance for x-chunk request `xc` (0: chosen).
static void tile_geometry(const HostInst& h, int request, int* xc, int* nz, int* ny, int* nx) {
    const TileShapeInfo sh = kernel_ops(h.set).shape(h.prec);
    *nz = (h.p.Z + 31) / 32;
    *ny = (h.p.Y + sh.rows - 1) / sh.rows;
    const int resident = num_sms() * sh.blocks;
    if (request > 0)
        *xc = request < h.p.X ? request : h.p.X;
    else
        *xc = choose_chunk(h.p.X, *nz * *ny, resident, sh.blocks);
    *nx = (h.p.X + *xc - 1) / *xc;
}

static int launch_control(const Group& g, int ib, int ie, int mode, cudaStream_t st) {
    if (ie <= ib) return SKY_OK;
    if (g.prec)
        k_engine_control<double><<<ie - ib, 32 * kControlWarps, 0, st>>>(reinterpret_cast<InstDesc<double>*>(g.d_desc), ib, ie, mode);
    else
        k_engine_control<float><<<ie - ib, 32 * kControlWarps, 0, st>>>(reinterpret_cast<InstDesc<float>*>(g.d_desc), ib, ie, mode);
    return check_cuda(cudaGetLastError(), "launch engine control", __LINE__);
}


// ---------------------------------------------------------------------------
// conversion kernels (FP64 reference layout <-> engine storage)
// ---------------------------------------------------------------------------
// The caller's arrays have rows of Z values, the engine's of Zp.
__device__ __forceinline__ int64_t caller_index(int64_t i, int Z, int Zp) {
    if (Z == Zp) return i;
    const uint32_t row = uint32_t(i) / uint32_t(Zp), z = uint32_t(i) - row * uint32_t(Zp);
    return z < uint32_t(Z) ? int64_t(row) * Z + z : -1;
}
// n: values of the engine's array, padding included (it reads as zero; a null src too)
template <typename S>
__global__ void k_convert_in(int64_t n, int Z, int Zp, const double* __restrict__ src, S* __restrict__ dst) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = caller_index(i, Z, Zp);
        dst[i] = src && j >= 0 ? S(src[j]) : S(0);
    }
}
// An instance's field (high plus low parts of a compensated one) and velocity in FP64; null: not
// wanted.  Which halves are current, and whether the velocity counts as zero (the reference zeroes V
// on arrest), is read from the device's own state: a read-back is then one launch and one
// synchronisation where it fetched that state to the host first (38 us of the 144 that a step, its
// record and the buffers of a frame take at 32^3 sites).
template <typename S>
__global__ void k_read_state(const InstDesc<S>* __restrict__ d, int64_t n, double* __restrict__ field,
                             double* __restrict__ velocity) {
    const S *F = d->F[d->cur], *Flo = d->Flo[d->cur], *V = d->arrested ? nullptr : d->V[d->cur];
    const int Z = d->p.Z, Zp = d->p.Zp;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = caller_index(i, Z, Zp);
        if (j < 0) continue;
        if (field) field[j] = Flo ? double(F[i]) + double(Flo[i]) : double(F[i]);
        if (velocity) velocity[j] = V ? double(V[i]) : 0.0;
    }
}
__global__ void k_f32_to_f64(int64_t n, const float* __restrict__ s, double* __restrict__ d) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        d[i] = double(s[i]);
}
__global__ void k_f64_to_f32(int64_t n, const double* __restrict__ s, float* __restrict__ d) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        d[i] = float(s[i]);
}
// FP64 -> compensated FP32 pair (hi = nearest float, lo = nearest float of the remainder).  Z: the
// source's rows, Zp unless it is the caller's array.
__global__ void k_f64_to_f32c(int64_t n, int Z, int Zp, const double* __restrict__ s, float* __restrict__ hi,
                              float* __restrict__ lo) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = caller_index(i, Z, Zp);
        const double v = j >= 0 ? s[j] : 0.0;
        const float h = float(v);
        hi[i] = h;
        lo[i] = float(v - double(h));
    }
}
__global__ void k_f32c_to_f64(int64_t n, const float* __restrict__ hi, const float* __restrict__ lo,
                              double* __restrict__ d, int zero) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        d[i] = zero ? 0.0 : double(hi[i]) + double(lo[i]);
}

// ---------------------------------------------------------------------------
// descriptors
// ---------------------------------------------------------------------------
// TMA plane maps of an instance's staged arrays: box hz z-values x (rows + 4) y x 1 plane x C
// components, the haloed plane of a stage tile; and of an energy tile.
template <typename S>
static int encode_maps(const HostInst& h, InstDesc<S>& d) {
    const TileShapeInfo sh = kernel_ops(h.set).shape(h.prec);
    const void* arrs[kNumMaps] = {h.F[0], h.F[1], h.Flo[0], h.Flo[1], h.V[0], h.V[1],
                                  h.L[0], h.L[1], h.L[2], h.Dlt};
    for (int k = 0; k < kNumMaps; ++k) {
        if (!arrs[k]) continue;
        int rc = encode_plane_map(&d.tm[k], arrs[k], (int)sizeof(S), h.p.X, h.p.Y, h.p.Z, h.p.Zp, sh.components, sh.hz,
                                  sh.rows + 4);
        if (!rc && h.set == SKY_THEORY_RHO)
            // the rho components: those of one isospin component are 3 N apart, and its planes X long
            rc = encode_plane_map(&d.tmr[k], reinterpret_cast<const S*>(arrs[k]) + 4 * h.N, (int)sizeof(S), 3 * h.p.X,
                                  h.p.Y, h.p.Z, h.p.Zp, 3, sh.hz, sh.rho_rows + 4);
        if (!rc && k < kNumEnergyMaps && split_energy(h.set, h.prec))
            rc = encode_plane_map(&d.tmc[k], reinterpret_cast<const S*>(arrs[k]) + 4 * h.N, (int)sizeof(S), 3 * h.p.X,
                                  h.p.Y, h.p.Z, h.p.Zp, 3, 40, kDensRows + 4);
        if (!rc && k < kNumEnergyMaps && energy_walk(h.set, h.prec))
            rc = encode_plane_map(&d.tme[k], arrs[k], (int)sizeof(S), h.p.X, h.p.Y, h.p.Z, h.p.Zp, sh.components, 40,
                                  kDensRows + 4);
        if (rc) return rc;
    }
    return SKY_OK;
}

template <typename S>
static InstDesc<S> make_desc(const HostInst& h, int tile_begin, int e_tile_begin, int r_tile_begin) {
    InstDesc<S> d;
    memset(&d, 0, sizeof(d));
    d.p = h.p;
    d.coef.init(h.p);
    MarchCoef<double> cd;
    cd.init(h.p);
    for (int i = 0; i < 3; ++i) d.r1d[i] = cd.r1[i];
    for (int i = 0; i < 2; ++i) {
        d.F[i] = reinterpret_cast<S*>(h.F[i]);
        d.Flo[i] = reinterpret_cast<S*>(h.Flo[i]);
        d.Dlt = reinterpret_cast<S*>(h.Dlt);
        d.V[i] = reinterpret_cast<S*>(h.V[i]);
    }
    for (int i = 0; i < 3; ++i) d.L[i] = reinterpret_cast<S*>(h.L[i]);
    d.epart = h.epart;
    d.curl = h.curl;
    d.e_parts = energy_partials(h.set, h.prec, h.entiles);
    d.bpart = h.bpart;
    d.gpart = h.gpart;
    d.stats = h.stats;
    d.stats_cap = kStatsCap;
    d.tile_begin = tile_begin;
    d.ntiles = h.ntiles;
    d.gtiles = grad_partials(h.set, h.ntiles, h.rgrid.count());
    d.tiles_nz = h.tnz;
    d.tiles_ny = h.tny;
    d.tiles_nx = h.tnx;
    d.xc = h.xc;
    d.r_tile_begin = r_tile_begin;
    d.r_grid = h.rgrid;
    d.e_tile_begin = e_tile_begin;
    d.e_ntiles = h.entiles;
    d.e_nz = h.etnz;
    d.e_ny = h.etny;
    d.e_nx = h.etnx;
    d.e_xc = h.exc;
    d.active = h.active ? 1 : 0;
    d.refresh_period = h.defect_period;
    return d;
}

static void drop_graphs(Engine& e) {
    for (StepGraph& g : e.graphs) cudaGraphExecDestroy(g.exec);
    e.graphs.clear();
}

// Rebuild a group's device descriptor array and tile list.  Device-updated
// control fields (e_prev, step, arrested, cur) of existing members are kept.
template <typename S>
static int rebuild_group_t(Engine& e, Group& g) {
    int rc0 = check_cuda(cudaStreamSynchronize(e.stream), "sync", __LINE__);
    drop_graphs(e);
    e.direct_steps = 0;
    if (rc0) return rc0;
    // gather current device state of the members (they may move slots)
    std::vector<InstDesc<S>> dev_old;
    if (g.d_desc && g.desc_cap > 0) {
        dev_old.resize(g.desc_cap);
        int rc = check_cuda(cudaMemcpyAsync(dev_old.data(), g.d_desc, sizeof(InstDesc<S>) * g.desc_cap,
                                            cudaMemcpyDeviceToHost, e.stream),
                            "read descriptors", __LINE__);
        if (rc) return rc;
        if ((rc = check_cuda(cudaStreamSynchronize(e.stream), "sync", __LINE__))) return rc;
    }
    std::vector<InstDesc<S>> descs;
    std::vector<int> tile_inst, e_tile_inst, r_tile_inst;
    int tb = 0;
    g.any_defect = false;
    g.all_tma = !g.members.empty();
    for (size_t k = 0; k < g.members.size(); ++k) {
        HostInst& h = e.insts[g.members[k]];
        InstDesc<S> d = make_desc<S>(h, tb, (int)e_tile_inst.size(), (int)r_tile_inst.size());
        d.status = e.d_status;
        if (h.tma) {
            const int rc = encode_maps<S>(h, d);
            if (rc) return rc;
            d.tma = 1;
        } else {
            g.all_tma = false;
        }
        if (h.group_slot >= 0 && h.group_slot < (int)dev_old.size()) {
            const InstDesc<S>& o = dev_old[h.group_slot];
            d.e_prev = o.e_prev;
            d.step = o.step;
            d.arrested = o.arrested;
            d.cur = o.cur;
            d.refresh = (o.refresh && d.Dlt != nullptr) ? 1 : 0;  // a pending defect refresh survives
        }
        h.group_slot = (int)k;
        if (h.defect) g.any_defect = true;
        descs.push_back(d);
        for (int t = 0; t < h.ntiles; ++t) tile_inst.push_back((int)k);
        if (energy_walk(h.set, h.prec)) e_tile_inst.insert(e_tile_inst.end(), h.entiles, (int)k);
        r_tile_inst.insert(r_tile_inst.end(), h.rgrid.count(), (int)k);
        tb += h.ntiles;
    }
    g.ntiles = tb;
    g.entiles = (int)e_tile_inst.size();
    g.rtiles = (int)r_tile_inst.size();
    tile_inst.insert(tile_inst.end(), e_tile_inst.begin(), e_tile_inst.end());
    tile_inst.insert(tile_inst.end(), r_tile_inst.begin(), r_tile_inst.end());
    if ((int)descs.size() > g.desc_cap) {
        if (g.d_desc) cudaFree(g.d_desc);
        g.desc_cap = (int)descs.size() * 2 + 4;
        int rc = check_cuda(cudaMalloc(&g.d_desc, sizeof(InstDesc<S>) * g.desc_cap), "cudaMalloc(desc)", __LINE__);
        if (rc) return rc;
        cudaMemsetAsync(g.d_desc, 0, sizeof(InstDesc<S>) * g.desc_cap, e.stream);
    }
    if (!g.d_done) {
        int rc = check_cuda(cudaMalloc(&g.d_done, sizeof(int)), "cudaMalloc(done)", __LINE__);
        if (rc) return rc;
        cudaMemsetAsync(g.d_done, 0, sizeof(int), e.stream);
    }
    if ((int)tile_inst.size() > g.tile_cap) {
        if (g.d_tile_inst) cudaFree(g.d_tile_inst);
        g.tile_cap = (int)tile_inst.size() * 2 + 64;
        int rc = check_cuda(cudaMalloc(&g.d_tile_inst, sizeof(int) * g.tile_cap), "cudaMalloc(tiles)", __LINE__);
        if (rc) return rc;
    }
    if (!descs.empty()) {
        int rc = check_cuda(cudaMemcpyAsync(g.d_desc, descs.data(), sizeof(InstDesc<S>) * descs.size(),
                                            cudaMemcpyHostToDevice, e.stream),
                            "write descriptors", __LINE__);
        if (rc) return rc;
        rc = check_cuda(cudaMemcpyAsync(g.d_tile_inst, tile_inst.data(), sizeof(int) * tile_inst.size(),
                                        cudaMemcpyHostToDevice, e.stream),
                        "write tile list", __LINE__);
        if (rc) return rc;
    }
    return check_cuda(cudaStreamSynchronize(e.stream), "sync", __LINE__);
}

static int rebuild_group(Engine& e, Group& g) {
    return g.prec ? rebuild_group_t<double>(e, g) : rebuild_group_t<float>(e, g);
}

// Detach an instance from its memory (h then owns none).
static void drop_arrays(HostInst& h) {
    h.arena = h.parts = nullptr;
    memset(h.F, 0, sizeof(h.F));
    memset(h.Flo, 0, sizeof(h.Flo));
    h.Dlt = nullptr;
    memset(h.V, 0, sizeof(h.V));
    memset(h.L, 0, sizeof(h.L));
    h.curl = nullptr;
    h.epart = h.bpart = nullptr;
    h.gpart = nullptr;
    h.stats = nullptr;
}

static void free_inst(HostInst& h) {
    if (h.arena) cudaFree(h.arena);
    if (h.parts) cudaFree(h.parts);
    drop_arrays(h);
}

// Carves arrays out of one allocation, each on 256 bytes; with a null base, only their total size.
struct Carver {
    char* base;
    size_t used = 0;
    template <typename T>
    void take(T*& out, size_t bytes) {
        if (base) out = reinterpret_cast<T*>(base + used);
        used += (bytes + 255) & ~size_t(255);
    }
};

// Per-tile partials of an instance (energy, baryon number, stage-4 gradient).
static void take_partials(Carver& c, HostInst& h) {
    c.take(h.epart, sizeof(KSum) * energy_partials(h.set, h.prec, h.entiles));
    c.take(h.bpart, sizeof(KSum) * h.ntiles);
    c.take(h.gpart, sizeof(double) * 4 * grad_partials(h.set, h.ntiles, h.rgrid.count()));
}

// Whether an instance's (theory, precision) has TMA kernels: every one but FP64 rho.
static bool tma_kernels(const HostInst& h) { return !(h.prec && theory_components(h.theory) > 5); }
// Whether its staging is the caller's to choose and see.  The arrays of the others, whose rows are
// padded, follow the library's option.
static bool tma_possible(const HostInst& h) { return rows_aligned(h.prec, h.p.Z) && tma_kernels(h); }
// Whether the z-pair flag applies to an instance (TMA staging, FP32, omega).
static bool pair_possible(const HostInst& h) { return h.prec == 0 && h.theory == SKY_THEORY_OMEGA; }

static int alloc_inst(Engine& e, HostInst& h) {
    const size_t es = h.prec ? sizeof(double) : sizeof(float);
    h.set = kernel_set(h.theory, h.prec, h.sites);
    h.tma = option(2) == 1 && tma_kernels(h);
    h.pair = h.tma && tma_possible(h) && option(3) == 1 && pair_possible(h);
    const size_t fb = es * (size_t)h.C * (size_t)h.N;
    if ((int64_t)h.C * h.sites >= ((int64_t)1 << 31) || (int64_t)h.C * h.N >= (int64_t)0xffffffff)
        return invalid("lattice too large for the marching kernels");
    tile_geometry(h, h.xc_request, &h.xc, &h.tnz, &h.tny, &h.tnx);
    h.ntiles = h.tnz * h.tny * h.tnx;
    h.entiles = h.ntiles;
    if (h.set == SKY_THEORY_RHO) {
        const TileShapeInfo sh = kernel_ops(h.set).shape(h.prec);
        h.rgrid.nz = h.tnz;
        h.rgrid.ny = (h.p.Y + sh.rho_rows - 1) / sh.rho_rows;
        h.rgrid.xc = choose_chunk(h.p.X, 3 * h.rgrid.nz * h.rgrid.ny, sh.rho_blocks * num_sms());
        h.rgrid.nx = (h.p.X + h.rgrid.xc - 1) / h.rgrid.xc;
    }
    if (energy_walk(h.set, h.prec)) {
        h.etnz = h.tnz;
        h.etny = (h.p.Y + kDensRows - 1) / kDensRows;
        h.exc = choose_chunk(h.p.X, h.etnz * h.etny,
                             (h.C > 5 ? 1 : 2) * num_sms());
        h.etnx = (h.p.X + h.exc - 1) / h.exc;
        h.entiles = h.etnz * h.etny * h.etnx;
    }
    // One allocation per instance: an admission and a removal each make one driver call that maps or
    // unmaps memory where they made thirteen.  Nuclear FP64, 64^3 sites: add 2.5 -> 0.55 ms, remove
    // 2.1 -> 0.40 ms, beside 12 ms of steps in a served request; and one call in a few hundred was
    // seen to take 10 to 900 ms.
    auto carve = [&](char* base) {
        Carver c{base};
        for (void** q : {&h.F[0], &h.F[1], &h.V[0], &h.V[1], &h.L[0], &h.L[1], &h.L[2]}) c.take(*q, fb);
        if (h.comp)
            for (int i = 0; i < 2; ++i) c.take(h.Flo[i], fb);
        if (h.defect) c.take(h.Dlt, fb);
        if (split_energy(h.set, h.prec)) c.take(h.curl, sizeof(double) * 9 * (size_t)h.N);
        c.take(h.stats, sizeof(StepStats) * kStatsCap);
        take_partials(c, h);
        return c.used;
    };
    h.bytes = carve(nullptr);
    if (cudaMalloc(&h.arena, h.bytes) != cudaSuccess) {
        cudaGetLastError();
        drop_arrays(h);
        return SKY_ERR_NOMEM;
    }
    carve(reinterpret_cast<char*>(h.arena));
    if (h.comp) cudaMemsetAsync(h.Flo[0], 0, fb, e.stream), cudaMemsetAsync(h.Flo[1], 0, fb, e.stream);
    if (h.defect) cudaMemsetAsync(h.Dlt, 0, fb, e.stream);
    cudaMemsetAsync(h.gpart, 0, sizeof(double) * 4 * grad_partials(h.set, h.ntiles, h.rgrid.count()), e.stream);
    cudaMemsetAsync(h.stats, 0, sizeof(StepStats) * kStatsCap, e.stream);
    return SKY_OK;
}

static int upload(Engine& e, HostInst& h, const double* field, const double* velocity, bool on_device) {
    const int64_t n = (int64_t)h.C * h.N, nc = (int64_t)h.C * h.sites;  // values here, and of the caller's
    const int Z = h.p.Z, Zp = h.p.Zp;
    double* tmp = nullptr;
    int rc = SKY_OK;
    const double* srcs[2] = {field, velocity};
    void* dsts[2] = {h.F[0], h.V[0]};
    for (int k = 0; k < 2; ++k) {
        const double* src = srcs[k];
        if (src && !on_device) {
            if (!tmp && (rc = check_cuda(cudaMalloc(&tmp, sizeof(double) * nc), "cudaMalloc(upload)", __LINE__)))
                return rc;
            if ((rc = check_cuda(cudaMemcpyAsync(tmp, src, sizeof(double) * nc, cudaMemcpyHostToDevice, e.stream),
                                 "upload", __LINE__)))
                break;
            src = tmp;
        }
        if (h.prec)
            k_convert_in<double><<<ew_blocks(n), 256, 0, e.stream>>>(n, Z, Zp, src, reinterpret_cast<double*>(dsts[k]));
        else if (k == 0 && h.comp)
            k_f64_to_f32c<<<ew_blocks(n), 256, 0, e.stream>>>(n, Z, Zp, src, reinterpret_cast<float*>(h.F[0]),
                                                              reinterpret_cast<float*>(h.Flo[0]));
        else
            k_convert_in<float><<<ew_blocks(n), 256, 0, e.stream>>>(n, Z, Zp, src, reinterpret_cast<float*>(dsts[k]));
        if ((rc = check_cuda(cudaGetLastError(), "convert", __LINE__))) break;
        if (tmp) cudaStreamSynchronize(e.stream);
    }
    if (tmp) {
        cudaStreamSynchronize(e.stream);
        cudaFree(tmp);
    }
    return rc;
}

// Stage 1 + control for one instance (admission or precision change).
static int init_instance(Engine& e, HostInst& h, int mode) {
    Group& g = e.groups[h.set][h.prec];
    int tb = 0, eb = 0, rb = 0;
    for (int id : g.members) {
        if (id == h.id) break;
        tb += e.insts[id].ntiles;
        eb += e.insts[id].entiles;
        rb += e.insts[id].rgrid.count();
    }
    int rc = launch_energy(g, StageArgs{eb, eb + h.entiles, 0, 0, 0, 0}, e.stream);
    if (!rc) rc = launch_stage_group(1, g, StageArgs{tb, tb + h.ntiles, 0, rb, rb + h.rgrid.count(), 0}, e.stream);
    if (rc) return rc;
    rc = launch_control(g, h.group_slot, h.group_slot + 1, mode, e.stream);
    if (rc) return rc;
    return check_cuda(cudaStreamSynchronize(e.stream), "sync", __LINE__);
}

// Launch kinds of one step: stage 2, stage 3 (+ the field's update), then stage 4 (+ the
// velocity's) and, independent of it, the defect refresh (groups with defect-corrected instances
// only), the energy of FP32 walks and stage 1, all on the new field.  Groups are independent, so
// each kind is issued for every non-empty group before the next kind.
enum { kKindS2 = 0, kKindS3, kKindS4, kKindDefect, kKindEnergy, kKindS1, kNumKinds };

// serial: every kind in one stream; else the first kind after the fork may follow an event's record,
// which changes nothing for a chained launch (launch_chain).  late: 1 the groups with a late update only, 0 the others only,
// -1 all.
static int launch_kind(Engine& e, int kind, bool serial, cudaStream_t st, int late = -1) {
    for (int t = 0; t < kNumKernelSets; ++t)
        for (int pr = 0; pr < 2; ++pr) {
            Group& g = e.groups[t][pr];
            if (g.members.empty() || (late >= 0 && late != int(late_update(t, pr)))) continue;
            const int chained = serial || kind == kKindS3 || kind == kKindEnergy || kind == kKindS1;
            const StageArgs a{0, g.ntiles, 1, 0, g.rtiles, chained};
            int rc = SKY_OK;
            switch (kind) {
                case kKindS2: rc = launch_stage_group(2, g, a, st); break;
                case kKindS3: rc = launch_stage_group(3, g, a, st); break;
                case kKindS4: rc = launch_stage_group(4, g, a, st); break;
                case kKindDefect: rc = launch_defect(g, st); break;
                case kKindEnergy: rc = launch_energy(g, StageArgs{0, g.entiles, 1, 0, 0, chained}, st); break;
                default: rc = launch_stage_group(1, g, a, st); break;
            }
            if (rc) return rc;
        }
    return SKY_OK;
}

// Whether stage 4 runs on a second stream, beside the work on the new field.  It gains where blocks
// of both fit an SM or the new field's work is more than one kernel: FP32, and rho in FP64 (graph
// step in us, one stream / two: omega FP32 128^3 323 / 313, nuclear FP32 64^3 84 / 80, rho FP64 64^3
// 404 / 373).  FP64 stages and the small FP32 rho lattices' fill an SM with one block, and there the
// programmatic launches of one stream are worth more (omega FP64 64^3 104 / 109, nuclear FP64 96^3
// 259 / 268, rho FP32 56^3 196 / 204).
static bool two_streams(const Engine& e) {
    if (option(4) == 1) return false;
    for (int t = 0; t < kNumKernelSets; ++t)
        for (int pr = 0; pr < 2; ++pr)
            if (!e.groups[t][pr].members.empty() && energy_walk(t, pr)) return true;
    return false;
}

// Record one step; refresh: it refreshes the defect corrections that are due.  The refresh replaces the
// correction that stage 4 reads: it and its stage 1 come after stage 4, and they alone.
static int record_step(Engine& e, bool refresh) {
    int rc;
    const bool fork = two_streams(e), serial = !fork;
    cudaStream_t side = fork ? e.side : e.stream;
    if ((rc = launch_kind(e, kKindS2, serial, e.stream)) || (rc = launch_kind(e, kKindS3, serial, e.stream))) return rc;
    if (fork) {
        if ((rc = check_cuda(cudaEventRecord(e.forked, e.stream), "fork", __LINE__)) ||
            (rc = check_cuda(cudaStreamWaitEvent(side, e.forked, 0), "fork", __LINE__)))
            return rc;
    }
    auto join = [&]() -> int {
        if (!fork) return SKY_OK;
        const int r = check_cuda(cudaEventRecord(e.joined, side), "join", __LINE__);
        return r ? r : check_cuda(cudaStreamWaitEvent(e.stream, e.joined, 0), "join", __LINE__);
    };
    // a late update's stage 4 comes before its stage 1
    if ((rc = launch_kind(e, kKindS4, serial, side, 0)) || (rc = launch_kind(e, kKindS4, serial, e.stream, 1)) ||
        (rc = launch_kind(e, kKindEnergy, serial, e.stream)))
        return rc;
    if (refresh && ((rc = join()) || (rc = launch_kind(e, kKindDefect, false, e.stream)))) return rc;
    if ((rc = launch_kind(e, kKindS1, serial, e.stream))) return rc;
    return refresh ? SKY_OK : join();
}

// Bit k: the k-th step from now refreshes an instance's defect correction (refresh_due, whose step
// count HostInst::steps mirrors).
static unsigned refresh_pattern(const Engine& e, int nsteps) {
    unsigned m = 0;
    for (const auto& kv : e.insts) {
        const HostInst& h = kv.second;
        if (!h.active || !h.defect) continue;
        const int period = h.defect_period > 0 ? h.defect_period : kDefectRefresh;
        for (int k = 0; k < nsteps; ++k)
            if ((h.steps + k + 1) % period == 0) m |= 1u << k;
    }
    return m;
}
static void count_steps(Engine& e, int n) {
    for (auto& kv : e.insts)
        if (kv.second.active) kv.second.steps += n;
}

// Kernels of a step without a defect refresh.
static int count_launches(Engine& e) {
    int n = 0;
    for (int t = 0; t < kNumKernelSets; ++t)
        for (int pr = 0; pr < 2; ++pr)
            if (!e.groups[t][pr].members.empty())
                // stages 2, 3, 4, 1 (rho: three kernels each), [energy] (FP32 rho: two)
                n += 4 * (t == SKY_THEORY_RHO ? 3 : 1) + (energy_walk(t, pr) ? (split_energy(t, pr) ? 2 : 1) : 0);
    return n;
}

// Capture `nsteps` steps of the current instance set into *exec.
static int capture_steps(Engine& e, int nsteps, unsigned refresh, cudaGraphExec_t* exec) {
    cudaGraph_t graph;
    int rc = check_cuda(cudaStreamBeginCapture(e.stream, cudaStreamCaptureModeThreadLocal), "begin capture",
                        __LINE__);
    if (rc) return rc;
    for (int s = 0; s < nsteps && rc == SKY_OK; ++s) rc = record_step(e, (refresh >> s & 1) != 0);
    cudaError_t ce = cudaStreamEndCapture(e.stream, &graph);
    if (rc) {
        if (ce == cudaSuccess) cudaGraphDestroy(graph);
        return rc;
    }
    if ((rc = check_cuda(ce, "end capture", __LINE__))) return rc;
    rc = check_cuda(cudaGraphInstantiate(exec, graph, 0), "graph instantiate", __LINE__);
    cudaGraphDestroy(graph);
    return rc;
}

// The step graphs: kGraphSteps steps, and one step for the remainder of a call, each captured
// when a call first wants it, for every pattern of refreshes that comes up (with one period and
// instances admitted between calls of whole periods: two).  Each step depends only on device-side
// state, so replaying them is the same as launching the kernels one by one.
static int step_graph(Engine& e, int nsteps, unsigned refresh, cudaGraphExec_t* exec) {
    for (;;) {
        for (const StepGraph& g : e.graphs)
            if (g.nsteps == nsteps && g.refresh == refresh) {
                *exec = g.exec;
                return SKY_OK;
            }
        const unsigned every = (1u << nsteps) - 1;
        if (e.graphs.size() < kMaxGraphs || refresh == every) break;
        refresh = every;
    }
    int rc = SKY_OK;
    for (int t = 0; t < kNumKernelSets; ++t)
        for (int pr = 0; pr < 2; ++pr)
            if (!e.groups[t][pr].members.empty() && (rc = setup_group(e.groups[t][pr]))) return rc;
    StepGraph g{nsteps, refresh, nullptr};
    if ((rc = capture_steps(e, nsteps, refresh, &g.exec))) return rc;
    e.graphs.push_back(g);
    *exec = g.exec;
    return SKY_OK;
}

// A statistics record written while the engine's error word was set: a stage
// kernel gave up waiting for a TMA copy, so the step's results are not valid.
static int status_error(const StepStats& st) {
    if (st.status == 0) return SKY_OK;
    char msg[160];
    snprintf(msg, sizeof(msg), "engine error word 0x%x: a stage kernel gave up waiting for a TMA plane copy",
             (unsigned)st.status);
    return fail(SKY_ERR_TIMEOUT, msg);
}

static HostInst* find(Engine* e, int id) {
    auto it = e->insts.find(id);
    return it == e->insts.end() ? nullptr : &it->second;
}

static int remove_from_group(Engine& e, HostInst& h) {
    Group& g = e.groups[h.set][h.prec];
    // the remaining members still carry their old slots, from which the
    // rebuild gathers their device control state
    std::vector<int> keep;
    for (int id : g.members)
        if (id != h.id) keep.push_back(id);
    g.members = keep;
    const int rc = rebuild_group(e, g);
    h.group_slot = -1;
    return rc;
}

}  // namespace sky

using namespace sky;

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

int sky_engine_create(int device, void** out) {
    if (!out) return invalid("null output");
    Engine* e = new Engine();
    e->device = device;
    int rc = check_cuda(cudaSetDevice(device), "cudaSetDevice", __LINE__);
    if (!rc) rc = check_cuda(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking), "stream", __LINE__);
    if (!rc) rc = check_cuda(cudaStreamCreateWithFlags(&e->side, cudaStreamNonBlocking), "stream", __LINE__);
    if (!rc) rc = check_cuda(cudaEventCreateWithFlags(&e->forked, cudaEventDisableTiming), "event", __LINE__);
    if (!rc) rc = check_cuda(cudaEventCreateWithFlags(&e->joined, cudaEventDisableTiming), "event", __LINE__);
    if (!rc) rc = check_cuda(cudaMalloc(&e->d_status, sizeof(int)), "cudaMalloc(status)", __LINE__);
    if (!rc) rc = check_cuda(cudaMemset(e->d_status, 0, sizeof(int)), "memset(status)", __LINE__);
    if (rc) {
        if (e->d_status) cudaFree(e->d_status);
        if (e->joined) cudaEventDestroy(e->joined);
        if (e->forked) cudaEventDestroy(e->forked);
        if (e->side) cudaStreamDestroy(e->side);
        if (e->stream) cudaStreamDestroy(e->stream);
        delete e;
        return rc;
    }
    for (int t = 0; t < kNumKernelSets; ++t)
        for (int p = 0; p < 2; ++p) {
            e->groups[t][p].set = t;
            e->groups[t][p].prec = p;
        }
    *out = e;
    return SKY_OK;
}

int sky_engine_destroy(void* handle) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return SKY_OK;
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    drop_graphs(*e);
    for (auto& kv : e->insts) free_inst(kv.second);
    for (int t = 0; t < kNumKernelSets; ++t)
        for (int p = 0; p < 2; ++p) {
            if (e->groups[t][p].d_desc) cudaFree(e->groups[t][p].d_desc);
            if (e->groups[t][p].d_tile_inst) cudaFree(e->groups[t][p].d_tile_inst);
            if (e->groups[t][p].d_done) cudaFree(e->groups[t][p].d_done);
        }
    if (e->d_status) cudaFree(e->d_status);
    cudaEventDestroy(e->joined);
    cudaEventDestroy(e->forked);
    cudaStreamDestroy(e->side);
    cudaStreamDestroy(e->stream);
    delete e;
    return SKY_OK;
}

int sky_engine_add(void* handle, int theory, const int32_t* p_i, int32_t n_pi, const double* p_f, int32_t n_pf,
                   int precision, const double* field, const double* velocity, int on_device, int* id_out) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e || !id_out || !field) return invalid("null argument");
    if (precision < 0 || precision > 3)
        return invalid("precision must be 0 (FP32), 1 (FP64), 2 (FP32 with a compensated field) or 3 "
                       "(compensated and defect-corrected FP32)");
    cudaSetDevice(e->device);
    HostInst h;
    int rc = pack_params(theory, p_i, n_pi, p_f, n_pf, &h.p);
    if (rc) return rc;
    h.id = e->next_id++;
    h.theory = theory;
    h.prec = precision == 1 ? 1 : 0;
    h.comp = precision >= 2 ? 1 : 0;
    h.defect = precision == 3 ? 1 : 0;
    h.sites = n_sites(h.p);
    h.p.Zp = row_pitch(h.p.Z);
    h.N = n_sites(h.p);
    h.C = h.p.C;
    if ((rc = alloc_inst(*e, h))) return rc;
    if ((rc = upload(*e, h, field, velocity, on_device != 0))) {
        free_inst(h);
        return rc;
    }
    e->insts[h.id] = h;
    Group& g = e->groups[h.set][h.prec];
    g.members.push_back(h.id);
    if ((rc = rebuild_group(*e, g)) || (rc = init_instance(*e, e->insts[h.id], 1))) {
        g.members.pop_back();
        free_inst(e->insts[h.id]);
        e->insts.erase(h.id);
        rebuild_group(*e, g);
        return rc;
    }
    e->bytes += (int64_t)h.bytes;
    *id_out = h.id;
    return SKY_OK;
}

int sky_engine_remove(void* handle, int id) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    HostInst* h = find(e, id);
    if (!h) return invalid("unknown instance id");
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    int rc = remove_from_group(*e, *h);
    e->bytes -= (int64_t)h->bytes;
    free_inst(*h);
    e->insts.erase(id);
    return rc;
}

int sky_engine_set_precision(void* handle, int id, int precision) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    HostInst* hp = find(e, id);
    if (!hp) return invalid("unknown instance id");
    if (precision < 0 || precision > 3) return invalid("precision must be 0, 1, 2 or 3");
    const int defect_new = precision == 3 ? 1 : 0;
    if ((hp->comp ? 2 + hp->defect : hp->prec) == precision) return SKY_OK;
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    HostInst& h = *hp;
    // read the control state of the instance
    int cur = 0, arrested = 0, step = 0;
    double e_prev = 0.0;
    {
        Group& g = e->groups[h.set][h.prec];
        if (h.prec) {
            InstDesc<double> d;
            cudaMemcpy(&d, reinterpret_cast<InstDesc<double>*>(g.d_desc) + h.group_slot, sizeof(d),
                       cudaMemcpyDeviceToHost);
            cur = d.cur, arrested = d.arrested, step = d.step, e_prev = d.e_prev;
        } else {
            InstDesc<float> d;
            cudaMemcpy(&d, reinterpret_cast<InstDesc<float>*>(g.d_desc) + h.group_slot, sizeof(d),
                       cudaMemcpyDeviceToHost);
            cur = d.cur, arrested = d.arrested, step = d.step, e_prev = d.e_prev;
        }
    }
    HostInst nh = h;
    nh.prec = precision == 1 ? 1 : 0;
    nh.comp = precision >= 2 ? 1 : 0;
    nh.defect = defect_new;
    nh.group_slot = -1;
    drop_arrays(nh);
    int rc = alloc_inst(*e, nh);
    if (rc) return rc;
    const int64_t n = (int64_t)h.C * h.N;
    const void* srcs[2] = {h.F[cur], h.V[cur]};
    void* dsts[2] = {nh.F[0], nh.V[0]};
    const size_t fb = (h.prec ? sizeof(double) : sizeof(float)) * (size_t)n;
    for (int k = 0; k < 2; ++k) {
        const bool fieldk = k == 0;
        if (nh.prec == h.prec) {  // FP32 <-> compensated FP32: the high part carries over
            cudaMemcpyAsync(dsts[k], srcs[k], fb, cudaMemcpyDeviceToDevice, e->stream);
            if (fieldk && h.comp && nh.comp)
                cudaMemcpyAsync(nh.Flo[0], h.Flo[cur], fb, cudaMemcpyDeviceToDevice, e->stream);
        } else if (nh.prec) {     // FP32 (+ low part) -> FP64
            if (fieldk && h.comp)
                k_f32c_to_f64<<<ew_blocks(n), 256, 0, e->stream>>>(n, (const float*)srcs[k], (const float*)h.Flo[cur],
                                                                   (double*)dsts[k], 0);
            else
                k_f32_to_f64<<<ew_blocks(n), 256, 0, e->stream>>>(n, (const float*)srcs[k], (double*)dsts[k]);
        } else {                  // FP64 -> FP32 (+ low part)
            if (fieldk && nh.comp)
                k_f64_to_f32c<<<ew_blocks(n), 256, 0, e->stream>>>(n, h.p.Zp, h.p.Zp, (const double*)srcs[k], (float*)dsts[k],
                                                                   (float*)nh.Flo[0]);
            else
                k_f64_to_f32<<<ew_blocks(n), 256, 0, e->stream>>>(n, (const double*)srcs[k], (float*)dsts[k]);
        }
    }
    // carry the stats history
    cudaMemcpyAsync(nh.stats, h.stats, sizeof(StepStats) * kStatsCap, cudaMemcpyDeviceToDevice, e->stream);
    if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "convert", __LINE__))) {
        free_inst(nh);
        return rc;
    }
    // leave the old group
    if ((rc = remove_from_group(*e, h))) {
        free_inst(nh);
        return rc;
    }
    free_inst(h);
    e->bytes += (int64_t)nh.bytes - (int64_t)h.bytes;
    h = nh;
    Group& g2 = e->groups[h.set][h.prec];
    g2.members.push_back(h.id);
    if ((rc = rebuild_group(*e, g2))) return rc;
    // restore the control state, then recompute l1 / energy of the converted field
    if (h.prec) {
        InstDesc<double>* dd = reinterpret_cast<InstDesc<double>*>(g2.d_desc) + h.group_slot;
        cudaMemcpyAsync(&dd->step, &step, sizeof(int), cudaMemcpyHostToDevice, e->stream);
        cudaMemcpyAsync(&dd->arrested, &arrested, sizeof(int), cudaMemcpyHostToDevice, e->stream);
        cudaMemcpyAsync(&dd->e_prev, &e_prev, sizeof(double), cudaMemcpyHostToDevice, e->stream);
    } else {
        InstDesc<float>* dd = reinterpret_cast<InstDesc<float>*>(g2.d_desc) + h.group_slot;
        cudaMemcpyAsync(&dd->step, &step, sizeof(int), cudaMemcpyHostToDevice, e->stream);
        cudaMemcpyAsync(&dd->arrested, &arrested, sizeof(int), cudaMemcpyHostToDevice, e->stream);
        cudaMemcpyAsync(&dd->e_prev, &e_prev, sizeof(double), cudaMemcpyHostToDevice, e->stream);
    }
    return init_instance(*e, h, 2);
}

int sky_engine_retile(void* handle, int id, int xc) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    HostInst* hp = find(e, id);
    if (!hp) return invalid("unknown instance id");
    if (xc < 0) return invalid("xc must be >= 0 (0: automatic)");
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    HostInst& h = *hp;
    int rc, nxc, tnz, tny, tnx;
    tile_geometry(h, xc, &nxc, &tnz, &tny, &tnx);
    const int ntiles = tnz * tny * tnx;
    const bool own_energy = energy_walk(h.set, h.prec);  // its energy tiles stay as they are
    HostInst nh = h;
    nh.ntiles = ntiles;
    nh.entiles = own_energy ? h.entiles : ntiles;
    Carver size{nullptr};
    take_partials(size, nh);
    void* parts = nullptr;
    if (cudaMalloc(&parts, size.used) != cudaSuccess) {
        cudaGetLastError();
        return SKY_ERR_NOMEM;
    }
    // The per-tile partials of the latest stage 1 feed the next control launch:
    // re-run stage 1 and the control in resume mode under the new geometry (the
    // pending arrest decision and the step's gradient statistics are kept).
    Carver place{reinterpret_cast<char*>(parts)};
    take_partials(place, nh);
    const int gtiles = grad_partials(h.set, ntiles, h.rgrid.count());
    cudaMemsetAsync(nh.gpart, 0, sizeof(double) * 4 * gtiles, e->stream);
    if (h.parts) {
        Carver old{nullptr};
        HostInst oh = h;
        take_partials(old, oh);
        h.bytes -= old.used;
        e->bytes -= (int64_t)old.used;
        cudaFree(h.parts);
    }
    h.parts = parts;
    h.epart = nh.epart;
    h.bpart = nh.bpart;
    h.gpart = nh.gpart;
    h.bytes += size.used;
    e->bytes += (int64_t)size.used;
    h.xc_request = xc;
    h.xc = nxc;
    h.tnx = tnx;
    h.ntiles = ntiles;  // the staging carries over
    h.entiles = nh.entiles;
    Group& g = e->groups[h.set][h.prec];
    if ((rc = rebuild_group(*e, g))) return rc;
    return init_instance(*e, h, 2);
}

int sky_engine_set_staging(void* handle, int id, int tma, int pair) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    HostInst* hp = find(e, id);
    if (!hp) return invalid("unknown instance id");
    if ((tma != 0 && tma != 1) || (pair != 0 && pair != 1)) return invalid("tma and pair must be 0 or 1");
    HostInst& h = *hp;
    if (tma && !tma_possible(h))
        return invalid("TMA staging needs Z * element size a multiple of 16 bytes (and no FP64 rho)");
    if (pair && !(tma && pair_possible(h))) return invalid("z-pair tiles need TMA staging and an FP32 omega instance");
    if (!tma_possible(h) || (h.tma == tma && h.pair == pair)) return SKY_OK;
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    h.tma = tma;
    h.pair = pair;
    return rebuild_group(*e, e->groups[h.set][h.prec]);  // keeps the control state
}

int sky_engine_get_staging(void* handle, int id, int* tma, int* pair) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e || !tma || !pair) return invalid("null argument");
    HostInst* hp = find(e, id);
    if (!hp) return invalid("unknown instance id");
    *tma = hp->tma && tma_possible(*hp);
    *pair = hp->pair;
    return SKY_OK;
}

int sky_engine_audit(void* handle, int id, double* out2) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    if (!out2) return invalid("null output");
    HostInst* hp = find(e, id);
    if (!hp) return invalid("unknown instance id");
    cudaSetDevice(e->device);
    return kernel_ops(hp->set).audit(e->groups[hp->set][hp->prec], *hp, e->stream, out2);
}

int sky_engine_set_defect_period(void* handle, int id, int period) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    HostInst* hp = find(e, id);
    if (!hp) return invalid("unknown instance id");
    if (period < 1) return invalid("defect refresh period must be >= 1");
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    hp->defect_period = period;
    Group& g = e->groups[hp->set][hp->prec];
    const size_t sz = hp->prec ? sizeof(InstDesc<double>) : sizeof(InstDesc<float>);
    const size_t off = hp->prec ? offsetof(InstDesc<double>, refresh_period) : offsetof(InstDesc<float>, refresh_period);
    char* base = reinterpret_cast<char*>(g.d_desc) + sz * hp->group_slot;
    int rc = check_cuda(cudaMemcpyAsync(base + off, &period, sizeof(int), cudaMemcpyHostToDevice, e->stream),
                        "write refresh period", __LINE__);
    if (rc) return rc;
    return check_cuda(cudaStreamSynchronize(e->stream), "sync", __LINE__);
}

int sky_engine_get_xc(void* handle, int id) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return -1;
    HostInst* h = find(e, id);
    return h ? h->xc : -1;
}

int sky_engine_set_active(void* handle, int id, int active) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    HostInst* h = find(e, id);
    if (!h) return invalid("unknown instance id");
    h->active = active != 0;
    Group& g = e->groups[h->set][h->prec];
    const int a = h->active ? 1 : 0;
    size_t off = h->prec ? offsetof(InstDesc<double>, active) : offsetof(InstDesc<float>, active);
    size_t sz = h->prec ? sizeof(InstDesc<double>) : sizeof(InstDesc<float>);
    char* base = reinterpret_cast<char*>(g.d_desc) + sz * h->group_slot + off;
    int rc = check_cuda(cudaMemcpyAsync(base, &a, sizeof(int), cudaMemcpyHostToDevice, e->stream), "set active",
                        __LINE__);
    if (rc) return rc;
    return check_cuda(cudaStreamSynchronize(e->stream), "sync", __LINE__);
}

int sky_engine_step(void* handle, int nsteps) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    if (nsteps < 0) return invalid("nsteps must be >= 0");
    cudaSetDevice(e->device);
    int rc;
    int done = 0;
    if (e->graph_pdl != option(4)) {
        cudaStreamSynchronize(e->stream);
        drop_graphs(*e);
        e->graph_pdl = option(4);
    }
    if (e->graphs.empty() && e->direct_steps + nsteps <= kDirectSteps) {
        for (; done < nsteps; ++done) {
            if ((rc = record_step(*e, refresh_pattern(*e, 1) != 0))) return rc;
            count_steps(*e, 1);
        }
        e->direct_steps += nsteps;
    }
    while (done < nsteps) {
        const int n = nsteps - done >= kGraphSteps ? kGraphSteps : 1;
        cudaGraphExec_t exec;
        if ((rc = step_graph(*e, n, refresh_pattern(*e, n), &exec))) return rc;
        if ((rc = check_cuda(cudaGraphLaunch(exec, e->stream), "graph launch", __LINE__))) return rc;
        count_steps(*e, n);
        done += n;
    }
    return SKY_OK;
}

int sky_engine_synchronize(void* handle) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    return check_cuda(cudaStreamSynchronize(e->stream), "sync", __LINE__);
}

void* sky_engine_stream(void* handle) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    return e ? (void*)e->stream : nullptr;
}

int sky_engine_stats(void* handle, int id, int64_t step, double* out6) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e || !out6) return invalid("null argument");
    HostInst* h = find(e, id);
    if (!h) return invalid("unknown instance id");
    if (step < 0) step = h->steps;
    if (step > h->steps || h->steps - step >= kStatsCap) return invalid("step outside the retained history");
    StepStats st;
    int rc = check_cuda(cudaMemcpyAsync(&st, h->stats + (step % kStatsCap), sizeof(st), cudaMemcpyDeviceToHost,
                                        e->stream),
                        "read stats", __LINE__);
    if (rc) return rc;
    if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "sync", __LINE__))) return rc;
    if ((rc = status_error(st))) return rc;
    out6[0] = st.energy;
    out6[1] = st.baryon;
    out6[2] = st.err;
    out6[3] = st.gabs;
    out6[4] = st.arrested;
    out6[5] = st.step;
    return SKY_OK;
}

int sky_engine_stats_ex(void* handle, int id, int64_t step, double* out8) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e || !out8) return invalid("null argument");
    HostInst* h = find(e, id);
    if (!h) return invalid("unknown instance id");
    if (step < 0) step = h->steps;
    if (step > h->steps || h->steps - step >= kStatsCap) return invalid("step outside the retained history");
    StepStats st;
    int rc = check_cuda(cudaMemcpyAsync(&st, h->stats + (step % kStatsCap), sizeof(st), cudaMemcpyDeviceToHost,
                                        e->stream),
                        "read stats", __LINE__);
    if (rc) return rc;
    if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "sync", __LINE__))) return rc;
    if ((rc = status_error(st))) return rc;
    out8[0] = st.energy;
    out8[1] = st.baryon;
    out8[2] = st.err;
    out8[3] = st.gabs;
    out8[4] = st.arrested;
    out8[5] = st.step;
    out8[6] = st.kinetic;
    out8[7] = h->comp ? 2 + h->defect : h->prec;
    return SKY_OK;
}

int sky_engine_stats_all(void* handle, int* ids_out, double* out7, int cap, int* count_out) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e || !count_out) return invalid("null argument");
    std::vector<StepStats> st(e->insts.size());
    std::vector<const HostInst*> hs;
    int k = 0;
    for (auto& kv : e->insts) {
        if (k >= cap) break;
        const HostInst& h = kv.second;
        int rc = check_cuda(cudaMemcpyAsync(&st[k], h.stats + (h.steps % kStatsCap), sizeof(StepStats),
                                            cudaMemcpyDeviceToHost, e->stream),
                            "read stats", __LINE__);
        if (rc) return rc;
        hs.push_back(&h);
        ++k;
    }
    int rc = check_cuda(cudaStreamSynchronize(e->stream), "sync", __LINE__);
    if (rc) return rc;
    for (int i = 0; i < k; ++i)
        if ((rc = status_error(st[i]))) return rc;
    for (int i = 0; i < k; ++i) {
        if (ids_out) ids_out[i] = hs[i]->id;
        if (out7) {
            double* o = out7 + 7 * i;
            o[0] = st[i].energy;
            o[1] = st[i].baryon;
            o[2] = st[i].err;
            o[3] = st[i].gabs;
            o[4] = st[i].arrested;
            o[5] = st[i].step;
            o[6] = hs[i]->comp ? 2 + hs[i]->defect : hs[i]->prec;
        }
    }
    *count_out = k;
    return SKY_OK;
}

int sky_engine_read(void* handle, int id, double* field, double* velocity, int on_device) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e) return invalid("null engine");
    HostInst* h = find(e, id);
    if (!h) return invalid("unknown instance id");
    cudaSetDevice(e->device);
    Group& g = e->groups[h->set][h->prec];
    const int64_t n = (int64_t)h->C * h->N, nc = (int64_t)h->C * h->sites;
    int rc = SKY_OK;
    auto convert = [&](double* f, double* v) {
        if (h->prec)
            k_read_state<double><<<ew_blocks(n), 256, 0, e->stream>>>(
                reinterpret_cast<const InstDesc<double>*>(g.d_desc) + h->group_slot, n, f, v);
        else
            k_read_state<float><<<ew_blocks(n), 256, 0, e->stream>>>(
                reinterpret_cast<const InstDesc<float>*>(g.d_desc) + h->group_slot, n, f, v);
        return check_cuda(cudaGetLastError(), "convert out", __LINE__);
    };
    if (on_device) {
        if ((field || velocity) && (rc = convert(field, velocity))) return rc;
        return check_cuda(cudaStreamSynchronize(e->stream), "sync", __LINE__);
    }
    double* tmp = nullptr;
    if ((rc = check_cuda(cudaMalloc(&tmp, sizeof(double) * nc), "cudaMalloc(read)", __LINE__))) return rc;
    double* outs[2] = {field, velocity};
    for (int k = 0; k < 2 && rc == SKY_OK; ++k) {
        if (!outs[k]) continue;
        rc = convert(k == 0 ? tmp : nullptr, k == 1 ? tmp : nullptr);
        if (!rc)
            rc = check_cuda(cudaMemcpyAsync(outs[k], tmp, sizeof(double) * nc, cudaMemcpyDeviceToHost, e->stream),
                            "download", __LINE__);
        if (!rc) rc = check_cuda(cudaStreamSynchronize(e->stream), "sync", __LINE__);
    }
    if (tmp) cudaFree(tmp);
    return rc;
}

int sky_engine_time_stages(void* handle, int nsteps, double* ms_out) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    if (!e || !ms_out) return invalid("null argument");
    if (nsteps < 1) return invalid("nsteps must be >= 1");
    cudaSetDevice(e->device);
    int rc = SKY_OK;
    for (int t = 0; t < kNumKernelSets; ++t)
        for (int pr = 0; pr < 2; ++pr)
            if (!e->groups[t][pr].members.empty() && (rc = setup_group(e->groups[t][pr]))) return rc;
    cudaEvent_t ev[kNumKinds + 1];
    for (int k = 0; k <= kNumKinds; ++k)
        if ((rc = check_cuda(cudaEventCreate(&ev[k]), "cudaEventCreate", __LINE__))) return rc;
    double acc[kNumKinds] = {0.0};
    for (int s = 0; s < nsteps && rc == SKY_OK; ++s) {
        for (int k = 0; k < kNumKinds && rc == SKY_OK; ++k) {
            cudaEventRecord(ev[k], e->stream);
            rc = launch_kind(*e, k, false, e->stream);
        }
        if (rc) break;
        cudaEventRecord(ev[kNumKinds], e->stream);
        if ((rc = check_cuda(cudaEventSynchronize(ev[kNumKinds]), "cudaEventSynchronize", __LINE__))) break;
        for (int k = 0; k < kNumKinds; ++k) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ev[k], ev[k + 1]);
            acc[k] += ms;
        }
    }
    for (int k = 0; k <= kNumKinds; ++k) cudaEventDestroy(ev[k]);
    if (rc) return rc;
    count_steps(*e, nsteps);
    // report in the order stage 1, 2, 3, 4, control, advance
    // stage 1 with the defect refresh and the FP32 energy walk
    ms_out[0] = (acc[kKindS1] + acc[kKindDefect] + acc[kKindEnergy]) / nsteps;
    ms_out[1] = acc[kKindS2] / nsteps;
    ms_out[2] = acc[kKindS3] / nsteps;
    ms_out[3] = acc[kKindS4] / nsteps;
    ms_out[4] = 0.0;  // the control and the advance run inside stages 1 and 4
    ms_out[5] = 0.0;
    return SKY_OK;
}

int sky_engine_launches_per_step(void* handle) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    return e ? count_launches(*e) : 0;
}

int sky_engine_count(void* handle) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    return e ? (int)e->insts.size() : 0;
}

int64_t sky_engine_bytes(void* handle) {
    Engine* e = reinterpret_cast<Engine*>(handle);
    return e ? e->bytes : 0;
}

}  // extern "C"
