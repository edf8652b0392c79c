// Launch side of the engine kernels for one theory: tile shapes, kernel variants (TMA or
// cp.async copies) and the table of entry points that sky_engine.cu calls.
#pragma once

#include <cmath>
#include <vector>

#include "sky_engine.cuh"
#include "sky_engine_host.h"

namespace sky {

// ---------------------------------------------------------------------------
// shapes and launches per (theory, precision)
// ---------------------------------------------------------------------------
// The theory of the stages' gradient walk: rho's is over the pion components and follows a walk
// over the rho components (sky_rho.cuh).
template <template <typename> class Th>
constexpr bool is_rho() {
    return Th<float>::kId == SKY_THEORY_RHO;
}
// Rows of a stage tile (32 columns).  FP64 walks: grad_rows64.  FP32 walks, which compute two
// sites per thread: rows and blocks per SM such that the ring, one staging slot and G and H of
// all blocks fit the SM's shared memory and the registers do not spill.  Gradient of 128^3 /
// 64^3 sites, in us: nuclear 16 rows x 2 blocks 54 / 13, 8 x 3 62 / 13; omega 8 x 3 40 / 9,
// 16 x 2 41 / 11; Coulomb 12 x 2 73 / 17, 8 x 2 80 / 15, 16 x 1 83 / 15 (one site per thread,
// 8 rows x 2 blocks: 83 / 17, 60 / 14, 103 / 21).  Omega's stages run 8 x 3: with 12 x 2 whole steps
// took longer and left more of a last tile empty (step in us, 12 x 2 / 16 x 2 / 8 x 3 / one site per
// thread with 8 x 2 blocks: 48^3 63 / 67 / 62 / 60, 64^3 78 / 83 / 72 / 74, 112^3 269 / 288 / 263 / 246,
// 128^3 315 / 331 / 311 / 322).  Rho's walk over the pions spills with 16.
template <template <typename> class Th, typename T>
constexpr int stage_rows() {
    if (sizeof(T) == 8) return grad_rows64<Th>(true);
    constexpr int id = Th<float>::kId;
    return id == SKY_THEORY_NUCLEAR || id == SKY_THEORY_LIGHTLY_BOUND ? 16 : id == SKY_THEORY_OMEGA ? 8 : 12;
}
// Resident blocks per SM the stages are compiled for, and their x-chunks chosen with.
template <template <typename> class Th, typename T>
constexpr int stage_blocks() {
    return sizeof(T) == 8 ? 1 : stage_rows<Th, T>() == 8 ? 3 : 2;
}
template <template <typename> class Th, typename T>
using MShape = MarchShape<is_rho<Th>() ? 4 : Th<T>::C, stage_rows<Th, T>(), true, sizeof(T) == 8 ? 2 : 4>;

template <template <typename> class Th, typename T, int STAGE, bool TMA>
struct StageKernel {
    using M = MShape<Th, T>;
    static auto kern() {
        if constexpr (is_rho<Th>())
            return k_grad_stage<RhoPion, M, T, STAGE, stage_blocks<Th, T>(), TMA>;
        else
            return k_grad_stage<Th, M, T, STAGE, stage_blocks<Th, T>(), TMA>;
    }
    static size_t smem() {
        if constexpr (is_rho<Th>())
            return grad_stage_bytes<RhoPion, M, T, STAGE, TMA>();
        else
            return grad_stage_bytes<Th, M, T, STAGE, TMA>();
    }
    static dim3 block() { return dim3(GradBlock<M, T>::TZ, M::BY); }
};
// Rho: the stage's walk over the rho components.
template <typename T>
constexpr int rho_rows() {
    return sizeof(T) == 8 ? 8 : 12;
}
template <typename T>
constexpr int rho_blocks() {
    return sizeof(T) == 8 ? 2 : 3;
}
template <template <typename> class Th, typename T, int STAGE, bool TMA>
struct RhoKernel {
    using M = MarchShape<3, rho_rows<T>(), true, sizeof(T) == 8 ? 2 : 4>;
    static auto kern() { return k_rho_stage<M, T, STAGE, rho_blocks<T>(), TMA>; }
    static size_t smem() { return rho_stage_bytes<M, T, STAGE, TMA>(); }
    static dim3 block() { return dim3(GradBlock<M, T>::TZ, M::BY); }
};

// One-time kernel attribute setup (kept out of stream capture); returns the
// number of resident blocks per SM.
template <class K>
static int kernel_setup(K kern, size_t smem, int threads, int* per_sm) {
    int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                        "cudaFuncSetAttribute(engine kernel)", __LINE__);
    if (rc) return rc;
    int n = 0;
    rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem), "occupancy query",
                    __LINE__);
    if (rc) return rc;
    *per_sm = n < 1 ? 1 : n;
    return SKY_OK;
}

template <class SK>
static int stage_setup(int* per_sm_out) {
    static int per_sm = 0;
    if (per_sm == 0) {
        const dim3 b = SK::block();
        const int rc = kernel_setup(SK::kern(), SK::smem(), int(b.x * b.y), &per_sm);
        if (rc) return rc;
    }
    *per_sm_out = per_sm;
    return SKY_OK;
}

// Launch, programmatically dependent on its predecessor where `chained` (a kernel of the step precedes
// it in the same stream) or when option 4 asks for it everywhere.  Every kernel of a step waits for its
// predecessor before it reads anything, so the dependence is transitive; what overlaps is the launch.
// An event recorded between the two (a fork, a timing pass) only turns the programmatic dependence of
// a launch outside a graph into a full one; in a captured step it leaves no node and no trace.
template <class... Args, class... Given>
static int launch_chain(bool chained, void (*kern)(Args...), int blocks, dim3 block, size_t smem, cudaStream_t st, Given... args) {
    if (chained || option(4) == 1) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return check_cuda(cudaLaunchKernelEx(&cfg, kern, static_cast<Args>(args)...), "launch engine kernel", __LINE__);
    }
    kern<<<blocks, block, smem, st>>>(args...);
    return check_cuda(cudaGetLastError(), "launch engine kernel", __LINE__);
}

template <template <typename> class Th, typename T, int STAGE, bool TMA>
static int launch_stage_w(const Group& g, const StageArgs& a, cudaStream_t st) {
    using SK = StageKernel<Th, T, STAGE, TMA>;
    int per_sm = 1;
    int rc = stage_setup<SK>(&per_sm);
    if (rc) return rc;
    const int n = a.t_end - a.t_begin;
    if (n <= 0) return SKY_OK;
    InstDesc<T>* d = reinterpret_cast<InstDesc<T>*>(g.d_desc);
    if constexpr (is_rho<Th>()) {
        using RK = RhoKernel<Th, T, STAGE, TMA>;
        int rho_per_sm = 1;
        if ((rc = stage_setup<RK>(&rho_per_sm))) return rc;
        const int resident = num_sms() * rho_per_sm, items = 3 * (a.r_end - a.r_begin);
        if ((rc = launch_chain(a.chained, RK::kern(), items < resident ? items : resident, RK::block(), RK::smem(), st, d,
                             g.d_tile_inst + g.ntiles + g.entiles, a.r_begin, a.r_end, a.in_step)))
            return rc;
    }
    const int blocks = n < num_sms() * per_sm ? n : num_sms() * per_sm;
    int total = 0;
    const bool tail = a.in_step && (STAGE == 1 || STAGE == 4);  // both stages' last launches share the tail counter
    if constexpr (is_rho<Th>()) {
        if ((rc = launch_chain(true, SK::kern(), blocks, SK::block(), SK::smem(), st, d, d, g.d_tile_inst, a.t_begin,
                               a.t_end, a.in_step, g.d_done, 0)))
            return rc;
        const int fi = kRhoFinishSplit * (a.r_end - a.r_begin), fb = fi < 4 * num_sms() ? fi : 4 * num_sms();
        if (tail) total = 2 * fb;
        return launch_chain(true, k_rho_finish<T, STAGE>, fb, dim3(kRhoFinishThreads), 0, st, d, d,
                          g.d_tile_inst + g.ntiles + g.entiles, a.r_begin, a.r_end, a.in_step, g.d_done, total);
    }
    if (tail) {
        int other = 1;
        if ((rc = stage_setup<StageKernel<Th, T, STAGE == 1 ? 4 : 1, TMA>>(&other))) return rc;
        total = blocks + (n < num_sms() * other ? n : num_sms() * other);
    }
    return launch_chain(a.chained, SK::kern(), blocks, SK::block(), SK::smem(), st, d, d, g.d_tile_inst, a.t_begin, a.t_end,
                      a.in_step, g.d_done, total);
}

template <template <typename> class Th, typename T, int STAGE>
static int launch_stage(const Group& g, const StageArgs& a, cudaStream_t st) {
    // (FP64 rho has no TMA maps: tma_possible)
    if constexpr (!(is_rho<Th>() && sizeof(T) == 8)) {
        if (g.all_tma) return launch_stage_w<Th, T, STAGE, true>(g, a, st);
    }
    return launch_stage_w<Th, T, STAGE, false>(g, a, st);
}

// Energy walk of a group's instances (energy_walk), energy tiles [t_begin, t_end).  CURL: FP32 rho's
// walk over the rho components, which comes first.
template <template <typename> class Th, typename T>
constexpr bool split_energy() {
    return is_rho<Th>() && sizeof(T) == 4;
}
template <template <typename> class Th, typename T, bool TMA, bool CURL>
struct EnergyKernel {
    using M = MarchShape<CURL ? 3 : split_energy<Th, T>() ? 4 : Th<double>::C, kDensRows, true, sizeof(T) == 8 ? 2 : 4>;
    using Pipe = DensPipe<M, T, sizeof(T) == 8 ? 1 : 2, TMA, CURL>;
    static auto kern() {
        if constexpr (split_energy<Th, T>())
            return k_energy<RhoPion, M, T, TMA, CURL>;
        else
            return k_energy<Th, M, T, TMA, CURL>;
    }
    static size_t smem() { return Pipe::bytes + (TMA ? 128 : 0); }
    static dim3 block() { return dim3(M::BZ, M::BY); }
};
template <class EK, typename T>
static int launch_energy_k(const Group& g, const StageArgs& a, int per, cudaStream_t st) {
    int per_sm = 1;
    int rc = stage_setup<EK>(&per_sm);
    if (rc) return rc;
    const int n = per * (a.t_end - a.t_begin);
    if (n <= 0) return SKY_OK;
    const int blocks = n < num_sms() * per_sm ? n : num_sms() * per_sm;
    return launch_chain(a.chained, EK::kern(), blocks, EK::block(), EK::smem(), st, reinterpret_cast<InstDesc<T>*>(g.d_desc),
                      g.d_tile_inst + g.ntiles, a.t_begin, a.t_end, a.in_step);
}
template <template <typename> class Th, typename T, bool TMA>
static int launch_energy_w(const Group& g, const StageArgs& a, cudaStream_t st) {
    if constexpr (split_energy<Th, T>()) {
        const int rc = launch_energy_k<EnergyKernel<Th, T, TMA, true>, T>(g, a, 3, st);
        if (rc) return rc;
        StageArgs b = a;
        b.chained = 1;
        return launch_energy_k<EnergyKernel<Th, T, TMA, false>, T>(g, b, 1, st);
    }
    return launch_energy_k<EnergyKernel<Th, T, TMA, false>, T>(g, a, 1, st);
}
template <template <typename> class Th, typename T>
static int launch_energy_p(const Group& g, const StageArgs& a, cudaStream_t st) {
    if constexpr (sizeof(T) == 4) {
        if (g.all_tma) return launch_energy_w<Th, T, true>(g, a, st);
    }
    return launch_energy_w<Th, T, false>(g, a, st);
}
template <template <typename> class Th>
static int launch_energy_t(const Group& g, const StageArgs& a, cudaStream_t st) {
    if (!g.prec) return launch_energy_p<Th, float>(g, a, st);
    if constexpr (energy_walk<double>(Th<double>::kId)) return launch_energy_p<Th, double>(g, a, st);
    return SKY_OK;
}
template <template <typename> class Th, typename T>
static int launch_stage_any(int stage, const Group& g, const StageArgs& a, cudaStream_t st) {
    switch (stage) {
        case 1: return launch_stage<Th, T, 1>(g, a, st);
        case 2: return launch_stage<Th, T, 2>(g, a, st);
        case 3: return launch_stage<Th, T, 3>(g, a, st);
        default: return launch_stage<Th, T, 4>(g, a, st);
    }
}

template <template <typename> class Th>
static int stage_dispatch_prec(int prec, int stage, const Group& g, const StageArgs& a, cudaStream_t st) {
    return prec ? launch_stage_any<Th, double>(stage, g, a, st) : launch_stage_any<Th, float>(stage, g, a, st);
}

template <template <typename> class Th, typename T, int STAGE, bool TMA>
static int setup_stage() {
    int n, rc = stage_setup<StageKernel<Th, T, STAGE, TMA>>(&n);
    if constexpr (is_rho<Th>()) {
        if (!rc) rc = stage_setup<RhoKernel<Th, T, STAGE, TMA>>(&n);
    }
    return rc;
}
template <template <typename> class Th, typename T, bool TMA>
static int setup_stages() {
    int n, rc;
    if ((rc = setup_stage<Th, T, 1, TMA>()) || (rc = setup_stage<Th, T, 2, TMA>()) ||
        (rc = setup_stage<Th, T, 3, TMA>()) || (rc = setup_stage<Th, T, 4, TMA>()))
        return rc;
    if constexpr (energy_walk<T>(Th<T>::kId)) {
        if constexpr (split_energy<Th, T>()) {
            if ((rc = stage_setup<EnergyKernel<Th, T, TMA, true>>(&n))) return rc;
        }
        return stage_setup<EnergyKernel<Th, T, TMA, false>>(&n);
    }
    return SKY_OK;
}
template <template <typename> class Th, typename T>
static int setup_prec(const Group& g) {
    if constexpr (!(is_rho<Th>() && sizeof(T) == 8)) {
        if (g.all_tma) return setup_stages<Th, T, true>();
    }
    return setup_stages<Th, T, false>();
}
// Kernel attributes of the variants that a group's steps launch (kept out of stream capture).
template <template <typename> class Th>
static int setup_group_kernels(const Group& g) {
    return g.prec ? setup_prec<Th, double>(g) : setup_prec<Th, float>(g);
}

// Tile geometry of a (theory, precision): rows of its stage tiles, the resident blocks per SM
// their x-chunk is chosen for, and the columns of a staged row (TMA boxes).  The geometry does
// not depend on the staging, so neither does the order of the per-tile partial sums.
template <template <typename> class Th>
static TileShapeInfo shape_of(int prec) {
    return prec ? TileShapeInfo{stage_rows<Th, double>(), stage_blocks<Th, double>(), MShape<Th, double>::HZ,
                                MShape<Th, double>::C, rho_rows<double>(),
                                rho_blocks<double>()}
                : TileShapeInfo{stage_rows<Th, float>(), stage_blocks<Th, float>(), MShape<Th, float>::HZ,
                                MShape<Th, float>::C, rho_rows<float>(),
                                rho_blocks<float>()};
}

// Defect refresh of the group's defect-corrected FP32 instances (those whose refresh is due; the
// others' tiles are skipped).
template <class M, int PER, class K>
static int launch_defect_k(bool chained, K kern, size_t smem, int* per_sm, const Group& g, cudaStream_t st) {
    int rc;
    if (*per_sm == 0 && (rc = kernel_setup(kern, smem, M::NTHREADS, per_sm))) return rc;
    const int n = PER * g.ntiles;
    if (n <= 0) return SKY_OK;
    const int blocks = n < num_sms() * *per_sm ? n : num_sms() * *per_sm;
    return launch_chain(chained, kern, blocks, dim3(M::BZ, M::BY), smem, st,
                        reinterpret_cast<InstDesc<float>*>(g.d_desc), g.d_tile_inst, 0, g.ntiles);
}
// TBY: rows of the stage tiles.
template <template <typename> class Th, int TBY = stage_rows<Th, float>()>
static int launch_defect_t(const Group& g, cudaStream_t st) {
    // two sub-tiles of a 16-row engine tile, one of the others
    constexpr int rows = TBY == 16 ? 8 : TBY;
    static int per_sm = 0;
    if constexpr (is_rho<Th>()) {
        using R = MarchShape<3, rows, true>;
        using M = MarchShape<4, rows, true>;
        static int rho_per_sm = 0;
        const int rc = launch_defect_k<R, 3>(false, k_defect<RhoPion, R, TBY, true>,
                                             RhoPipe<R, double, float, 2, false>::bytes, &rho_per_sm, g, st);
        if (rc) return rc;
        return launch_defect_k<M, 1>(true, k_defect<RhoPion, M, TBY, false>,
                                     GradPipe<RhoPion, M, double, float, 2, false>::bytes, &per_sm, g, st);
    } else {
        using M = MarchShape<Th<double>::C, rows, true>;
        return launch_defect_k<M, 1>(false, k_defect<Th, M, TBY, false>, GradPipe<Th, M, double, float, 2, false>::bytes,
                                     &per_sm, g, st);
    }
}

// Energy audit of the RK4 dynamics (k_engine_audit).
template <template <typename> class Th>
constexpr int audit_rows() {
    return Th<double>::C > 5 ? 4 : kDensRows;  // a 13-component FP64 ring with staged FP32 sources fits
}

template <template <typename> class Th, typename S>
static int audit_t(const Group& g, const HostInst& h, cudaStream_t st, double* out2) {
    using M = MarchShape<Th<double>::C, audit_rows<Th>(), true, std::is_same<S, double>::value ? 2 : 4>;
    constexpr int NSRC = std::is_same<S, double>::value ? 1 : 2;
    auto kern = k_engine_audit<Th, M, S>;
    const size_t smem = DensPipe<M, S, NSRC, false>::bytes;
    static bool configured = false;
    if (!configured) {
        int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                            "cudaFuncSetAttribute(audit)", __LINE__);
        if (rc) return rc;
        configured = true;
    }
    const MarchGrid g0 = march_grid<M>(h.p, h.p.X);
    const MarchGrid mg = march_grid<M>(h.p, choose_chunk(h.p.X, g0.nz * g0.ny, num_sms()));
    const int blocks = mg.count() < num_sms() ? mg.count() : num_sms();
    double* parts = nullptr;
    int rc = check_cuda(cudaMalloc(&parts, sizeof(double) * 4 * blocks), "cudaMalloc(audit)", __LINE__);
    if (rc) return rc;
    const InstDesc<S>* d = reinterpret_cast<const InstDesc<S>*>(g.d_desc) + h.group_slot;
    kern<<<blocks, dim3(M::BZ, M::BY), smem, st>>>(d, mg, parts);
    rc = check_cuda(cudaGetLastError(), "launch audit", __LINE__);
    std::vector<double> hp(4 * (size_t)blocks);
    if (!rc)
        rc = check_cuda(cudaMemcpyAsync(hp.data(), parts, sizeof(double) * hp.size(), cudaMemcpyDeviceToHost, st),
                        "read audit", __LINE__);
    if (!rc) rc = check_cuda(cudaStreamSynchronize(st), "sync audit", __LINE__);
    cudaFree(parts);
    if (rc) return rc;
    // fixed-order compensated sum of the block partials
    for (int q = 0; q < 2; ++q) {
        double sum = 0.0, comp = 0.0;
        for (int b = 0; b < blocks; ++b) {
            for (int k = 0; k < 2; ++k) {
                const double v = hp[4 * b + 2 * q + k];
                const double t = sum + v;
                comp += (std::fabs(sum) >= std::fabs(v)) ? ((sum - t) + v) : ((v - t) + sum);
                sum = t;
            }
        }
        out2[q] = sum + comp;
    }
    return SKY_OK;
}

template <template <typename> class Th>
static int audit_prec(const Group& g, const HostInst& h, cudaStream_t st, double* out2) {
    return h.prec ? audit_t<Th, double>(g, h, st, out2) : audit_t<Th, float>(g, h, st, out2);
}

template <template <typename> class Th>
constexpr TheoryOps make_ops() {
    return TheoryOps{shape_of<Th>, setup_group_kernels<Th>, stage_dispatch_prec<Th>, launch_energy_t<Th>, launch_defect_t<Th>,
                     audit_prec<Th>};
}

}  // namespace sky
