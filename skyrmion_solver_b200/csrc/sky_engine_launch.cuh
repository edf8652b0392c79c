// Launch side of the engine kernels for one theory: tile shapes, kernel variants (wide or
// narrow rows, TMA or cp.async copies) and the table of entry points that sky_engine.cu calls.
#pragma once

#include <cmath>
#include <vector>

#include "sky_engine.cuh"
#include "sky_engine_host.h"

namespace sky {

// ---------------------------------------------------------------------------
// shapes and launches per (theory, precision)
// ---------------------------------------------------------------------------
// Theories of at most five components run the gradient walk (sky_grad.cuh) in both precisions,
// rho the marching tile (sky_march.cuh).
template <template <typename> class Th>
constexpr bool is_walk() {
    return Th<float>::C <= 5;
}
// Rows of a stage tile (32 columns).  FP64 walks: grad_rows64.  FP32 walks, which compute two
// sites per thread: rows and blocks per SM such that the ring, one staging slot and G and H of
// all blocks fit the SM's shared memory and the registers do not spill.  Gradient of 128^3 /
// 64^3 sites, in us: nuclear 16 rows x 2 blocks 54 / 13, 8 x 3 62 / 13; omega 8 x 3 40 / 9,
// 16 x 2 41 / 11; Coulomb 12 x 2 73 / 17, 8 x 2 80 / 15, 16 x 1 83 / 15 (one site per thread,
// 8 rows x 2 blocks: 83 / 17, 60 / 14, 103 / 21).  Rho: 8 rows, or 4 in FP64, whose ring takes
// 150 KB then (narrow rows only, two of stage 3/4's three sources staged).
template <template <typename> class Th, typename T>
constexpr int stage_rows() {
    if (!is_walk<Th>()) return sizeof(T) == 8 ? 4 : 8;
    if (sizeof(T) == 8) return grad_rows64<Th>(true);
    constexpr int id = Th<float>::kId;
    return (id == SKY_THEORY_NUCLEAR || id == SKY_THEORY_LIGHTLY_BOUND) ? 16 : 12;
}
// Resident blocks per SM the stages are compiled for, and their x-chunks chosen with.
template <template <typename> class Th, typename T>
constexpr int stage_blocks() {
    return (sizeof(T) == 4 && is_walk<Th>()) ? 2 : 1;
}
// Wide-row (16-byte copies) or narrow-row shape; FP64 rho has narrow rows only.
template <template <typename> class Th, typename T>
constexpr bool wide_allowed() {
    return is_walk<Th>() || sizeof(T) == 4;
}
template <template <typename> class Th, typename T, bool WIDE>
using MShape = MarchShape<Th<T>::C, stage_rows<Th, T>(), WIDE && wide_allowed<Th, T>(),
                          (sizeof(T) == 8 && is_walk<Th>()) ? 2 : 4>;

template <template <typename> class Th, typename T, int STAGE, bool WIDE, bool TMA>
struct StageKernel {
    using M = MShape<Th, T, WIDE>;
    static auto kern() {
        if constexpr (is_walk<Th>())
            return k_grad_stage<Th, M, T, STAGE, stage_blocks<Th, T>(), TMA>;
        else
            return k_march_stage<Th, M, T, STAGE, TMA>;
    }
    static size_t smem() {
        if constexpr (is_walk<Th>())
            return grad_stage_bytes<Th, M, T, STAGE, TMA>();
        else
            return march_stage_bytes<M, T, STAGE, TMA>();
    }
    static dim3 block() { return is_walk<Th>() ? dim3(GradBlock<M, T>::TZ, M::BY) : dim3(M::BZ, M::BY); }
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

template <template <typename> class Th, typename T, int STAGE, bool WIDE, bool TMA>
static int stage_setup(int* per_sm_out) {
    static int per_sm = 0;
    using SK = StageKernel<Th, T, STAGE, WIDE, TMA>;
    if (per_sm == 0) {
        const dim3 b = SK::block();
        const int rc = kernel_setup(SK::kern(), SK::smem(), int(b.x * b.y), &per_sm);
        if (rc) return rc;
    }
    *per_sm_out = per_sm;
    return SKY_OK;
}

// Launch with programmatic dependent launch when option 4 asks for it.
template <class... Args, class... Given>
static int launch_pdl(void (*kern)(Args...), int blocks, dim3 block, size_t smem, cudaStream_t st, Given... args) {
    if (option(4) == 1) {
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

template <template <typename> class Th, typename T, int STAGE, bool WIDE, bool TMA>
static int launch_stage_w(const Group& g, const StageArgs& a, cudaStream_t st) {
    int per_sm = 1;
    int rc = stage_setup<Th, T, STAGE, WIDE, TMA>(&per_sm);
    if (rc) return rc;
    const int n = a.t_end - a.t_begin;
    if (n <= 0) return SKY_OK;
    const int blocks = n < num_sms() * per_sm ? n : num_sms() * per_sm;
    int total = 0;
    if (a.in_step && (STAGE == 1 || STAGE == 4)) {  // both launches that share the step's tail counter
        int other = 1;
        if ((rc = stage_setup<Th, T, STAGE == 1 ? 4 : 1, WIDE, TMA>(&other))) return rc;
        total = blocks + (n < num_sms() * other ? n : num_sms() * other);
    }
    InstDesc<T>* d = reinterpret_cast<InstDesc<T>*>(g.d_desc);
    using SK = StageKernel<Th, T, STAGE, WIDE, TMA>;
    return launch_pdl(SK::kern(), blocks, SK::block(), SK::smem(), st, d, d, g.d_tile_inst, a.t_begin, a.t_end,
                      a.in_step, g.d_done, total);
}

template <template <typename> class Th, typename T, int STAGE>
static int launch_stage(const Group& g, const StageArgs& a, cudaStream_t st) {
    if constexpr (wide_allowed<Th, T>()) {
        if (g.all_tma) return launch_stage_w<Th, T, STAGE, true, true>(g, a, st);
        if (g.all_wide) return launch_stage_w<Th, T, STAGE, true, false>(g, a, st);
    }
    return launch_stage_w<Th, T, STAGE, false, false>(g, a, st);
}

// Energy walk of a group's FP32 instances (theories of at most five components; the others'
// energy is summed by stage 1), energy tiles [t_begin, t_end).
template <template <typename> class Th, bool WIDE, bool TMA>
static int energy_setup(int* per_sm_out) {
    static int per_sm = 0;
    using M = MarchShape<Th<double>::C, kEnergyRows, WIDE, 4>;
    using Pipe = DensPipe<M, float, 2, TMA>;
    if (per_sm == 0) {
        const int rc = kernel_setup(k_energy<Th, M, TMA>, Pipe::bytes + (TMA ? 128 : 0), M::NTHREADS, &per_sm);
        if (rc) return rc;
    }
    *per_sm_out = per_sm;
    return SKY_OK;
}
template <template <typename> class Th, bool WIDE, bool TMA>
static int launch_energy_w(const Group& g, const StageArgs& a, cudaStream_t st) {
    using M = MarchShape<Th<double>::C, kEnergyRows, WIDE, 4>;
    using Pipe = DensPipe<M, float, 2, TMA>;
    int per_sm = 1;
    int rc = energy_setup<Th, WIDE, TMA>(&per_sm);
    if (rc) return rc;
    const int n = a.t_end - a.t_begin;
    if (n <= 0) return SKY_OK;
    const int blocks = n < num_sms() * per_sm ? n : num_sms() * per_sm;
    return launch_pdl(k_energy<Th, M, TMA>, blocks, dim3(M::BZ, M::BY), Pipe::bytes + (TMA ? 128 : 0), st,
                      reinterpret_cast<InstDesc<float>*>(g.d_desc), g.d_tile_inst + g.ntiles, a.t_begin, a.t_end,
                      a.in_step);
}
template <template <typename> class Th>
static int launch_energy_t(const Group& g, const StageArgs& a, cudaStream_t st) {
    if constexpr (is_walk<Th>()) {
        if (g.all_tma) return launch_energy_w<Th, true, true>(g, a, st);
        if (g.all_wide) return launch_energy_w<Th, true, false>(g, a, st);
        return launch_energy_w<Th, false, false>(g, a, st);
    }
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

template <template <typename> class Th, typename T, bool WIDE, bool TMA>
static int setup_stages() {
    int n, rc;
    if ((rc = stage_setup<Th, T, 1, WIDE, TMA>(&n)) || (rc = stage_setup<Th, T, 2, WIDE, TMA>(&n)) ||
        (rc = stage_setup<Th, T, 3, WIDE, TMA>(&n)) || (rc = stage_setup<Th, T, 4, WIDE, TMA>(&n)))
        return rc;
    if constexpr (sizeof(T) == 4 && is_walk<Th>()) return energy_setup<Th, WIDE, TMA>(&n);
    return SKY_OK;
}
template <template <typename> class Th, typename T>
static int setup_all() {
    int rc;
    if ((rc = setup_stages<Th, T, false, false>())) return rc;
    if constexpr (wide_allowed<Th, T>()) {
        if ((rc = setup_stages<Th, T, true, false>()) || (rc = setup_stages<Th, T, true, true>())) return rc;
    }
    return SKY_OK;
}

template <template <typename> class Th>
static int setup_prec(int prec) {
    return prec ? setup_all<Th, double>() : setup_all<Th, float>();
}

// Tile geometry of a (theory, precision): rows of its stage tiles, the resident blocks per SM
// their x-chunk is chosen for, and the columns of a staged row (TMA boxes).  The geometry does
// not depend on the staging, so neither does the order of the per-tile partial sums.
template <template <typename> class Th>
static TileShapeInfo shape_of(int prec) {
    return prec ? TileShapeInfo{stage_rows<Th, double>(), stage_blocks<Th, double>(), MShape<Th, double, true>::HZ}
                : TileShapeInfo{stage_rows<Th, float>(), stage_blocks<Th, float>(), MShape<Th, float, true>::HZ};
}

// Defect refresh of the group's defect-corrected FP32 instances (those whose
// refresh flag the stage-4 advance just set; the others' tiles are skipped).
template <template <typename> class Th, bool WIDE>
static int launch_defect_t(const Group& g, cudaStream_t st) {
    // 4-row sub-tiles of an engine tile's rows, or 8 where they divide them and the ring fits
    constexpr int rows = is_walk<Th>() && stage_rows<Th, float>() % 8 == 0 ? 8 : 4;
    using M = MarchShape<Th<double>::C, rows, WIDE && is_walk<Th>()>;
    auto kern = k_march_defect<Th, M, stage_rows<Th, float>()>;
    size_t smem;
    if constexpr (is_walk<Th>())
        smem = GradPipe<Th, M, double, float, 2, false>::bytes;
    else
        smem = M::template smem_bytes<double, float>(2);
    static int per_sm = 0;
    if (per_sm == 0) {
        int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                            "cudaFuncSetAttribute(defect)", __LINE__);
        if (rc) return rc;
        int n = 0;
        rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, M::NTHREADS, smem), "occupancy",
                        __LINE__);
        if (rc) return rc;
        per_sm = n < 1 ? 1 : n;
    }
    const int n = g.ntiles;
    if (n <= 0) return SKY_OK;
    const int blocks = n < num_sms() * per_sm ? n : num_sms() * per_sm;
    kern<<<blocks, dim3(M::BZ, M::BY), smem, st>>>(reinterpret_cast<InstDesc<float>*>(g.d_desc), g.d_tile_inst, 0,
                                                   n);
    return check_cuda(cudaGetLastError(), "launch defect refresh", __LINE__);
}

template <template <typename> class Th>
static int launch_defect_w(const Group& g, cudaStream_t st) {
    return g.all_wide ? launch_defect_t<Th, true>(g, st) : launch_defect_t<Th, false>(g, st);
}

// Energy audit of the RK4 dynamics (k_engine_audit).
template <template <typename> class Th>
constexpr int audit_rows() {
    return Th<double>::C > 5 ? 4 : kDensRows;  // a 13-component FP64 ring with staged FP32 sources fits
}

template <template <typename> class Th, typename S>
static int audit_t(const Group& g, const HostInst& h, cudaStream_t st, double* out2) {
    using M = MarchShape<Th<double>::C, audit_rows<Th>(), false>;
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
    return TheoryOps{shape_of<Th>, setup_prec<Th>, stage_dispatch_prec<Th>, launch_energy_t<Th>, launch_defect_w<Th>,
                     audit_prec<Th>};
}

}  // namespace sky
