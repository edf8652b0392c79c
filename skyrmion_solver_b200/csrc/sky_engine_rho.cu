// Engine kernels of the rho theory.
#include "sky_engine_launch.cuh"

namespace sky {

// FP32 rho of at most kFusedRhoSites sites: 8 rows of all thirteen components, one site per thread.
constexpr int kFusedRows = 8;
template <int STAGE, bool TMA>
struct FusedKernel {
    using M = MarchShape<13, kFusedRows, true>;
    static auto kern() { return k_rho_fused<M, STAGE, TMA>; }
    static size_t smem() { return rho_fused_bytes<M, STAGE, TMA>(); }
    static dim3 block() { return dim3(M::BZ, M::BY); }
};
template <int STAGE, bool TMA>
static int launch_fused_w(const Group& g, const StageArgs& a, cudaStream_t st) {
    using FK = FusedKernel<STAGE, TMA>;
    int per_sm = 1;
    int rc = stage_setup<FK>(&per_sm);
    if (rc) return rc;
    const int n = a.t_end - a.t_begin, blocks = n < num_sms() ? n : num_sms();
    if (n <= 0) return SKY_OK;
    InstDesc<float>* d = reinterpret_cast<InstDesc<float>*>(g.d_desc);
    return launch_chain(a.chained, FK::kern(), blocks, FK::block(), FK::smem(), st, d, d, g.d_tile_inst, a.t_begin,
                        a.t_end, a.in_step, g.d_done, a.in_step && (STAGE == 1 || STAGE == 4) ? 2 * blocks : 0);
}
template <int STAGE>
static int launch_fused(const Group& g, const StageArgs& a, cudaStream_t st) {
    return g.all_tma ? launch_fused_w<STAGE, true>(g, a, st) : launch_fused_w<STAGE, false>(g, a, st);
}
static int fused_stage(int, int stage, const Group& g, const StageArgs& a, cudaStream_t st) {
    switch (stage) {
        case 1: return launch_fused<1>(g, a, st);
        case 2: return launch_fused<2>(g, a, st);
        case 3: return launch_fused<3>(g, a, st);
        default: return launch_fused<4>(g, a, st);
    }
}
template <bool TMA>
static int setup_fused_w() {
    int n, rc;
    if ((rc = stage_setup<FusedKernel<1, TMA>>(&n)) || (rc = stage_setup<FusedKernel<2, TMA>>(&n)) ||
        (rc = stage_setup<FusedKernel<3, TMA>>(&n)))
        return rc;
    return stage_setup<FusedKernel<4, TMA>>(&n);
}
static int setup_fused(const Group& g) {
    return g.all_tma ? setup_fused_w<true>() : setup_fused_w<false>();
}
static TileShapeInfo fused_shape(int) {
    return TileShapeInfo{kFusedRows, 1, MarchShape<13, kFusedRows, true>::HZ, 13, 0, 0};
}

extern const TheoryOps kRhoOps = make_ops<Rho>();
extern const TheoryOps kFusedRhoOps = {fused_shape, setup_fused, fused_stage, launch_energy_t<Rho>,
                                       launch_defect_t<Rho, kFusedRows>, audit_prec<Rho>};
}  // namespace sky
