// Host structures of the resident engine, and what each theory's translation unit provides.
#pragma once

#include <vector>

#include "sky_common.cuh"
#include "sky_host.h"

namespace sky {

struct StepStats;

struct HostInst {
    int id = -1;
    int theory = 0;
    int set = 0;   // kernel set (kernel_set)
    int prec = 0;  // storage: 0 = FP32 storage/arithmetic, 1 = FP64
    int comp = 0;    // FP32 storage with a compensated (hi + lo) field
    int defect = 0;  // ... and a defect-corrected gradient (precision 3)
    int defect_period = kDefectRefresh;  // steps between refreshes of the correction
    Params p{};
    int64_t sites = 0;  // lattice sites: values of a component in the caller's arrays
    int64_t N = 0;      // values of a component here, rows padded to p.Zp (n_sites)
    int C = 0;
    void* arena = nullptr;  // one allocation that holds every array below
    void* parts = nullptr;  // the partials' own allocation once sky_engine_retile has changed their sizes
    void* F[2] = {nullptr, nullptr};
    void* Flo[2] = {nullptr, nullptr};
    void* Dlt = nullptr;
    void* V[2] = {nullptr, nullptr};
    void* L[3] = {nullptr, nullptr, nullptr};
    double* curl = nullptr;  // FP32 rho: curls of the energy walks
    KSum* epart = nullptr;
    KSum* bpart = nullptr;
    double* gpart = nullptr;
    StepStats* stats = nullptr;
    int ntiles = 0, tnz = 0, tny = 0, tnx = 0;
    int entiles = 0, etnz = 0, etny = 0, etnx = 0, exc = 0;  // energy tiles (entiles = ntiles: stage 1 sums it)
    MarchGrid rgrid{0, 0, 0, 1};  // rho: tiles of the walk over the rho components
    int xc = 0;          // x-chunk of the marching kernels
    int xc_request = 0;  // x-chunk asked for by the caller (0: automatic)
    bool tma = false;    // the stage kernels stage this instance with TMA box copies
    bool pair = false;   // the caller's z-pair flag (option 3): every FP32 walk computes z-pairs
    int group_slot = -1;
    int64_t steps = 0;  // host mirror of the device step counter
    bool active = true;
    size_t bytes = 0;
};

struct Group {
    int set = 0, prec = 0;
    std::vector<int> members;  // instance ids in slot order
    void* d_desc = nullptr;    // InstDesc<S>[cap]
    int* d_tile_inst = nullptr;   // stage tiles, energy tiles, tiles of the walk over the rho components
    int* d_done = nullptr;     // blocks of the current step's stage-1 and stage-4 launches finished (0 between steps)
    int desc_cap = 0, tile_cap = 0;
    int ntiles = 0, entiles = 0, rtiles = 0;
    bool any_defect = false;  // holds a defect-corrected instance (launch the defect refresh)
    bool all_tma = false;     // every member has TMA plane maps (launch the TMA stage kernels)
};

// Shapes and launches of one theory (sky_engine_launch.cuh, instantiated per theory in
// sky_engine_<theory>.cu).
struct TileShapeInfo {
    int rows, blocks, hz;  // rows of a stage tile; resident blocks per SM its x-chunk is chosen for; staged columns
    int components;        // of the gradient walk (rho: the pion field's four)
    int rho_rows, rho_blocks;  // rows and resident blocks per SM of the walk over the rho components
};
// Tiles [t_begin, t_end) of a stage or energy launch.  in_step: part of a step (the work on the
// new field; stages 1 and 4 share the control tail); 0: on the current field alone (admission,
// precision change).
// [r_begin, r_end): tiles of rho's walk over the rho components.
struct StageArgs {
    int t_begin, t_end, in_step, r_begin, r_end;
    int chained;  // a kernel of the step precedes the launch in its stream (launch_chain)
};
struct TheoryOps {
    TileShapeInfo (*shape)(int prec);
    int (*setup)(const Group& g);
    int (*stage)(int prec, int stage, const Group& g, const StageArgs& a, cudaStream_t st);
    int (*energy)(const Group& g, const StageArgs& a, cudaStream_t st);  // groups with an energy walk
    int (*defect)(const Group& g, cudaStream_t st);
    int (*audit)(const Group& g, const HostInst& h, cudaStream_t st, double* out2);
};
const TheoryOps& kernel_ops(int set);
extern const TheoryOps kNuclearOps, kOmegaOps, kCoulombOps, kRhoOps, kBergerOps, kLightlyBoundOps, kFusedRhoOps;

// FP32 rho sums the energy in two walks, whose tiles have four partials (the pions' and the three
// isospin components').
inline bool split_energy(int set, int prec) { return set == SKY_THEORY_RHO && prec == 0; }
inline int energy_partials(int set, int prec, int entiles) { return split_energy(set, prec) ? 4 * entiles : entiles; }
// Entries of an instance's stage-4 partials: one per tile, and those of rho's epilogue of the rho
// components (rtiles: tiles of the walk over them).
inline int grad_partials(int set, int ntiles, int rtiles) {
    return ntiles + (set == SKY_THEORY_RHO ? kRhoFinishSplit * rtiles : 0);
}
inline bool late_update(int set, int prec) { return prec ? late_update<double>(set) : late_update<float>(set); }
inline bool energy_walk(int set, int prec) { return prec ? energy_walk<double>(set) : energy_walk<float>(set); }

}  // namespace sky
