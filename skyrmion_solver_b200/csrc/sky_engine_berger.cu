// Engine kernels of the berger theory.
#include "sky_engine_launch.cuh"

namespace sky {
extern const TheoryOps kBergerOps = make_ops<Berger>();
}  // namespace sky
