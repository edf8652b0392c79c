// Engine kernels of the lightly bound theory.
#include "sky_engine_launch.cuh"

namespace sky {
extern const TheoryOps kLightlyBoundOps = make_ops<LightlyBound>();
}  // namespace sky
