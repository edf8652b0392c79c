// Engine kernels of the rho theory.
#include "sky_engine_launch.cuh"

namespace sky {
extern const TheoryOps kRhoOps = make_ops<Rho>();
}  // namespace sky
