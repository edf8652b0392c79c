// Engine kernels of the omega theory.
#include "sky_engine_launch.cuh"

namespace sky {
extern const TheoryOps kOmegaOps = make_ops<Omega>();
}  // namespace sky
