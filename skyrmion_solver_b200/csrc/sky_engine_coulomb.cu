// Engine kernels of the coulomb theory.
#include "sky_engine_launch.cuh"

namespace sky {
extern const TheoryOps kCoulombOps = make_ops<Coulomb>();
}  // namespace sky
