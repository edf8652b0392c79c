// Engine kernels of the nuclear theory.
#include "sky_engine_launch.cuh"

namespace sky {
extern const TheoryOps kNuclearOps = make_ops<Nuclear>();
}  // namespace sky
