// The resident SIMPLE loop in the fast binary64 form (built with FMA contraction).
#include "ixb_loop.cuh"

namespace ixb {
template cudaError_t loop_launch_form<IXB_SOLVER_HYBRID>(const LoopArgs&, cudaStream_t);
}  // namespace ixb
