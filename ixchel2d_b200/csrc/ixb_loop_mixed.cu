// The resident SIMPLE loop with binary32 line solves around binary64 rows (built with FMA contraction).
#include "ixb_loop.cuh"

namespace ixb {
template cudaError_t loop_launch_form<SOLVER_MIXED>(const LoopArgs&, cudaStream_t);
}  // namespace ixb
