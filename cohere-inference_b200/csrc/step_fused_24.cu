// The fused small-batch step (step_fused.cuh) for one weight mode, its own translation unit so the modes compile in
// parallel.
#include "step_fused.cuh"

namespace b200dec_detail {
int launch_fused_24(const FArgs& a, int head_dim, bool q8, cudaStream_t s) { return launch_fused_mode<FM_INT8_24>(a, head_dim, q8, s); }
}  // namespace b200dec_detail
