// adj_f32.cu -- the FP32 adjoint sweeps.  Build with --use_fast_math, as the
// FP32-bulk step whose branches they follow (step_f32.cu).
#include "adj_sweep.cuh"

namespace mhd {
namespace adj {
cudaError_t launch_adj_sweep_f32(const AdjSweepArgs& a, cudaStream_t st) { return launch_adj<float>(a, st); }
}  // namespace adj
}  // namespace mhd
