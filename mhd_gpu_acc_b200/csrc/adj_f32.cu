// adj_f32.cu -- the FP32 adjoint sweeps.
#include "adj_sweep.cuh"

namespace mhd {
namespace adj {
cudaError_t launch_adj_sweep_f32(const AdjSweepArgs& a, cudaStream_t st) { return launch_adj<float>(a, st); }
}  // namespace adj
}  // namespace mhd
