// adj_f64.cu -- the FP64 adjoint sweeps.
#include "adj_sweep.cuh"

namespace mhd {
namespace adj {
cudaError_t launch_adj_sweep_f64(const AdjSweepArgs& a, cudaStream_t st) { return launch_adj<double>(a, st); }
}  // namespace adj
}  // namespace mhd
