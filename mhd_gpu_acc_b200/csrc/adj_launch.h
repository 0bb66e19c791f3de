// adj_launch.h -- entry points of the adjoint sweeps' translation units.
#pragma once

#include <cuda_runtime.h>

#include "mhd_common.cuh"

namespace mhd {
namespace adj {

// One adjoint sweep: lamIn = (sweep)^T lamOut along dir (0: x, 1: y) about the
// sweep's input U, periodic.  lamOut is read with the cotangents of the ghost
// cells that copy its interior across the OTHER direction's periodic side
// (x: its ghost rows, y: its ghost columns); lamIn is written for interior
// lines, ghost positions along dir included.  dir 1 also reverses the psi
// damping: lamOut's psi is scaled by `damp` and its sum with Unext's psi over
// damp goes to acc[2].  acc[0], acc[1] += the cotangents of dt/d and c_h.
struct AdjSweepArgs {
    DevGrid U, lamOut, lamIn, Unext;
    int dir, limiter, solver;
    double gamma, dtd, ch, damp;
    double* acc;
};

cudaError_t launch_adj_sweep_f64(const AdjSweepArgs& a, cudaStream_t st);
cudaError_t launch_adj_sweep_f32(const AdjSweepArgs& a, cudaStream_t st);

// Resident CTAs of 8 warps that the register budget is cut for.
template <typename R, int SOLVER>
struct AdjShape;
template <int SOLVER>
struct AdjShape<float, SOLVER> { static constexpr int kBlocks = SOLVER == HLL ? 2 : 1; };
template <int SOLVER>
struct AdjShape<double, SOLVER> { static constexpr int kBlocks = 1; };

}  // namespace adj
}  // namespace mhd
