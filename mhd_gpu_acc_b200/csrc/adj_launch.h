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

// Resident CTAs that the register budgets are cut for: y CTAs of 8 warps, x CTAs
// of 4.  Measured per sweep: FP32 HLL at 512^2 y 37 us with 2 (128 registers, 0.2
// KB of spills) against 42 us with 1 (237, none); x 30 us with 3 x 4 warps (168);
// FP32 HLLD y 74, x 56 us; FP64 at 256^2 HLL y 29, x 21 us, HLLD y 57, x 52 us.  Shapes
// compared with reciprocals good to 2 ulp (FP32: fast math): FP32 HLL x 29.6 us
// against 30.5 us with 2 x 8 warps (128) and 36 us with 1 x 8 (235); FP64 HLLD x 48.5 us
// with 2 x 4 against 50.3 us with 1 x 8 (255 either way).
template <typename R, int SOLVER>
struct AdjShape;
template <int SOLVER>
struct AdjShape<float, SOLVER> { static constexpr int kYBlocks = SOLVER == HLL ? 2 : 1, kXBlocks = 3; };
template <int SOLVER>
struct AdjShape<double, SOLVER> { static constexpr int kYBlocks = 1, kXBlocks = 2; };

}  // namespace adj
}  // namespace mhd
