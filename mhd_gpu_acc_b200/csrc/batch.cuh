// batch.cuh -- many independent instances of uneven size advanced together.
//
// Each instance (its own grid, gamma, CFL, c_r, boundary types, t_end and
// device clock) is cut into the same tasks the single-grid sweeps use: row
// segments marched by one warp each (x_segment) and row bands of 32-column
// strips (y_march), in equal lengths up to the longest that suits the size of the
// whole batch, the last eighth of its rows in a third of that.  Four consecutive
// tasks of one instance and length form a unit, the work of one CTA.  The units
// of all instances form one global list, longest tasks first, so that the launch
// ends on short ones; a table gives each unit's segment (one per instance and
// length).  One launch per sweep phase advances every instance; the kernel
// boundary between the x and y phases is the only synchronisation a step needs,
// and a CUDA graph of two steps replays the loop.
// The first unit of an instance performs the clock duties the single-grid
// kernels give to CTA (0, 0).
//
// By default a CTA takes one unit and the hardware deals them out: at 96
// instances of 64..1024 cells a side (29.5M cells, FP32 HLLD, van Leer) x 1.21 ->
// 0.89 ms and y 1.99 -> 1.19 ms against 444 CTAs striding over the list in fixed
// order with one task length (kDefaultBatchXRpw, kDefaultYSeg; of the y gain 0.2 ms
// is the ghost scatter's).  An explicit tuning sets the task lengths, how many of
// the x CTAs are resident at a time, and the CTAs that stride over the y list.
#pragma once

#include <algorithm>

#include "dispatch.cuh"

namespace mhd {

constexpr int BX_WARPS = 4;  // warps per batched x-sweep CTA

// The device table holds every instance twice, with P.parity 0 and then 1, so that
// the kernels can read an instance's parameters where they lie.
struct BatchInst {
    DevGrid U;
    void* T;       // the x-swept state, of U's layout
    StepParams P;  // physics, boundary types, t_end, clock and step parity of this instance
};

// n tasks of `len` cells (the last may be shorter) per row / strip, covering
// [lo, hi) of each of the `width` rows (x) or strips (y) from idx0 on of an
// instance; `lead`: the segment's first unit (`unit` of the list) does the
// instance's clock duties.
struct BatchSeg {
    int inst, lo, hi, len, n, idx0, width, lead, unit;
};

// Task `task` of a segment: false past its last.
__device__ __forceinline__ bool seg_task(const BatchSeg& s, int task, int& idx, int& start, int& len) {
    if (task >= s.n * s.width) return false;
    idx = s.idx0 + task % s.width;
    start = s.lo + task / s.width * s.len;
    len = min(s.len, s.hi - start);
    return true;
}

// Dynamic shared memory of the batched x-sweep: one x_segment ring per warp.
template <class PH>
constexpr int bx_smem_bytes() { return BX_WARPS * XRing<PH>::kWarpBytes; }

// CTA u takes unit u, under any tuning: with a loop over units the march spills 8
// bytes (908 against 892 us at 96 instances of 64..1024 cells a side), and a second
// kernel with the loop contracts other FP32 multiply-adds, which would make results
// depend on the launch shape.
template <class PH>
__global__ void __launch_bounds__(32 * BX_WARPS, PH::kXBlocks)
    batch_x_kernel(const BatchInst* __restrict__ inst, const BatchSeg* __restrict__ seg, const int* __restrict__ unit_seg) {
    using V = typename Slot16<typename PH::Real>::V;
    extern __shared__ __align__(16) unsigned char bx_smem[];
    const int warp = threadIdx.x >> 5;
    V* ring = reinterpret_cast<V*>(bx_smem + warp * XRing<PH>::kWarpBytes);
    const BatchSeg s = seg[__ldg(unit_seg + blockIdx.x)];
    const int local = (int)blockIdx.x - s.unit;
    const bool lead = s.lead && local == 0 && threadIdx.x == 0;
    const StepParams& P = inst[s.inst].P;
    double dt, ch, damp;
    if (!step_scalars(P, dt, ch, damp)) {
        if (lead) clock_flag_skip(P);
        return;
    }
    if (lead) P.clock->maxbits[P.parity ^ 1] = 0ull;
    int row, c0, len;
    if (seg_task(s, local * BX_WARPS + warp, row, c0, len)) {  // whole warp
        const DevGrid in = inst[s.inst].U;
        DevGrid out = in;
        out.data = inst[s.inst].T;
        x_segment<PH>(in, out, P, dt, ch, in.ng + row, c0, len, ring);
    }
}

template <class PH>
__global__ void __launch_bounds__(32 * YS_WARPS, PH::kYBlocks)
    batch_y_kernel(const BatchInst* __restrict__ inst, const BatchSeg* __restrict__ seg, const int* __restrict__ unit_seg,
                   int total) {
    using R = typename PH::Real;
    __shared__ __align__(16) R carry[PH::kYCarry ? YS_WARPS * YCarry<PH>::kSlots * 32 : 1];
    // The instance in shared memory, read where it is used: held in registers (as
    // the single-grid sweep holds nothing, its parameters being constants) it
    // makes the march spill, and spills miss in the L1 that the windows leave.
    __shared__ BatchInst I;
    __shared__ DevGrid T;
    for (int u = blockIdx.x; u < total; u += gridDim.x) {
        const BatchSeg s = seg[__ldg(unit_seg + u)];
        const int local = u - s.unit;
        const bool lead = s.lead && local == 0 && threadIdx.x == 0 && threadIdx.y == 0;
        static_assert(sizeof(BatchInst) % 4 == 0 && sizeof(BatchInst) / 4 <= 32 * YS_WARPS, "copied a word per thread");
        __syncthreads();  // the unit before may still be reading I
        const int q = threadIdx.y * 32 + threadIdx.x;
        if (q < (int)(sizeof(BatchInst) / 4)) reinterpret_cast<int*>(&I)[q] = reinterpret_cast<const int*>(&inst[s.inst])[q];
        __syncthreads();
        if (q == 0) {
            T = I.U;
            T.data = I.T;
        }
        __syncthreads();
        const StepParams& P = I.P;
        double dt, ch, damp;
        if (!step_scalars(P, dt, ch, damp)) {
            if (lead) clock_flag_skip(P);
            continue;
        }
        double vmax = 0.0;
        unsigned reverts = 0;
        int strip, r0, count;
        if (seg_task(s, local * YS_WARPS + threadIdx.y, strip, r0, count)) {
            y_march<PH>(T, I.U, P, dt, ch, damp, strip, T.ng + r0, count, vmax, reverts,
                        carry + threadIdx.y * YCarry<PH>::kSlots * 32);
        }
        y_fold(P, vmax, reverts);
        if (lead) clock_advance(P);
    }
}

// CFL maximum of every instance (compute_dt's, floored by the instance's ch) into
// maxbits[0] of its clock, which starts at 0: CTAs of 256 threads take
// kMaxUnit cells of one instance each, one atomic per CTA.
constexpr int kMaxUnit = 4096;
// Unit k of an instance: n cells in row order from column i0 of row j0 on (an
// instance may have 2^31 cells and more).
__host__ __device__ __forceinline__ long long max_units(const DevGrid& g) {
    return ((long long)g.nx * g.ny + kMaxUnit - 1) / kMaxUnit;
}
__host__ __device__ __forceinline__ void max_unit(const DevGrid& g, int k, int& i0, int& j0, int& n) {
    const long long c0 = (long long)k * kMaxUnit, left = (long long)g.nx * g.ny - c0;
    j0 = c0 <= 0xffffffffLL ? (int)((unsigned)c0 / (unsigned)g.nx) : (int)(c0 / g.nx);
    i0 = (int)(c0 - (long long)j0 * g.nx);
    n = left < kMaxUnit ? (int)left : kMaxUnit;
}
template <class PH>
__global__ void __launch_bounds__(256) batch_max_kernel(const BatchInst* __restrict__ inst,
                                                       const BatchSeg* __restrict__ seg,
                                                       const int* __restrict__ unit_seg,
                                                       const double* __restrict__ ch) {
    using R = typename PH::Real;
    __shared__ double part[8];
    const BatchSeg s = seg[__ldg(unit_seg + blockIdx.x)];
    const BatchInst& I = inst[s.inst];
    const DevGrid g = I.U;
    const double gamma = I.P.gamma, floor_ch = ch[s.inst];
    int i0, j0, n;
    max_unit(g, (int)blockIdx.x - s.unit, i0, j0, n);
    double vmax = 0.0;
    for (int c = threadIdx.x; c < n; c += 256) {
        const unsigned q = (unsigned)i0 + c, dj = q / (unsigned)g.nx;
        R U[NV];
        load_cell(g, g.ng + (int)(q - dj * (unsigned)g.nx), g.ng + j0 + (int)dj, U);
        const double v = PH::speed(U, gamma, floor_ch);
        vmax = (vmax < v) ? v : vmax;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_xor_sync(FULL, vmax, o);
        vmax = (vmax < t) ? t : vmax;
    }
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = vmax;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) vmax = (vmax < part[w]) ? part[w] : vmax;
        atomic_max_pos(&I.P.clock->maxbits[0], vmax);
    }
}

// Dynamic shared memory of an x phase of which `ctas` CTAs (0: as many as fit) are
// to be resident at a time: an even share of the SM for each.
template <class PH>
int bx_smem_of(int ctas) {
    const int per_sm = ctas > 0 ? std::max(1, ctas / kSMs) : PH::kXBlocks;
    return per_sm < PH::kXBlocks ? kSmemPerSM / per_sm - kSmemPerCTAReserve : bx_smem_bytes<PH>();
}

// The x phase's dynamic shared memory opt-in (once per policy and device,
// before any stream capture: mhd_batch_run makes a which = 0 call first).
template <class PH>
cudaError_t bx_setup() {
    static_assert(PH::kXBlocks * (bx_smem_bytes<PH>() + kSmemPerCTAReserve) <= kSmemPerSM,
                  "batched x-phase rings of kXBlocks CTAs exceed an SM's shared memory");
    static PerDeviceOnce once;
    return once.run([] {
        const auto k = batch_x_kernel<PH>;
        cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bx_smem_of<PH>(1));
        if (r == cudaSuccess)
            r = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
        // the y phase's window and parameters are a little over the 40 KB of which
        // four CTAs fit the 164 KB split that the runtime picks: ask for the next one,
        // 196 of 228 KB (85 %; more leaves too little L1)
        if (r == cudaSuccess)
            r = cudaFuncSetAttribute(batch_y_kernel<PH>, cudaFuncAttributePreferredSharedMemoryCarveout, 85);
        return r;
    });
}

// One phase's work list.
struct BatchList {
    const BatchSeg* seg;
    const int* unit_seg;  // the segment of each unit
    int units;
};

struct BatchLaunch {
    const BatchInst* inst;
    BatchList list;
    int n, parity, which, ctas;
    cudaStream_t st;
    template <class PH>
    cudaError_t run() const {
        const cudaError_t attr = bx_setup<PH>();
        if (attr != cudaSuccess || which == 0) return attr;  // which 0: the set-up alone
        const BatchInst* I = inst + parity * n;
        const dim3 yb(32, YS_WARPS);
        if (which == 2)
            batch_y_kernel<PH><<<ctas > 0 ? ctas : list.units, yb, 0, st>>>(I, list.seg, list.unit_seg, list.units);
        else
            batch_x_kernel<PH><<<list.units, 32 * BX_WARPS, bx_smem_of<PH>(ctas), st>>>(I, list.seg, list.unit_seg);
        return cudaGetLastError();
    }
};

template <template <int, int> class POL>
cudaError_t dispatch_batch(const BatchInst* inst, const BatchList& list, const double* ch, int n, int parity, int which,
                           int solver, int limiter, int ctas, cudaStream_t st) {
    if (which == 3) {
        batch_max_kernel<POL<HLL, MINMOD>><<<list.units, 256, 0, st>>>(inst, list.seg, list.unit_seg, ch);
        return cudaGetLastError();
    }
    BatchLaunch go{inst, list, n, parity, which, ctas, st};
    return with_policy<POL>(solver, limiter, go);
}

// Longest x and y tasks by the size of the whole batch (iterations of all
// instances over the resident warps), as the single-grid sweeps take theirs.
template <class PH>
void batch_task_lens(long long x_work, long long y_work, TaskLen& x, TaskLen& y) {
    x = task_len(x_work, kSMs * PH::kXBlocks * BX_WARPS, PH::kXTask, 4 * PH::kXRpw, kXOneWave);
    y = task_len(y_work, kSMs * PH::kYBlocks * YS_WARPS, PH::kYTask, PH::kYBand, kYOneWave);
}

}  // namespace mhd
