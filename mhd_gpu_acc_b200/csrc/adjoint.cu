// adjoint.cu -- discrete adjoint of the split GLM-MHD step (HLL or HLLD, van
// Leer or minmod, periodic boundaries) and the Orszag-Tang gradient problem of
// the C ABI (mhd_adjoint_*).
//
// Forward step n (the sweeps of mhd_advance; dt_n, c_h,n and f_n are formed on
// the device from the CFL maximum that the step before folded, and logged):
//   m_n = max(c_h,n-1, max_cells s(U^n)),  c_h,n = m_n,  dt_n = cfl dmin / m_n,
//   T = X(U^n) (x-sweep + ghost fill),  V = Y(T) (y-sweep + ghost fill),
//   U^{n+1} = V with interior psi scaled by f_n = exp(-dt_n c_h,n / c_r)
//   (ghost psi undamped, as the reference orders it).
// Reverse step n, with lambda = dJ/dU^{n+1} on the cells the next x-sweep reads:
//   (a) lambda_T = Y^T lambda_V about the stored T, lambda_V being lambda with the
//       ghost-column cotangents folded onto their periodic sources and the damping
//       applied; sums for dJ/d(dt/dy), dJ/dc_h and dJ/df_n;
//   (b) lambda_U = X^T lambda_T about the stored U^n, lambda_T with its ghost rows
//       folded; sums for dJ/d(dt/dx), dJ/dc_h;
//   (c) dJ/dm_n from dt_n, c_h,n and f_n (plus the next step's floor when it
//       was c_h,n itself) goes to the argmax cell of U^n through the CFL speed.
//       Only a step whose own maximum set c_h has such a cell; the sums of the
//       steps between wait until then.
// Every branch is re-evaluated from the stored forward states, i.e. the
// adjoint differentiates the branches the forward took.
// Storage for N steps in segments of S: the states of one segment and a
// checkpoint per segment, from which the segments before the last are
// recomputed with the logged dt, c_h and f (N/S + S + 1 states).  Where S more
// fit an eighth of the free memory the segment keeps each step's T too; else the
// reverse recomputes T.  One segment of all steps (no recomputation) is the
// default where that fits the same eighth: 512^2 x 400 steps take 8.6 GB in FP32.
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/mhd_b200.h"
#include "adj_launch.h"
#include "adj_physics.cuh"
#include "launch.h"
#include "sweep.cuh"

namespace mhd {
int report_error(int code, const char* msg);
void count_launches(unsigned n);
}

namespace mhd {
namespace adj {

// J = 1/2 sum_interior (rho - target)^2 (added to *J) and, with lam.data,
// lambda_N = (rho - target) e_rho.  One atomic per CTA.
template <typename R>
__global__ void __launch_bounds__(256) objective_kernel(DevGrid U, const double* target, DevGrid lam, double* J) {
    __shared__ double part[8];
    const long long n = (long long)U.nx * U.ny;
    double s = 0.0;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(k / U.nx) + U.ng, i = (int)(k % U.nx) + U.ng;
        const double d = (double)static_cast<const R*>(U.data)[U.idx(i, j)] - target[k];
        s += 0.5 * d * d;
        if (lam.data) static_cast<R*>(lam.data)[lam.idx(i, j)] = (R)d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) s += part[w];
        atomicAdd(J, s);
    }
}

// Reverse of the CFL speed of the argmax cell (*idx; INT_MAX: none) with weight
// *lm (the step's combined dt / c_h cotangent, from step_scalars_kernel).
template <typename R>
__global__ void speed_adj_kernel(DevGrid U, DevGrid lam, const int* idx_p, R g, const double* lm_p) {
    const int idx = *idx_p;
    if (idx == INT_MAX) return;
    const R lm = (R)*lm_p;
    const int j = idx / U.nx + U.ng, i = idx % U.nx + U.ng;
    R u[NV], l[NV];
    load_cell(U, i, j, u);
    load_cell(lam, i, j, l);
    int branch = 0;
    raw_speed(u, g, &branch);
    raw_speed_adj(u, g, branch, lm, l);
    store_cell(lam, i, j, l);
}

// Scalars of the reverse pass, on the device so that it needs no host round
// trip.  Step n's sums sc[5 n ..]: [0, 1] the y-sweep's dt/dy and c_h, [2]
// sum(lambda_psi psi / f) of the damping, [3, 4] the x-sweep's dt/dx and c_h.
// Called for a step n1 whose own maximum set c_h, with the steps n1 .. n2 not
// yet combined: a step n > n1 passes its weight on as the floor of step n - 1
// and step n1's argmax cell takes *lm.  Explicit round-to-nearest operations.
// One warp: the terms of 32 steps at once, then their chain in step order (a
// one-thread loop waited for memory at every step: 22 -> 4 us for 30 steps).
__global__ void __launch_bounds__(32) step_scalars_kernel(const double* sc, const double* log, int n1, int n2, double cr,
                                                         double dx, double dy, double* lm, int* idx) {
    double carry = 0.0;
    for (int top = n2; top >= n1; top -= 32) {
        const int n = top - (int)threadIdx.x;
        double own = 0.0, slope = 0.0;
        if (n >= n1) {
            const double* s = sc + 5 * n;
            const double dt = log[3 * n], ch = log[3 * n + 1], f = log[3 * n + 2];
            const double ldt = __dadd_rn(__dadd_rn(__ddiv_rn(s[3], dx), __ddiv_rn(s[0], dy)),
                                         __dmul_rn(__dmul_rn(s[2], f), __ddiv_rn(-ch, cr)));
            own = __dadd_rn(__dadd_rn(s[4], s[1]), __dmul_rn(__dmul_rn(s[2], f), __ddiv_rn(-dt, cr)));
            slope = __dmul_rn(ldt, __ddiv_rn(-dt, ch));
        }
        for (int k = 0; k < 32 && top - k >= n1; ++k)
            carry = __dadd_rn(__dadd_rn(__shfl_sync(FULL, own, k), carry), __shfl_sync(FULL, slope, k));
    }
    if (threadIdx.x == 0) {
        *lm = carry;
        *idx = INT_MAX;
    }
}

// grad_k += sum over every cell (ghosts included) of lambda_0 . dU0/da_k for the
// perturbed Orszag-Tang initial data (mhd_initialise_orszag_tang).  Mode m of
// wave vector (mx, my) is sin(2 pi (mx x + my y)) / |(mx, my)|: with x fixed for
// a thread that walks down a column, a cell costs one sincos of y (sums and
// doubled angles give the eight modes) instead of eight sines, and a CTA adds
// its 16 sums once: 127 -> 14 us at 512^2 FP32.
constexpr int IC_ROWS = 8;
__host__ __device__ inline unsigned ic_blocks_across(const DevGrid& g) { return (g.tnx() + 255) / 256; }
template <typename R>
__global__ void __launch_bounds__(256) ic_grad_kernel(DevGrid lam, DevGrid U0, double x0, double y0, double dx,
                                                      double dy, double* grad) {
    __shared__ double part[16][8];
    const double T = 2.0 * 3.14159265358979323846, h2 = 0.70710678118654752440, h5 = 0.44721359549995793928;
    const unsigned across = ic_blocks_across(lam);
    const int i = blockIdx.x % across * 256 + threadIdx.x, j0 = blockIdx.x / across * IC_ROWS;
    double gk[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) gk[k] = 0.0;
    if (i < lam.tnx()) {
        double sx, cx;
        sincos(T * (x0 + ((double)(i - lam.ng) + 0.5) * dx), &sx, &cx);
        const double sx2 = 2.0 * sx * cx, cx2 = (cx - sx) * (cx + sx);
        for (int j = j0; j < min(j0 + IC_ROWS, lam.tny()); ++j) {
            double sy, cy;
            sincos(T * (y0 + ((double)(j - lam.ng) + 0.5) * dy), &sy, &cy);
            const double sy2 = 2.0 * sy * cy, cy2 = (cy - sy) * (cy + sy);
            R l[NV], u[NV];
            load_cell(lam, i, j, l);
            load_cell(U0, i, j, u);
            const double rho = u[RHO], uu = u[MX] / rho, vv = u[MY] / rho, bx = u[BX], by = u[BY], lE = l[EN];
            // cotangents of (u, v) and of (Bx, By)
            const double lu = (double)l[MX] * rho + lE * rho * uu, lv = (double)l[MY] * rho + lE * rho * vv;
            const double lbx = (double)l[BX] + lE * bx, lby = (double)l[BY] + lE * by;
            // d(u, v)/d amp = sin (-my, mx) / |m|
            const double m[8] = {sx, sy, (sx * cy + cx * sy) * h2, (sx * cy - cx * sy) * h2, sx2 * 0.5, sy2 * 0.5,
                                 (sx2 * cy + cx2 * sy) * h5, (sx * cy2 + cx * sy2) * h5};
            constexpr double mx[8] = {1, 0, 1, 1, 2, 0, 2, 1}, my[8] = {0, 1, 1, -1, 0, 2, 1, 2};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                gk[k] += m[k] * (mx[k] * lv - my[k] * lu);
                gk[8 + k] += m[k] * (mx[k] * lby - my[k] * lbx);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        double v = gk[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        if ((threadIdx.x & 31) == 0) part[k][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 16) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += part[threadIdx.x][w];
        atomicAdd(grad + threadIdx.x, v);
    }
}

unsigned blocks_for(long long n) {
    long long b = (n + 255) / 256;
    if (b > 8 * kSMs) b = 8 * kSMs;
    return (unsigned)(b < 1 ? 1 : b);
}

}  // namespace adj
}  // namespace mhd

// ---------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------
struct mhd_adjoint {
    int nx = 0, ny = 0, dtype = MHD_F64, limiter = MHD_LIMITER_VANLEER, solver = MHD_HLL, nsteps = 0, every = 1;
    double gamma = 5.0 / 3.0, cfl = 0.4, cr = 0.18, b0 = 0.0;
    void* slab = nullptr;                // the states below, one allocation
    std::vector<mhd_grid> ckpt;          // U at the start of each segment (empty with one segment)
    std::vector<mhd_grid> seg, segT;     // the segment's U (S + 1) and x-swept T (S, or one for all steps)
    mhd_grid lamA{}, lamB{}, lamT{};
    mhd_workspace* ws = nullptr;
    double* d_target = nullptr;          // ny * nx
    mhd::DevClock* d_clock = nullptr;    // of the forward solve
    unsigned long long* d_acc = nullptr;  // the CFL maximum's scratch (MaxOut), zero between launches
    double* d_log = nullptr;             // {dt, ch, damp} of each step, then J: one block that the host reads once
    double* d_sc = nullptr;              // 5 reverse sums per step, then the argmax weight
    double* d_grad = nullptr;            // 16
    int* d_idx = nullptr;
    std::vector<double> log;             // the host's copy of d_log
    bool have_target = false;

    double* d_J() const { return d_log + 3 * nsteps; }
    size_t log_len() const { return (size_t)3 * nsteps + 1; }
};

namespace {

using mhd::DevGrid;

int aerr(int code, const char* msg) { return mhd::report_error(code, msg); }

#define ACK(call)                                                                \
    do {                                                                         \
        cudaError_t e_ = (call);                                                 \
        if (e_ != cudaSuccess) return aerr(MHD_ERR_CUDA, cudaGetErrorString(e_)); \
    } while (0)
#define ARC(call)               \
    do {                        \
        int r_ = (call);        \
        if (r_) return r_;      \
    } while (0)

DevGrid dg(const mhd_grid& g) { return DevGrid{g.data, g.pitch, g.plane, g.nx, g.ny, g.ng, 0}; }

bool f64(const mhd_adjoint* a) { return a->dtype == MHD_F64; }

int grid_copy(const mhd_grid& dst, const mhd_grid& src, cudaStream_t st) {
    const size_t eb = src.dtype == MHD_F32 ? 4 : 8;
    ACK(cudaMemcpyAsync(dst.data, src.data, (size_t)src.plane * MHD_NV * eb, cudaMemcpyDeviceToDevice, st));
    return MHD_OK;
}

int zero_grid(const mhd_grid& g, cudaStream_t st) {
    const size_t eb = g.dtype == MHD_F32 ? 4 : 8;
    ACK(cudaMemsetAsync(g.data, 0, (size_t)g.plane * MHD_NV * eb, st));
    return MHD_OK;
}

mhd::StepParams step_params(const mhd_adjoint* a) {  // bc: all periodic (0)
    mhd::StepParams P{};
    const double dx = 1.0 / a->nx, dy = 1.0 / a->ny;
    P.gamma = a->gamma; P.cr = a->cr; P.cfl = a->cfl; P.dx = dx; P.dy = dy; P.dmin = dy < dx ? dy : dx;
    P.solver = a->solver; P.limiter = a->limiter;
    return P;
}

mhd_grid& slot_T(mhd_adjoint* a, int i) { return a->segT[a->segT.size() > 1 ? i : 0]; }

cudaError_t launch_sweeps(const mhd_adjoint* a, const mhd_grid& U, const mhd_grid& T, const mhd_grid& V,
                          const mhd::StepParams& P, int which) {
    mhd::count_launches(which == 3 ? 2 : 1);
    return f64(a) ? mhd::launch_step_f64(dg(U), dg(T), dg(V), P, nullptr, mhd::kDefaultYBand, which)
                  : mhd::launch_step_f32(dg(U), dg(T), dg(V), P, nullptr, mhd::kDefaultYBand, which);
}

// Forward step n of segment slot i; `first`: dt and c_h on the device clock, which
// logs them and folds the next maximum; else (a recomputation) from the log.
int fwd_step(mhd_adjoint* a, int n, int i, bool first) {
    mhd::StepParams P = step_params(a);
    if (first) {
        P.clock = a->d_clock;
        P.parity = n & 1;
        P.accumulate = 1;
        P.t_end = HUGE_VAL;  // nsteps steps, whatever the time
        P.dt_min = 0.0;
    } else {
        P.dt = a->log[3 * n]; P.ch = a->log[3 * n + 1]; P.damp = a->log[3 * n + 2];
    }
    ACK(launch_sweeps(a, a->seg[i], slot_T(a, i), a->seg[i + 1], P, 3));
    return MHD_OK;
}

// Forward solve from amp: leaves the last segment's states in seg / segT, the
// others' starts in ckpt, and the steps' scalars in log.  lam (may be null)
// receives lambda_N.
int forward(mhd_adjoint* a, const double* amp, double* J, double* rho_final, const mhd_grid* lam) {
    cudaStream_t st = nullptr;
    ACK(cudaMemsetAsync(a->d_log, 0, sizeof(double) * a->log_len(), st));
    ARC(mhd_initialise_orszag_tang(a->ws, &a->seg[0], a->b0, a->gamma, amp));
    if (!a->ckpt.empty()) ARC(grid_copy(a->ckpt[0], a->seg[0], st));
    mhd::MaxOut out{};
    out.acc = a->d_acc;
    out.count = reinterpret_cast<unsigned*>(a->d_acc + 1);
    out.clock = a->d_clock;
    out.log = a->d_log;
    ACK(f64(a) ? mhd::launch_max_speed_f64(dg(a->seg[0]), a->gamma, 0.0, out, st)
               : mhd::launch_max_speed_f32(dg(a->seg[0]), a->gamma, 0.0, out, st));
    int last = 0;
    for (int n = 0; n < a->nsteps; ++n) {
        const int i = n % a->every;
        if (i == 0 && n > 0) {
            ARC(grid_copy(a->seg[0], a->seg[a->every], st));
            ARC(grid_copy(a->ckpt[n / a->every], a->seg[0], st));
        }
        ARC(fwd_step(a, n, i, true));
        last = i + 1;
    }
    if (a->have_target) {
        const DevGrid U = dg(a->seg[last]);
        const DevGrid l = lam ? dg(*lam) : DevGrid{nullptr, U.pitch, U.plane, U.nx, U.ny, U.ng, 0};
        const unsigned blocks = mhd::adj::blocks_for((long long)a->nx * a->ny);
        if (f64(a)) mhd::adj::objective_kernel<double><<<blocks, 256, 0, st>>>(U, a->d_target, l, a->d_J());
        else mhd::adj::objective_kernel<float><<<blocks, 256, 0, st>>>(U, a->d_target, l, a->d_J());
        ACK(cudaGetLastError());
    }
    mhd::count_launches(a->have_target ? 2 : 1);
    a->log.resize(a->log_len());
    ACK(cudaMemcpy(a->log.data(), a->d_log, sizeof(double) * a->log_len(), cudaMemcpyDeviceToHost));
    for (int n = 0; n < a->nsteps; ++n)  // a step that was not taken logged nothing
        if (!(a->log[3 * n] > 0.0))
            return aerr(MHD_ERR_NO_SPEED, "mhd_adjoint: non-positive maximum wave speed");
    if (J) *J = a->log[3 * a->nsteps];
    if (rho_final) {
        std::vector<double> h((size_t)MHD_NV * (a->nx + 4) * (a->ny + 4));
        ARC(mhd_grid_download(&a->seg[last], h.data()));
        const int tnx = a->nx + 4;
        for (int j = 0; j < a->ny; ++j)
            for (int i = 0; i < a->nx; ++i) rho_final[(size_t)j * a->nx + i] = h[(size_t)(j + 2) * tnx + i + 2];
    }
    return MHD_OK;
}

// Reverse of step n (segment slot i): lam_next -> lam_out.  `pending`: the last
// step whose sums no argmax cell has taken yet.
int reverse_step(mhd_adjoint* a, int n, int i, const mhd_grid& lam_next, const mhd_grid& lam_out, int* pending) {
    cudaStream_t st = nullptr;
    const double dt = a->log[3 * n], ch = a->log[3 * n + 1], f = a->log[3 * n + 2];
    const double dx = 1.0 / a->nx, dy = 1.0 / a->ny;
    if (a->segT.size() == 1 && a->every > 1) {
        mhd::StepParams P = step_params(a);
        P.dt = dt; P.ch = ch; P.damp = f;
        ACK(launch_sweeps(a, a->seg[i], a->segT[0], a->segT[0], P, 1));
    }
    const auto sweep = f64(a) ? mhd::adj::launch_adj_sweep_f64 : mhd::adj::launch_adj_sweep_f32;
    mhd::adj::AdjSweepArgs s{};
    s.limiter = a->limiter; s.solver = a->solver; s.gamma = a->gamma; s.ch = ch; s.damp = f;
    s.dir = 1; s.U = dg(slot_T(a, i)); s.lamOut = dg(lam_next); s.lamIn = dg(a->lamT); s.Unext = dg(a->seg[i + 1]);
    s.dtd = dt / dy; s.acc = a->d_sc + 5 * n;
    ACK(sweep(s, st));
    s.dir = 0; s.U = dg(a->seg[i]); s.lamOut = dg(a->lamT); s.lamIn = dg(lam_out);
    s.dtd = dt / dx; s.acc = a->d_sc + 5 * n + 3;
    ACK(sweep(s, st));
    mhd::count_launches(2);
    // the time step and cleaning speed: dt = cfl dmin / c_h with c_h the larger of
    // this step's maximum speed and the previous c_h
    const double ch_prev = n > 0 ? a->log[3 * n - 2] : 0.0;
    if (ch > ch_prev) {
        double* lm = a->d_sc + 5 * a->nsteps;
        mhd::adj::step_scalars_kernel<<<1, 32, 0, st>>>(a->d_sc, a->d_log, n, *pending, a->cr, dx, dy, lm, a->d_idx);
        ACK(cudaGetLastError());
        ACK(f64(a) ? mhd::launch_argmax_f64(dg(a->seg[i]), a->gamma, ch_prev, ch, a->d_idx, st)
                   : mhd::launch_argmax_f32(dg(a->seg[i]), a->gamma, ch_prev, ch, a->d_idx, st));
        if (f64(a)) mhd::adj::speed_adj_kernel<double><<<1, 1, 0, st>>>(dg(a->seg[i]), dg(lam_out), a->d_idx, a->gamma, lm);
        else mhd::adj::speed_adj_kernel<float><<<1, 1, 0, st>>>(dg(a->seg[i]), dg(lam_out), a->d_idx, (float)a->gamma, lm);
        ACK(cudaGetLastError());
        mhd::count_launches(3);
        *pending = n - 1;
    }
    return MHD_OK;
}

int gradient(mhd_adjoint* a, const double* amp, double* J, double* grad) {
    cudaStream_t st = nullptr;
    // cells that no launch writes (ghost rows and corners) stay zero
    ARC(zero_grid(a->lamA, st));
    ARC(zero_grid(a->lamB, st));
    ACK(cudaMemsetAsync(a->d_sc, 0, sizeof(double) * ((size_t)5 * a->nsteps + 1), st));
    ACK(cudaMemsetAsync(a->d_grad, 0, sizeof(double) * 16, st));
    ARC(forward(a, amp, J, nullptr, &a->lamA));
    const mhd_grid *lam_next = &a->lamA, *lam_cur = &a->lamB;
    const int nseg = (a->nsteps + a->every - 1) / a->every;
    int pending = a->nsteps - 1;
    for (int k = nseg - 1; k >= 0; --k) {
        const int n0 = k * a->every, n1 = std::min(a->nsteps, n0 + a->every);
        if (k < nseg - 1) {  // the forward solve left the last segment in place
            ARC(grid_copy(a->seg[0], a->ckpt[k], st));
            for (int n = n0; n < n1; ++n) ARC(fwd_step(a, n, n - n0, false));
        }
        for (int n = n1 - 1; n >= n0; --n) {
            ARC(reverse_step(a, n, n - n0, *lam_next, *lam_cur, &pending));
            std::swap(lam_next, lam_cur);
        }
    }
    // lam_next now holds dJ/dU^0 (ghosts included) and seg[0] U^0: contract with dU^0/da
    // one dimension: the others of a grid end at 65,535 blocks, 524,280 rows here
    const unsigned grid = mhd::adj::ic_blocks_across(dg(a->seg[0])) * ((a->ny + 4 + mhd::adj::IC_ROWS - 1) / mhd::adj::IC_ROWS);
    if (f64(a))
        mhd::adj::ic_grad_kernel<double><<<grid, 256, 0, st>>>(dg(*lam_next), dg(a->seg[0]), 0.0, 0.0, 1.0 / a->nx, 1.0 / a->ny, a->d_grad);
    else
        mhd::adj::ic_grad_kernel<float><<<grid, 256, 0, st>>>(dg(*lam_next), dg(a->seg[0]), 0.0, 0.0, 1.0 / a->nx, 1.0 / a->ny, a->d_grad);
    ACK(cudaGetLastError());
    mhd::count_launches(1);
    ACK(cudaMemcpy(grad, a->d_grad, sizeof(double) * 16, cudaMemcpyDeviceToHost));
    return MHD_OK;
}

}  // namespace

extern "C" {

int mhd_adjoint_create(int nx, int ny, int dtype, int limiter, double gamma, double cfl, double cr, int nsteps,
                       int checkpoint_every, mhd_adjoint** out) {
    if (!out || nx < 4 || ny < 4 || nsteps < 1 || (dtype != MHD_F64 && dtype != MHD_F32) ||
        (limiter != MHD_LIMITER_MINMOD && limiter != MHD_LIMITER_VANLEER) || !(gamma > 1.0) || !(cfl > 0.0) ||
        !(cr > 0.0))
        return aerr(MHD_ERR_ARG, "mhd_adjoint_create: invalid arguments");
    *out = nullptr;
    mhd_adjoint* a = new mhd_adjoint();
    a->nx = nx; a->ny = ny; a->dtype = dtype; a->limiter = limiter; a->gamma = gamma; a->cfl = cfl; a->cr = cr;
    a->nsteps = nsteps;
    a->b0 = 1.0 / std::sqrt(4.0 * M_PI);
    // the states' common layout, as mhd_grid_alloc pads it
    const size_t eb = dtype == MHD_F32 ? 4 : 8;
    const long long per = 256 / (long long)eb;
    mhd_grid shape{};
    shape.nx = nx; shape.ny = ny; shape.ng = 2; shape.dtype = dtype;
    shape.x_max = shape.y_max = 1.0;
    shape.pitch = (nx + 4LL + per - 1) / per * per;
    shape.plane = (shape.pitch * (ny + 4LL) + per - 1) / per * per;
    const size_t state = (size_t)shape.plane * MHD_NV * eb;
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    const double room = (double)free_b / 8.0 / (double)state;
    const int root = std::max(1, (int)std::lround(std::sqrt((double)nsteps)));
    a->every = checkpoint_every > 0 ? std::min(checkpoint_every, nsteps) : (2.0 * nsteps + 4.0 <= room ? nsteps : root);
    const int nck = (nsteps + a->every - 1) / a->every;
    a->ckpt.assign(nck > 1 ? nck : 0, shape);
    a->seg.assign(a->every + 1, shape);
    a->segT.assign(a->ckpt.size() + 2.0 * a->every + 4.0 <= room ? a->every : 1, shape);
    a->lamA = a->lamB = a->lamT = shape;
    std::vector<mhd_grid*> all;
    for (auto* v : {&a->ckpt, &a->seg, &a->segT})
        for (auto& g : *v) all.push_back(&g);
    all.insert(all.end(), {&a->lamA, &a->lamB, &a->lamT});
    int rc = MHD_OK;
    if (cudaMalloc(&a->slab, state * all.size()) != cudaSuccess) {
        a->slab = nullptr;
        cudaGetLastError();
        rc = aerr(MHD_ERR_NOMEM, "mhd_adjoint_create: states");
    } else {
        cudaMemset(a->slab, 0, state * all.size());
        for (size_t k = 0; k < all.size(); ++k) all[k]->data = static_cast<char*>(a->slab) + k * state;
    }
    if (!rc) rc = mhd_workspace_create(&a->seg[0], &a->ws);
    if (!rc) rc = mhd_set_gamma(a->ws, gamma);
    if (!rc) rc = mhd_set_limiter(a->ws, limiter);
    if (!rc) rc = mhd_set_cr(a->ws, cr);
    if (!rc && (cudaMalloc(&a->d_target, sizeof(double) * (size_t)nx * ny) != cudaSuccess ||
                cudaMalloc(&a->d_clock, sizeof(mhd::DevClock)) != cudaSuccess ||
                cudaMalloc(&a->d_acc, 2 * sizeof(unsigned long long)) != cudaSuccess ||
                cudaMemset(a->d_acc, 0, 2 * sizeof(unsigned long long)) != cudaSuccess ||
                cudaMalloc(&a->d_log, sizeof(double) * a->log_len()) != cudaSuccess ||
                cudaMalloc(&a->d_grad, sizeof(double) * 16) != cudaSuccess ||
                cudaMalloc(&a->d_idx, sizeof(int)) != cudaSuccess ||
                cudaMalloc(&a->d_sc, sizeof(double) * ((size_t)5 * nsteps + 1)) != cudaSuccess))
        rc = aerr(MHD_ERR_NOMEM, "mhd_adjoint_create: device buffers");
    if (rc) {
        mhd_adjoint_destroy(a);
        return rc;
    }
    *out = a;
    return MHD_OK;
}

int mhd_adjoint_set_solver(mhd_adjoint* a, int solver) {
    if (!a) return aerr(MHD_ERR_STATE, "mhd_adjoint_set_solver: null adjoint");
    if (solver != MHD_HLL && solver != MHD_HLLD)
        return aerr(MHD_ERR_ARG, "mhd_adjoint_set_solver: the adjoint differentiates HLL or HLLD");
    a->solver = solver;
    return MHD_OK;
}

int mhd_adjoint_destroy(mhd_adjoint* a) {
    if (!a) return MHD_OK;
    if (a->slab) cudaFree(a->slab);
    if (a->ws) mhd_workspace_destroy(a->ws);
    if (a->d_target) cudaFree(a->d_target);
    if (a->d_clock) cudaFree(a->d_clock);
    if (a->d_acc) cudaFree(a->d_acc);
    if (a->d_log) cudaFree(a->d_log);
    if (a->d_grad) cudaFree(a->d_grad);
    if (a->d_idx) cudaFree(a->d_idx);
    if (a->d_sc) cudaFree(a->d_sc);
    delete a;
    return MHD_OK;
}

int mhd_adjoint_set_target(mhd_adjoint* a, const double* rho_target) {
    if (!a || !rho_target) return aerr(MHD_ERR_ARG, "mhd_adjoint_set_target: null argument");
    ACK(cudaMemcpy(a->d_target, rho_target, sizeof(double) * (size_t)a->nx * a->ny, cudaMemcpyHostToDevice));
    a->have_target = true;
    return MHD_OK;
}

int mhd_adjoint_forward(mhd_adjoint* a, const double* amp16, double* J, double* rho_final) {
    mhd::NvtxRange nvtx_range("mhd_adjoint_forward");
    if (!a) return aerr(MHD_ERR_STATE, "mhd_adjoint_forward: null handle");
    return forward(a, amp16, J, rho_final, nullptr);
}

int mhd_adjoint_gradient(mhd_adjoint* a, const double* amp16, double* J, double* grad16) {
    mhd::NvtxRange nvtx_range("mhd_adjoint_gradient");
    if (!a || !grad16) return aerr(MHD_ERR_ARG, "mhd_adjoint_gradient: null argument");
    if (!a->have_target) return aerr(MHD_ERR_STATE, "mhd_adjoint_gradient: no target set");
    return gradient(a, amp16, J, grad16);
}

}  // extern "C"
