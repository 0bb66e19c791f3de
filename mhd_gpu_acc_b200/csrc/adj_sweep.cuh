// adj_sweep.cuh -- one adjoint sweep in one launch: lamIn = (sweep)^T lamOut,
// with the fold of ghost cotangents onto their periodic sources and, for the
// y-sweep, the psi damping's reverse applied as lamOut is read.
//
// One lane owns one cell of a line along the sweep and exchanges neighbour
// values by shuffles; a warp covers 32 cells of which 26 are its own (a cell's
// cotangent depends on faces and reconstructions up to three cells away).
// x lines are rows, read as they lie.  y lines are columns: a CTA stages a
// block of 32 rows by eight columns through shared memory, so that global
// memory is read and written in 32-byte (FP64: 64-byte) runs, and each warp
// walks one of the columns (row stride 9, so lanes on 32 rows meet 32 banks).
#pragma once

#include "adj_launch.h"
#include "adj_pair.cuh"
#include "sweep.cuh"

namespace mhd {
namespace adj {

constexpr int AT = 26;      // outputs per warp: 32 lanes minus a 3-cell halo on each side
constexpr int AWARPS = 8;   // warps per y CTA: the columns of its block
constexpr int AXWARPS = 4;  // warps per x CTA
constexpr int APITCH = AWARPS + 1;

template <typename R>
__device__ __forceinline__ R value(const DevGrid& g, int f, int i, int j) {
    return static_cast<const R*>(g.data)[f * g.plane + g.idx(i, j)];
}

// The sum of lam over the ghost cells that copy interior cell (i, j) across the
// periodic side along FD (0: columns, 1: rows).
template <typename R, int FD>
__device__ __forceinline__ R ghosts(const DevGrid& lam, int f, int i, int j) {
    const int c = FD == 0 ? i : j, n = FD == 0 ? lam.nx : lam.ny;
    R v = R(0);
    if (c < 2 * lam.ng) v = FD == 0 ? value<R>(lam, f, i + n, j) : value<R>(lam, f, i, j + n);
    if (c >= n) v += FD == 0 ? value<R>(lam, f, i - n, j) : value<R>(lam, f, i, j - n);
    return v;
}

// One cell of a line (lane), all lanes of the warp: its conserved state Uc and
// the cotangent lT of its updated value (0 outside the interior) -> the
// cotangent lU of Uc; adds to the sums of dt/d and c_h for owned work.
template <typename R, int LIM, int SOLVER>
__device__ __forceinline__ void adj_cell(const R* Uc, const R* lT, int p, int lo, int hi, bool own, R dtd, R ch, R g,
                                         R gm1, R igm1, R* lU, R& ldtd, R& lch) {
    const int lane = threadIdx.x & 31;
    const R gr = g * igm1;
    // c2p with the correctly rounded reciprocal in either precision: the slopes'
    // signs, which a last bit of W can flip where they are at rounding, then do
    // not depend on the build's flags (FP32 gradients moved by 1e-5 otherwise)
    const R ir = rcp(Uc[RHO]);
    R W[NV];
    c2p_ir(Uc, ir, g, W);
    R Wm[NV], Wp[NV];
    shfl_up_n<NV>(W, Wm, 1);
    shfl_down_n<NV>(W, Wp, 1);
    const bool do_recon = lane >= 1 && lane <= 30 && p >= lo - 1 && p <= hi;
    const bool do_face = lane >= 1 && lane <= 29 && p >= lo - 1 && p <= hi - 1;
    Recon<R> rc;
    Pr<R> S[NV], V[NV], ir2;
    if (do_recon) {
        recon2<LIM>(Wm, W, Wp, dtd, ch, gm1, igm1, rc, S, V, ir2);
    } else {
        ir2 = dup(R(1));
#pragma unroll
        for (int k = 0; k < NV; ++k) S[k] = V[k] = dup(R(0));
    }
    // face (p | p + 1): this cell's right state and the next one's left state
    Pr<R> U2[NV], W2[NV], irf, lF2[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        U2[k] = {S[k].y, __shfl_down_sync(FULL, S[k].x, 1)};
        const bool same = k == RHO || k == BX || k == BY || k == BZ || k == PSI;  // in U and in W
        if (same) W2[k] = U2[k];
        else W2[k] = {V[k].y, __shfl_down_sync(FULL, V[k].x, 1)};
        lF2[k] = dup(R(0));
    }
    irf = {ir2.y, __shfl_down_sync(FULL, ir2.x, 1)};
    R d[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) d[k] = __shfl_down_sync(FULL, lT[k], 1) - lT[k];
    if (do_face) {
        R sd = R(0), sc = R(0);
        if (SOLVER == HLL) hll_pair(U2, W2, irf, ch, g, gm1, gr, dtd, d, lF2, sd, sc);
        else hlld_pair(U2, ch, g, dtd, d, lF2, sd, sc);
        if (own) { ldtd += sd; lch += sc; }
    }
    Pr<R> lS[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) lS[k] = {__shfl_up_sync(FULL, lF2[k].y, 1), lF2[k].x};
    R lWm[NV], lWc[NV], lWp[NV];
    zero(lWm);
    zero(lWc);
    zero(lWp);
    // the neighbours' W again (18 shuffles) rather than held across the face, which
    // needs the registers
    shfl_up_n<NV>(W, Wm, 1);
    shfl_down_n<NV>(W, Wp, 1);
    if (do_recon) {
        R sd = R(0), sc = R(0);
        recon_adj2<LIM>(Wm, W, Wp, rc, dtd, ch, igm1, gr, lS, lWm, lWc, lWp, sd, sc);
        if (own) { ldtd += sd; lch += sc; }
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        // the W_{p+1} role in cell p - 1 and the W_{p-1} role in cell p + 1
        lWc[k] += __shfl_up_sync(FULL, lWp[k], 1) + __shfl_down_sync(FULL, lWm[k], 1);
        lU[k] = lT[k];  // T_p = U_p - dtd (F_{p+1/2} - F_{p-1/2})
    }
    const R q = gm1 * lWc[PP], u = W[PU], v = W[PV], w = W[PW];
    lU[EN] += q;
    lU[MX] += lWc[PU] * ir - q * u;
    lU[MY] += lWc[PV] * ir - q * v;
    lU[MZ] += lWc[PW] * ir - q * w;
    lU[RHO] += lWc[RHO] - (lWc[PU] * u + lWc[PV] * v + lWc[PW] * w) * ir + q * R(0.5) * (u * u + v * v + w * w);
    lU[BX] += lWc[BX] - q * W[BX];
    lU[BY] += lWc[BY] - q * W[BY];
    lU[BZ] += lWc[BZ] - q * W[BZ];
    lU[PSI] += lWc[PSI];
}

// Sums of a CTA of WARPS warps into acc[0..N): one atomic per value and CTA.
template <int N, int WARPS>
__device__ __forceinline__ void block_add(const double* v, double* acc) {
    __shared__ double part[N][WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        double s = v[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) part[q][warp] = s;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) s += part[threadIdx.x][w];
        if (s != 0.0) atomicAdd(acc + threadIdx.x, s);
    }
}

// x: rows, one tile of a row per warp; lamOut's ghost rows folded on read.
template <typename R, int LIM, int SOLVER>
__global__ void __launch_bounds__(32 * AXWARPS, AdjShape<R, SOLVER>::kXBlocks)
    adj_x_kernel(DevGrid U, DevGrid lamOut, DevGrid lamIn, R g, R gm1, R igm1, R dtd, R ch, double* acc) {
    const int lane = threadIdx.x & 31;
    const long long warp = (long long)blockIdx.x * AXWARPS + (threadIdx.x >> 5);
    const int ng = U.ng, lo = ng, hi = ng + U.nx;
    const int ntile = (U.nx + 4 + AT - 1) / AT;
    const int row = (int)(warp / ntile), tile = (int)(warp - (long long)row * ntile);
    R ldtd = R(0), lch = R(0);
    if (row < U.ny) {
        const int j = ng + row, p = ng - 2 + tile * AT + lane - 3;
        R Uc[NV], lT[NV], lU[NV];
        zero(Uc);
        zero(lT);
        Uc[RHO] = R(1);
        if (p >= 0 && p < U.tnx()) load_cell(U, p, j, Uc);
        if (p >= lo && p < hi) {
#pragma unroll
            for (int k = 0; k < NV; ++k) lT[k] = value<R>(lamOut, k, p, j) + ghosts<R, 1>(lamOut, k, p, j);
        }
        const bool own = lane >= 3 && lane <= 28;
        adj_cell<R, LIM, SOLVER>(Uc, lT, p, lo, hi, own, dtd, ch, g, gm1, igm1, lU, ldtd, lch);
        if (own && p >= lo - 2 && p < hi + 2) store_cell(lamIn, p, j, lU);
    }
    const double v[2] = {(double)ldtd, (double)lch};
    block_add<2, AXWARPS>(v, acc);
}

// y: columns, eight per CTA; lamOut's ghost columns folded and its interior psi
// cotangent scaled by the damping factor f on read, sum(lambda_psi psi_next / f)
// to acc[2].
template <typename R, int LIM, int SOLVER>
__global__ void __launch_bounds__(32 * AWARPS, AdjShape<R, SOLVER>::kYBlocks)
    adj_y_kernel(DevGrid U, DevGrid lamOut, DevGrid lamIn, DevGrid Unext, R g, R gm1, R igm1, R dtd, R ch, double f,
                 double* acc) {
    extern __shared__ __align__(16) unsigned char ay_smem[];
    R* const sU = reinterpret_cast<R*>(ay_smem);          // [9][32][APITCH]
    R* const sL = sU + NV * 32 * APITCH;                   // [9][32][APITCH], then the results
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ng = U.ng, lo = ng, hi = ng + U.ny;
    const unsigned across = (U.nx + AWARPS - 1) / AWARPS;  // blocks side by side (one-dimensional launch: any number of rows)
    const int i0 = ng + blockIdx.x % across * AWARPS, j0 = ng - 2 + blockIdx.x / across * AT - 3;
    double sf = 0.0;
    // thread t: column t % 8, rows t / 8 (all fields of a cell by one thread)
    {
        const int c = threadIdx.x % AWARPS, r = threadIdx.x / AWARPS, i = i0 + c, j = j0 + r;
        const bool col = i < ng + U.nx;
        const bool in = col && j >= 0 && j < U.tny(), interior = col && j >= lo && j < hi;
        R u[NV], l[NV];
        zero(u);
        zero(l);
        u[RHO] = R(1);
        if (in) load_cell(U, i, j, u);
        if (interior) {
#pragma unroll
            for (int k = 0; k < NV; ++k) l[k] = value<R>(lamOut, k, i, j);
            if (r >= 3 && r <= 28) sf = (double)l[PSI] * (double)value<R>(Unext, PSI, i, j) / f;
            l[PSI] *= (R)f;  // the step damps psi in the interior after the ghosts have copied it
#pragma unroll
            for (int k = 0; k < NV; ++k) l[k] += ghosts<R, 0>(lamOut, k, i, j);
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            sU[(k * 32 + r) * APITCH + c] = u[k];
            sL[(k * 32 + r) * APITCH + c] = l[k];
        }
    }
    __syncthreads();
    R ldtd = R(0), lch = R(0);
    {
        R Uc[NV], lT[NV], lU[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            Uc[k] = sU[(k * 32 + lane) * APITCH + warp];
            lT[k] = sL[(k * 32 + lane) * APITCH + warp];
        }
        rot(Uc);
        rot(lT);
        const bool own = lane >= 3 && lane <= 28;
        const int p = i0 + warp < ng + U.nx ? j0 + lane : -8;  // no work past the last column
        adj_cell<R, LIM, SOLVER>(Uc, lT, p, lo, hi, own, dtd, ch, g, gm1, igm1, lU, ldtd, lch);
        rot(lU);
#pragma unroll
        for (int k = 0; k < NV; ++k) sL[(k * 32 + lane) * APITCH + warp] = lU[k];
    }
    __syncthreads();
    {
        const int c = threadIdx.x % AWARPS, r = threadIdx.x / AWARPS, i = i0 + c, j = j0 + r;
        if (i < ng + U.nx && r >= 3 && r <= 28 && j >= lo - 2 && j < hi + 2) {
            R l[NV];
#pragma unroll
            for (int k = 0; k < NV; ++k) l[k] = sL[(k * 32 + r) * APITCH + c];
            store_cell(lamIn, i, j, l);
        }
    }
    const double v[3] = {(double)ldtd, (double)lch, sf};
    block_add<3, AWARPS>(v, acc);
}

template <typename R, int LIM, int SOLVER>
cudaError_t launch_one(const AdjSweepArgs& a, cudaStream_t st) {
    const R g = (R)a.gamma, gm1 = (R)(a.gamma - 1.0), igm1 = (R)(1.0 / (a.gamma - 1.0));
    if (a.dir == 0) {
        const long long warps = (long long)a.U.ny * ((a.U.nx + 4 + AT - 1) / AT);
        adj_x_kernel<R, LIM, SOLVER><<<(unsigned)((warps + AXWARPS - 1) / AXWARPS), 32 * AXWARPS, 0, st>>>(
            a.U, a.lamOut, a.lamIn, g, gm1, igm1, (R)a.dtd, (R)a.ch, a.acc);
    } else {
        constexpr int bytes = 2 * NV * 32 * APITCH * (int)sizeof(R);
        static_assert(bytes <= 48 * 1024, "the y block's stage needs an opt-in");
        const unsigned grid = (a.U.nx + AWARPS - 1) / AWARPS * ((a.U.ny + 4 + AT - 1) / AT);
        adj_y_kernel<R, LIM, SOLVER><<<grid, 32 * AWARPS, bytes, st>>>(a.U, a.lamOut, a.lamIn, a.Unext, g, gm1, igm1,
                                                                      (R)a.dtd, (R)a.ch, a.damp, a.acc);
    }
    return cudaGetLastError();
}

template <typename R>
cudaError_t launch_adj(const AdjSweepArgs& a, cudaStream_t st) {
    if (a.solver == HLLD)
        return a.limiter == VANLEER ? launch_one<R, VANLEER, HLLD>(a, st) : launch_one<R, MINMOD, HLLD>(a, st);
    return a.limiter == VANLEER ? launch_one<R, VANLEER, HLL>(a, st) : launch_one<R, MINMOD, HLL>(a, st);
}

}  // namespace adj
}  // namespace mhd
