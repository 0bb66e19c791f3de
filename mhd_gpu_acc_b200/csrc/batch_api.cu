// batch_api.cu -- C ABI of the batched engine (mhd_batch_*) and its autotuner.
//
// A batch owns, per instance, the state U and the x-swept state T (padded slabs
// as mhd_grid_alloc makes them), a device clock, and one shared instance table
// and work lists (batch.cuh).  mhd_batch_run starts every clock from the CFL
// maximum of its instance (one launch for all) and replays a CUDA graph of two
// steps (four launches) until max_steps steps or every instance's t_end.
//
// Autotuner (mhd_batch_tune): the x-sweep phase maps U -> T and the y-sweep
// phase maps T -> U without touching the clock slots they read, so each phase
// can be launched repeatedly on unchanged input.  The tuner times every x
// candidate (rows per warp x persistent CTAs) and then every y candidate
// (segment length x persistent CTAs) with CUDA events, keeping the fastest of
// each.  The default values are among the candidates and stand for the shape by the
// size of the batch.  The instances end one step ahead of where they started.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <exception>
#include <string>
#include <vector>

#include "../../include/mhd_b200.h"
#include "batch.cuh"
#include "launch.h"

namespace mhd {
int report_error(int code, const char* msg);
}

namespace {

int berr(int code, const char* msg) { return mhd::report_error(code, msg); }

#define BCK(call)                                                             \
    do {                                                                      \
        cudaError_t e_ = (call);                                              \
        if (e_ != cudaSuccess) return berr(MHD_ERR_CUDA, cudaGetErrorString(e_)); \
    } while (0)

}  // namespace

struct mhd_batch {
    int n = 0, dtype = MHD_F32, solver = MHD_HLLD, limiter = MHD_LIMITER_VANLEER, nsm = 148;
    std::vector<mhd_instance_desc> desc;
    std::vector<mhd_grid> U, T;
    std::vector<double> ch;  // per-instance c_h carried between runs (floor of the next CFL maximum)
    std::vector<mhd::BatchInst> host_inst;  // 2 n: step parity 0, then 1
    mhd::BatchInst* d_inst = nullptr;
    // work lists of the x phase, the y phase and the CFL maximum: segments (up to
    // 2 n each for x and y, n for the maximum) and the segment of every unit
    mhd::BatchSeg* d_seg = nullptr;
    int* d_units = nullptr;
    size_t units_cap = 0;
    mhd::BatchList lists[3] = {};
    double* d_ch = nullptr;
    mhd::DevClock* d_clock = nullptr;
    cudaStream_t stream = nullptr;
    mhd_batch_tuning tune{mhd::kDefaultBatchXRpw, mhd::kDefaultYSeg, 0, 0};
    cudaGraphExec_t graph = nullptr;
    long long cells = 0;
};

namespace {

// Candidate launch shapes the autotuner times (mhd_batch_tune), exported by
// mhd_batch_tune_candidates.
const int kTuneXrpw[] = {2, 4, 8, 16};             // x-sweep rows per warp
const int kTuneYseg[] = {16, 24, 32, 48, 64, 128};  // y-sweep segment rows
const int kTuneCtasPerSm[] = {2, 3, 4};             // persistent CTAs per SM, both phases

// A phase at its default tuning takes its lengths by the size of the batch and one
// CTA per unit; any other tuning is taken as it is.  So the four values say all
// there is to a shape: those that get_tuning or the tuner give make the same one
// when they are set, on this batch or another.
int default_ctas(const mhd_batch* b) { return 3 * b->nsm; }
bool by_size_x(const mhd_batch* b) { return b->tune.xrpw == mhd::kDefaultBatchXRpw && b->tune.ctas_x == default_ctas(b); }
bool by_size_y(const mhd_batch* b) { return b->tune.yseg == mhd::kDefaultYSeg && b->tune.ctas_y == default_ctas(b); }

cudaError_t phase(mhd_batch* b, int parity, int which, cudaStream_t st) {
    const int ctas = which == 1 ? (by_size_x(b) ? 0 : b->tune.ctas_x) : which == 2 ? (by_size_y(b) ? 0 : b->tune.ctas_y) : 0;
    const mhd::BatchList& list = b->lists[which > 0 ? which - 1 : 0];
    return b->dtype == MHD_F64 ? mhd::launch_batch_f64(b->d_inst, list, b->d_ch, b->n, parity, which, b->solver, b->limiter, ctas, st)
                               : mhd::launch_batch_f32(b->d_inst, list, b->d_ch, b->n, parity, which, b->solver, b->limiter, ctas, st);
}

// Work lists for the current shape; uploads the tables and drops the graph.  Without
// memory for a longer table the lists, and the graph that holds their addresses,
// stay as they were.
int build_worklist(mhd_batch* b) try {
    const int n = b->n;
    long long x_work = 0, y_work = 0;
    for (int i = 0; i < n; ++i) {
        const mhd_instance_desc& d = b->desc[i];
        x_work += (long long)d.ny * ((d.nx + 31) / 32);
        y_work += (long long)d.ny * mhd::y_strips(b->host_inst[i].U);
    }
    mhd::TaskLen tx{}, ty{};
    if (b->dtype == MHD_F64) mhd::batch_task_lens_f64(x_work, y_work, tx, ty);
    else mhd::batch_task_lens_f32(x_work, y_work, tx, ty);
    static_assert(mhd::BX_WARPS == mhd::YS_WARPS, "a unit is four tasks in both phases");
    std::vector<mhd::BatchSeg> segs;
    std::vector<int> units;
    size_t seg0[4] = {}, unit0[4] = {};
    for (int l = 0; l < 3; ++l) {
        for (int i = 0; i < n; ++i) {
            const int nx = b->desc[i].nx, ny = b->desc[i].ny, strips = mhd::y_strips(b->host_inst[i].U);
            if (l == 2) {
                segs.push_back({i, 0, 0, 0, 0, 0, 0, 0, 0});
                continue;
            }
            const bool by_size = l == 0 ? by_size_x(b) : by_size_y(b);
            const mhd::TaskLen& t = l == 0 ? tx : ty;
            const int cut = by_size && !t.one_wave ? ny - ny / 8 : ny;  // rows from here on in shorter tasks
            for (int p = 0; p < 2; ++p) {
                const int r0 = p == 0 ? 0 : cut, r1 = p == 0 ? cut : ny, most = p == 0 ? t.len : (t.len + 2) / 3;
                if (r0 == r1) continue;
                if (l == 0) {
                    int len = mhd::x_seg_len(4 * b->tune.xrpw);
                    if (by_size) {  // equal segments, the fewest of `most` chunks
                        const int k = mhd::x_seg_len(most), parts = (nx + k - 1) / k;
                        len = mhd::x_seg_len(((nx + parts - 1) / parts + 4 + 31) / 32);
                    }
                    segs.push_back({i, 0, nx, len, (nx + len - 1) / len, r0, r1 - r0, 0, 0});
                } else {
                    int len = b->tune.yseg;
                    if (by_size) {
                        const int parts = (r1 - r0 + most - 1) / most;
                        len = (r1 - r0 + parts - 1) / parts;
                    }
                    segs.push_back({i, r0, r1, len, (r1 - r0 + len - 1) / len, 0, strips, 0, 0});
                }
            }
        }
        const auto begin = segs.begin() + seg0[l];
        if (l < 2) std::stable_sort(begin, segs.end(), [](const mhd::BatchSeg& p, const mhd::BatchSeg& q) { return p.len > q.len; });
        std::vector<char> led(n, 0);
        for (auto s = begin; s != segs.end(); ++s) {
            const long long count = l < 2 ? ((long long)s->n * s->width + mhd::YS_WARPS - 1) / mhd::YS_WARPS
                                          : mhd::max_units(b->host_inst[s->inst].U);
            s->lead = !led[s->inst];
            led[s->inst] = 1;
            s->unit = (int)(units.size() - unit0[l]);
            if ((long long)s->unit + count > 0x7fffffff) return berr(MHD_ERR_ARG, "batch: too many work units");
            units.insert(units.end(), (size_t)count, (int)(s - begin));
        }
        seg0[l + 1] = segs.size();
        unit0[l + 1] = units.size();
    }
    for (int i = 0; i < n; ++i) {
        b->host_inst[n + i] = b->host_inst[i];
        b->host_inst[n + i].P.parity = 1;
    }
    int* d_units = b->d_units;
    if (units.size() > b->units_cap && cudaMalloc(&d_units, sizeof(int) * units.size()) != cudaSuccess) {
        cudaGetLastError();
        return berr(MHD_ERR_NOMEM, "batch: work list");
    }
    if (b->graph) {
        cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    }
    if (d_units != b->d_units) {
        if (b->d_units) cudaFree(b->d_units);  // waits for launches that read it
        b->d_units = d_units;
        b->units_cap = units.size();
    }
    for (auto& l : b->lists) l = {};  // no units until the tables are there
    BCK(cudaMemcpyAsync(b->d_inst, b->host_inst.data(), sizeof(mhd::BatchInst) * b->host_inst.size(),
                        cudaMemcpyHostToDevice, b->stream));
    BCK(cudaMemcpyAsync(b->d_seg, segs.data(), sizeof(mhd::BatchSeg) * segs.size(), cudaMemcpyHostToDevice, b->stream));
    BCK(cudaMemcpyAsync(b->d_units, units.data(), sizeof(int) * units.size(), cudaMemcpyHostToDevice, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    for (int l = 0; l < 3; ++l)
        b->lists[l] = {b->d_seg + seg0[l], b->d_units + unit0[l], (int)(unit0[l + 1] - unit0[l])};
    return MHD_OK;
} catch (const std::exception& e) {
    return berr(MHD_ERR_NOMEM, e.what());
}

// Every clock from its instance's CFL maximum (floored by the carried c_h).
int start_clocks(mhd_batch* b) {
    BCK(cudaMemsetAsync(b->d_clock, 0, sizeof(mhd::DevClock) * b->n, b->stream));  // t = 0, no steps, running
    BCK(cudaMemcpyAsync(b->d_ch, b->ch.data(), sizeof(double) * b->n, cudaMemcpyHostToDevice, b->stream));
    BCK(phase(b, 0, 3, b->stream));
    return MHD_OK;
}

void fill_ctas(mhd_batch* b) {
    if (b->tune.ctas_x <= 0) b->tune.ctas_x = default_ctas(b);
    if (b->tune.ctas_y <= 0) b->tune.ctas_y = default_ctas(b);
}

}  // namespace

extern "C" {

int mhd_batch_create(const mhd_instance_desc* desc, int n, int dtype, int solver, int limiter, mhd_batch** out) {
    if (!out || !desc || n < 1) return berr(MHD_ERR_ARG, "mhd_batch_create: need n >= 1 descriptors and an output");
    *out = nullptr;
    if (dtype != MHD_F64 && dtype != MHD_F32) return berr(MHD_ERR_ARG, "mhd_batch_create: bad dtype");
    if (solver < MHD_HLL || solver > MHD_FORCE) return berr(MHD_ERR_ARG, "mhd_batch_create: bad solver");
    if (limiter != MHD_LIMITER_MINMOD && limiter != MHD_LIMITER_VANLEER)
        return berr(MHD_ERR_ARG, "mhd_batch_create: bad limiter");
    for (int i = 0; i < n; ++i) {
        const mhd_instance_desc& d = desc[i];
        if (d.ng < 2 || d.ng > MHD_MAX_NG || d.nx < d.ng || d.ny < d.ng || !(d.gamma > 1.0) || !(d.cfl > 0.0) ||
            !(d.cr > 0.0) || !(d.t_end > 0.0) || !std::isfinite(d.t_end) || !(d.x_max > d.x_min) ||
            !(d.y_max > d.y_min))
            return berr(MHD_ERR_ARG, "mhd_batch_create: invalid instance descriptor");
        for (int k = 0; k < 4; ++k)
            if (d.bc[k] < MHD_BC_PERIODIC || d.bc[k] > MHD_BC_REFLECTING)
                return berr(MHD_ERR_ARG, "mhd_batch_create: boundary types are periodic, transmissive or reflecting");
    }
    mhd_batch* b = new mhd_batch();
    b->n = n;
    b->dtype = dtype;
    b->solver = solver;
    b->limiter = limiter;
    b->desc.assign(desc, desc + n);
    b->U.assign(n, mhd_grid{});
    b->T.assign(n, mhd_grid{});
    b->ch.assign(n, 0.0);
    b->host_inst.assign(2 * (size_t)n, mhd::BatchInst{});
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&b->nsm, cudaDevAttrMultiProcessorCount, dev);
    if (b->nsm <= 0) b->nsm = 148;
    fill_ctas(b);
    int rc = MHD_OK;
    for (int i = 0; i < n && rc == MHD_OK; ++i) {
        const mhd_instance_desc& d = desc[i];
        rc = mhd_grid_alloc(&b->U[i], d.nx, d.ny, d.ng, dtype, d.x_min, d.x_max, d.y_min, d.y_max);
        if (!rc) rc = mhd_grid_alloc(&b->T[i], d.nx, d.ny, d.ng, dtype, d.x_min, d.x_max, d.y_min, d.y_max);
        b->cells += (long long)d.nx * d.ny;
    }
    if (!rc && (cudaMalloc(&b->d_inst, sizeof(mhd::BatchInst) * 2 * n) != cudaSuccess ||
                cudaMalloc(&b->d_seg, sizeof(mhd::BatchSeg) * 5 * n) != cudaSuccess ||
                cudaMalloc(&b->d_ch, sizeof(double) * n) != cudaSuccess ||
                cudaMalloc(&b->d_clock, sizeof(mhd::DevClock) * n) != cudaSuccess))
        rc = berr(MHD_ERR_NOMEM, "mhd_batch_create: device tables");
    if (rc) {
        mhd_batch_destroy(b);
        return rc;
    }
    for (int i = 0; i < n; ++i) {
        const mhd_instance_desc& d = desc[i];
        mhd::BatchInst& I = b->host_inst[i];
        I.U = mhd::DevGrid{b->U[i].data, b->U[i].pitch, b->U[i].plane, d.nx, d.ny, d.ng, 0};
        I.T = b->T[i].data;
        mhd::StepParams& P = I.P;
        std::memset(&P, 0, sizeof P);
        P.gamma = d.gamma;
        P.cr = d.cr;
        P.cfl = d.cfl;
        P.dx = (d.x_max - d.x_min) / d.nx;
        P.dy = (d.y_max - d.y_min) / d.ny;
        P.dmin = (P.dy < P.dx) ? P.dy : P.dx;
        P.t_end = d.t_end;
        P.dt_min = 1.0e-8 * d.t_end;
        P.clock = b->d_clock + i;
        P.solver = solver;
        P.limiter = limiter;
        for (int k = 0; k < 4; ++k) P.bc[k] = d.bc[k];
        P.any_dirichlet = 0;
        P.accumulate = 1;
    }
    rc = build_worklist(b);
    if (rc) {
        mhd_batch_destroy(b);
        return rc;
    }
    *out = b;
    return MHD_OK;
}

int mhd_batch_destroy(mhd_batch* b) {
    if (!b) return MHD_OK;
    if (b->graph) cudaGraphExecDestroy(b->graph);
    for (auto& g : b->U) mhd_grid_free(&g);
    for (auto& g : b->T) mhd_grid_free(&g);
    if (b->d_inst) cudaFree(b->d_inst);
    if (b->d_units) cudaFree(b->d_units);
    if (b->d_clock) cudaFree(b->d_clock);
    if (b->d_seg) cudaFree(b->d_seg);
    if (b->d_ch) cudaFree(b->d_ch);
    delete b;
    return MHD_OK;
}

int mhd_batch_set_stream(mhd_batch* b, void* stream) {
    if (!b) return berr(MHD_ERR_STATE, "mhd_batch_set_stream: null batch");
    if (b->graph) {
        cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    }
    b->stream = static_cast<cudaStream_t>(stream);
    return MHD_OK;
}

int mhd_batch_grid(const mhd_batch* b, int i, mhd_grid* out) {
    if (!b || !out || i < 0 || i >= b->n) return berr(MHD_ERR_ARG, "mhd_batch_grid: bad instance");
    *out = b->U[i];
    return MHD_OK;
}

int mhd_batch_cells(const mhd_batch* b, long long* cells) {
    if (!b || !cells) return berr(MHD_ERR_ARG, "mhd_batch_cells: null argument");
    *cells = b->cells;
    return MHD_OK;
}

int mhd_batch_get_tuning(const mhd_batch* b, mhd_batch_tuning* t) {
    if (!b || !t) return berr(MHD_ERR_ARG, "mhd_batch_get_tuning: null argument");
    *t = b->tune;
    return MHD_OK;
}

int mhd_batch_set_tuning(mhd_batch* b, const mhd_batch_tuning* t) {
    if (!b || !t) return berr(MHD_ERR_ARG, "mhd_batch_set_tuning: null argument");
    if (t->xrpw < 1 || t->xrpw > 64 || t->yseg < 4 || t->yseg > 4096 || t->ctas_x < 0 || t->ctas_y < 0)
        return berr(MHD_ERR_ARG, "mhd_batch_set_tuning: out of range");
    const mhd_batch_tuning tune = b->tune;
    b->tune = *t;
    fill_ctas(b);
    const int rc = build_worklist(b);
    if (rc) b->tune = tune;  // the lists are still the former ones
    return rc;
}

int mhd_batch_run(mhd_batch* b, int max_steps, mhd_run_info* info) {
    mhd::NvtxRange nvtx_range("mhd_batch_run");
    if (!b) return berr(MHD_ERR_STATE, "mhd_batch_run: null batch");
    if (max_steps < 1) return berr(MHD_ERR_ARG, "mhd_batch_run: max_steps must be >= 1");
    int rc = start_clocks(b);
    if (rc) return rc;
    if (!b->graph) {
        cudaStream_t cap = b->stream;
        bool own = false;
        if (!cap) {
            BCK(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
            own = true;
        }
        cudaGraph_t gr = nullptr;
        BCK(phase(b, 0, 0, cap));  // kernel attribute set-up, outside the capture
        BCK(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
        cudaError_t e = cudaSuccess;
        for (int p = 0; p < 2 && e == cudaSuccess; ++p) {
            e = phase(b, p, 1, cap);
            if (e == cudaSuccess) e = phase(b, p, 2, cap);
        }
        const cudaError_t e2 = cudaStreamEndCapture(cap, &gr);
        if (own) cudaStreamDestroy(cap);
        if (e != cudaSuccess || e2 != cudaSuccess) {
            if (gr) cudaGraphDestroy(gr);
            return berr(MHD_ERR_CUDA, "mhd_batch_run: graph capture failed");
        }
        const cudaError_t e3 = cudaGraphInstantiate(&b->graph, gr, 0);
        cudaGraphDestroy(gr);
        if (e3 != cudaSuccess) {
            b->graph = nullptr;
            return berr(MHD_ERR_CUDA, "mhd_batch_run: graph instantiation failed");
        }
    }
    for (int p = 0; p < max_steps / 2; ++p) BCK(cudaGraphLaunch(b->graph, b->stream));
    if (max_steps & 1) {
        BCK(phase(b, 0, 1, b->stream));
        BCK(phase(b, 0, 2, b->stream));
    }
    std::vector<mhd::DevClock> hc(b->n);
    BCK(cudaMemcpyAsync(hc.data(), b->d_clock, sizeof(mhd::DevClock) * b->n, cudaMemcpyDeviceToHost, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    int worst = MHD_OK;
    for (int i = 0; i < b->n; ++i) {
        const mhd::DevClock& c = hc[i];
        if (c.steps > 0) b->ch[i] = c.last_ch;
        int code = MHD_OK;
        if (c.status == mhd::CLK_NO_SPEED) code = MHD_ERR_NO_SPEED;
        else if (c.status == mhd::CLK_BAD_DT) code = MHD_ERR_BAD_DT;
        else if (c.status == mhd::CLK_TINY_DT) code = MHD_ERR_TINY_DT;
        if (code != MHD_OK) worst = code;
        if (info) {
            info[i].t = c.t[c.steps & 1];
            info[i].last_dt = c.last_dt;
            info[i].ch = b->ch[i];
            info[i].steps = c.steps;
            info[i].status = code;
            info[i].fallbacks = c.flux_fallbacks;
            info[i].pad_ = 0;
        }
    }
    if (worst != MHD_OK) return berr(worst, "mhd_batch_run: an instance's step loop stopped (see its info.status)");
    return MHD_OK;
}

int mhd_batch_tune_candidates(int which, int* out, int cap) {
    const int* src = nullptr;
    int n = 0;
    switch (which) {
        case 0: src = kTuneXrpw; n = (int)(sizeof(kTuneXrpw) / sizeof(int)); break;
        case 1: src = kTuneYseg; n = (int)(sizeof(kTuneYseg) / sizeof(int)); break;
        case 2: src = kTuneCtasPerSm; n = (int)(sizeof(kTuneCtasPerSm) / sizeof(int)); break;
        default: return berr(MHD_ERR_ARG, "mhd_batch_tune_candidates: which must be 0, 1 or 2");
    }
    for (int k = 0; out && k < n && k < cap; ++k) out[k] = src[k];
    return n;
}

// The tuner's search between its events: leaves the lists of the best shape.
static int tune_shapes(mhd_batch* b, int reps, cudaEvent_t e0, cudaEvent_t e1) {
    int rc = start_clocks(b);
    if (rc) return rc;
    mhd_batch_tuning best = b->tune;
    const auto& xr = kTuneXrpw;
    const auto& xc = kTuneCtasPerSm;
    const auto& ys = kTuneYseg;
    const auto& yc = kTuneCtasPerSm;
    auto time_phase = [&](int which, float* ms) -> int {
        BCK(phase(b, 0, which, b->stream));  // warm
        BCK(cudaEventRecord(e0, b->stream));
        for (int r = 0; r < reps; ++r) BCK(phase(b, 0, which, b->stream));
        BCK(cudaEventRecord(e1, b->stream));
        BCK(cudaEventSynchronize(e1));
        BCK(cudaEventElapsedTime(ms, e0, e1));
        return MHD_OK;
    };
    float best_ms = 1e30f, ms = 0.f;
    for (int r : xr)
        for (int c : xc) {
            b->tune.xrpw = r;
            b->tune.ctas_x = c * b->nsm;
            if ((rc = build_worklist(b))) return rc;
            if ((rc = time_phase(1, &ms))) return rc;
            if (ms < best_ms) {
                best_ms = ms;
                best.xrpw = r;
                best.ctas_x = c * b->nsm;
            }
        }
    b->tune.xrpw = best.xrpw;
    b->tune.ctas_x = best.ctas_x;
    best_ms = 1e30f;
    for (int s : ys)
        for (int c : yc) {
            b->tune.yseg = s;
            b->tune.ctas_y = c * b->nsm;
            if ((rc = build_worklist(b))) return rc;
            if ((rc = time_phase(2, &ms))) return rc;
            if (ms < best_ms) {
                best_ms = ms;
                best.yseg = s;
                best.ctas_y = c * b->nsm;
            }
        }
    b->tune = best;
    return build_worklist(b);
}

int mhd_batch_tune(mhd_batch* b, int reps, mhd_batch_tuning* best_out) {
    mhd::NvtxRange nvtx_range("mhd_batch_tune");
    if (!b) return berr(MHD_ERR_STATE, "mhd_batch_tune: null batch");
    const mhd_batch_tuning tune = b->tune;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    int rc = cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess
                 ? tune_shapes(b, reps < 1 ? 3 : reps, e0, e1)
                 : berr(MHD_ERR_CUDA, "mhd_batch_tune: events");
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (rc) {  // back to the shape that was there (its lists fit the tables)
        b->tune = tune;
        const std::string what = mhd_last_error();
        build_worklist(b);
        return berr(rc, what.c_str());
    }
    if (best_out) *best_out = b->tune;
    return MHD_OK;
}

}  // extern "C"
