// Host-side checks of the batched engine's work lists and error paths
// (csrc/batch_api.cu) on a fake runtime (fake_cuda.h; built and run by
// test_batch_lists.py, no GPU).  The fake launches look through the lists they are
// given, which have to lie in live device memory, as the kernels would.
//   large: instances about and past 2^31 cells.
//   round_trip: the values that get_tuning and the tuner give make the shape that
//   is in force when they are set, on the same batch and on another.
//   no_memory: a longer work list that finds no memory leaves the batch as it was.
#include <cstdio>

#include "../include/mhd_b200.h"
#include "batch.cuh"
#include "fake_cuda.h"

static int failures = 0;
#define CHECK(x) \
    do { if (!(x)) { ++failures; std::printf("line %d: %s\n", __LINE__, #x); } } while (0)

struct Launch {
    int which, units, ctas;
    std::vector<mhd::BatchSeg> seg;  // of each unit
};
static std::vector<Launch> launches;
static std::function<void(const mhd::BatchInst*, const mhd::BatchList&, int, bool)> on_launch;

static void look(const mhd::BatchInst* inst, const mhd::BatchList& list, int n, int which, int ctas) {
    if (which == 0) return;
    const bool live = fake::in(fake::device, list.unit_seg, sizeof(int) * list.units) && fake::in(fake::device, inst, sizeof *inst * 2 * n);
    CHECK(live);
    if (!live) return;
    Launch l{which, list.units, ctas, {}};
    std::vector<long long> cells(n, 0);
    for (int u = 0; u < list.units; ++u) {
        const mhd::BatchSeg* s = list.seg + list.unit_seg[u];
        CHECK(fake::in(fake::device, s, sizeof *s) && s->inst >= 0 && s->inst < n && u >= s->unit);
        l.seg.push_back(*s);
        const mhd::DevGrid& g = inst[s->inst].U;
        const int local = u - s->unit;
        if (which == 3) {  // consecutive runs of cells
            int i0, j0, c;
            mhd::max_unit(g, local, i0, j0, c);
            CHECK(i0 >= 0 && i0 < g.nx && j0 >= 0 && j0 < g.ny && c > 0 && (long long)j0 * g.nx + i0 == cells[s->inst]);
            cells[s->inst] += c;
        } else {  // tasks of len cells of a row (x) or rows of a strip (y)
            for (int k = 0; k < 4; ++k) {
                const int task = 4 * local + k;
                if (task >= s->n * s->width) break;
                const int start = s->lo + task / s->width * s->len, len = std::min(s->len, s->hi - start);
                CHECK(start >= 0 && len > 0 && start + len <= (which == 1 ? g.nx : g.ny));
                cells[s->inst] += len;
            }
        }
    }
    for (int i = 0; i < n; ++i) {
        const mhd::DevGrid& g = inst[i].U;
        CHECK(cells[i] == (which == 2 ? (long long)mhd::y_strips(g) * g.ny : (long long)g.nx * g.ny));
    }
    launches.push_back(l);
}

namespace mhd {
cudaError_t launch_batch_f32(const BatchInst* inst, const BatchList& list, const double*, int n, int, int which, int, int,
                             int ctas, cudaStream_t st) {
    look(inst, list, n, which, ctas);
    if (on_launch && which > 0) on_launch(inst, list, which, st == (cudaStream_t)8);
    return cudaSuccess;
}
cudaError_t launch_batch_f64(const BatchInst* inst, const BatchList& list, const double*, int n, int, int which, int, int,
                             int ctas, cudaStream_t st) {
    look(inst, list, n, which, ctas);
    if (on_launch && which > 0) on_launch(inst, list, which, st == (cudaStream_t)8);
    return cudaSuccess;
}
void batch_task_lens_f32(long long x, long long y, TaskLen& tx, TaskLen& ty) {
    tx = task_len(x, kSMs * 16, 2.2, 32, kXOneWave);
    ty = task_len(y, kSMs * 16, 1.85, 28, kYOneWave);
}
void batch_task_lens_f64(long long x, long long y, TaskLen& tx, TaskLen& ty) {
    tx = task_len(x, kSMs * 8, 2.8, 64, kXOneWave);
    ty = task_len(y, kSMs * 8, 2.2, 56, kYOneWave);
}
}  // namespace mhd

static std::vector<int> shape_of_launches() {  // units, CTAs and the lengths of every segment
    std::vector<int> v;
    for (const Launch& l : launches) {
        v.insert(v.end(), {l.which, l.units, l.ctas});
        for (const mhd::BatchSeg& s : l.seg) v.push_back(s.len);
    }
    return v;
}

static mhd_instance_desc desc(int nx, int ny) {
    mhd_instance_desc d{};
    d.nx = nx;
    d.ny = ny;
    d.ng = 2;
    d.x_max = d.y_max = d.t_end = 1.0;
    d.gamma = 1.4;
    d.cfl = 0.4;
    d.cr = 0.18;
    return d;
}

static void large() {
    // 2^31 - 2 cells (the last unit ends past 2^31), just past 2^31, and one row's worth
    fake::hollow = true;
    for (const mhd_instance_desc& d : {desc(49981, 42966), desc(46341, 46341), desc(2147483, 1001)}) {
        mhd_batch* b = nullptr;
        CHECK(mhd_batch_create(&d, 1, MHD_F32, MHD_HLLD, MHD_LIMITER_VANLEER, &b) == MHD_OK && b);
        if (!b) continue;
        launches.clear();
        CHECK(mhd_batch_run(b, 1, nullptr) == MHD_OK && launches.size() >= 3);
        CHECK(mhd_batch_destroy(b) == MHD_OK);
    }
    CHECK(fake::device.empty());
    fake::hollow = false;
}

static void no_memory() {
    std::vector<mhd_instance_desc> d = {desc(1300, 1301), desc(61, 517), desc(4, 4)};
    mhd_batch* b = nullptr;
    CHECK(mhd_batch_create(d.data(), 3, MHD_F64, MHD_HLLD, MHD_LIMITER_VANLEER, &b) == MHD_OK);
    auto run = [&] {  // every launch, the captured graph's among them, on live lists that cover the grids
        launches.clear();
        mhd_run_info info[3];
        CHECK(mhd_batch_run(b, 3, info) == MHD_OK);
        return launches.back().units;
    };
    mhd::BatchInst* inst = nullptr;
    std::vector<std::pair<int, mhd::BatchList>> captured;
    on_launch = [&](const mhd::BatchInst* i, const mhd::BatchList& l, int which, bool graph) {
        inst = const_cast<mhd::BatchInst*>(i);
        if (graph) captured.push_back({which, l});
    };
    fake::graph_launch = [&] {
        CHECK(captured.size() >= 4);
        for (size_t k = captured.size() - 4; k < captured.size(); ++k) look(inst, captured[k].second, 3, captured[k].first, 0);
    };
    const int units = run();
    mhd_batch_tuning was{}, now{};
    CHECK(mhd_batch_get_tuning(b, &was) == MHD_OK);
    const mhd_batch_tuning fine{1, 4, 0, 0};
    for (int k = 0; k < 2; ++k) {  // through set_tuning and through the tuner
        fake::fail_malloc_at = fake::mallocs;
        CHECK((k == 0 ? mhd_batch_set_tuning(b, &fine) : mhd_batch_tune(b, 1, nullptr)) == MHD_ERR_NOMEM);
        fake::fail_malloc_at = -1;
        CHECK(mhd_batch_get_tuning(b, &now) == MHD_OK && std::memcmp(&was, &now, sizeof now) == 0);
        CHECK(run() == units && launches.back().ctas == 0);
    }
    CHECK(mhd_batch_set_tuning(b, &fine) == MHD_OK && run() > units);
    CHECK(mhd_batch_tune(b, 1, nullptr) == MHD_OK);
    run();
    on_launch = nullptr;
    fake::graph_launch = nullptr;
    CHECK(mhd_batch_destroy(b) == MHD_OK);
    CHECK(fake::device.empty());
}

static void round_trip() {
    const std::vector<mhd_instance_desc> d = {desc(1300, 1301), desc(61, 517)};
    for (int kind = 0; kind < 4; ++kind) {  // untuned, tuned, explicit, explicit in one phase
        mhd_batch *b = nullptr, *other = nullptr;
        CHECK(mhd_batch_create(d.data(), 2, MHD_F32, MHD_HLLD, MHD_LIMITER_VANLEER, &b) == MHD_OK);
        CHECK(mhd_batch_create(d.data(), 2, MHD_F32, MHD_HLLD, MHD_LIMITER_VANLEER, &other) == MHD_OK);
        const mhd_batch_tuning both{2, 7, 148, 296}, one{8, 16, 0, 0};
        mhd_batch_tuning best{}, got{};
        if (kind == 1) CHECK(mhd_batch_tune(b, 1, &best) == MHD_OK);
        if (kind >= 2) CHECK(mhd_batch_set_tuning(b, kind == 2 ? &both : &one) == MHD_OK);
        auto run = [](mhd_batch* x) {
            mhd_run_info info[2];
            launches.clear();
            CHECK(mhd_batch_run(x, 1, info) == MHD_OK);
            return shape_of_launches();
        };
        CHECK(mhd_batch_get_tuning(b, &got) == MHD_OK);
        if (kind == 1) CHECK(std::memcmp(&got, &best, sizeof got) == 0);
        run(b);
        const std::vector<int> was = run(b);
        CHECK(mhd_batch_set_tuning(b, &got) == MHD_OK && mhd_batch_set_tuning(other, &got) == MHD_OK);
        run(b);  // captures the graph anew
        run(other);
        CHECK(run(b) == was && run(other) == was);
        CHECK(mhd_batch_destroy(b) == MHD_OK && mhd_batch_destroy(other) == MHD_OK);
    }
}

int main() {
    round_trip();
    no_memory();
    large();
    std::printf("%d failures\n", failures);
    return failures ? 1 : 0;
}
