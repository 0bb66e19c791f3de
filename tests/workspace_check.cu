// Host-side checks of the workspace's scratch (csrc/capi.cu) on a fake runtime
// (fake_cuda.h; built and run by test_workspace.py, no GPU).
//   order: the CFL maximum's accumulator and arrival counter are zero before its
//   first launch, on a non-blocking stream, with work queued on the default stream,
//   for which the host does not wait.
//   slots: workspaces share one page-locked block, made after many read-backs of the
//   process and never by workspaces that read nothing; each gets its own result from several
//   threads at once, with more workspaces than slots, and with no block to be had.
#include <cstdio>
#include <thread>

#include "../include/mhd_b200.h"
#include "fake_cuda.h"
#include "launch.h"

static int failures = 0;
#define CHECK(x) \
    do { if (!(x)) { ++failures; std::printf("line %d: %s\n", __LINE__, #x); } } while (0)

// The maximum: gamma, delivered as the kernel's last CTA does.
namespace mhd {
cudaError_t launch_max_speed_f64(const DevGrid&, double gamma, double, const MaxOut& out, cudaStream_t st) {
    fake::put(st, [=] {
        CHECK(*out.acc == 0 && *out.count == 0);
        if (out.clock) {
            *out.clock = DevClock{};
            std::memcpy(&out.clock->maxbits[0], &gamma, 8);
        }
        if (out.host) {
            CHECK(fake::in(fake::host, out.host, 16) || fake::in(fake::device, out.host, 16));
            std::memcpy(&out.host[0], &gamma, 8);
            out.host[1] = (unsigned long long)*out.fault;
        }
    });
    return cudaSuccess;
}
}  // namespace mhd

static mhd_grid shape() {
    static double cells[1];  // never read
    mhd_grid g{};
    g.data = cells;
    g.nx = g.ny = 16;
    g.ng = 2;
    g.dtype = MHD_F64;
    g.pitch = 32;
    g.plane = 32 * 20;
    g.x_max = g.y_max = 1.0;
    return g;
}

static void order() {
    const mhd_grid g = shape();
    for (const bool capture : {false, true}) {
        mhd_workspace* ws = nullptr;
        const int waits = fake::default_waits;
        CHECK(mhd_workspace_create(&g, &ws) == MHD_OK && fake::default_waits == waits);
        fake::capturing = capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
        CHECK(mhd_workspace_set_stream(ws, (void*)16) == MHD_OK);
        fake::capturing = cudaStreamCaptureStatusNone;
        double dt = 0.0;
        CHECK(mhd_set_gamma(ws, 2.0) == MHD_OK);
        CHECK(mhd_compute_dt(ws, &g, 0.4, &dt) == MHD_OK && dt == 0.4 / 16 / 2.0);
        CHECK(mhd_workspace_destroy(ws) == MHD_OK);
    }
    CHECK(fake::device.empty());
}

// n workspaces alive at once, each reading its own maximum and its clock twice over.
static void read_back(int n, double first) {
    const mhd_grid g = shape();
    std::vector<mhd_workspace*> ws(n);
    for (int k = 0; k < n; ++k) {
        CHECK(mhd_workspace_create(&g, &ws[k]) == MHD_OK);
        CHECK(mhd_workspace_set_stream(ws[k], (void*)16) == MHD_OK);
        CHECK(mhd_set_gamma(ws[k], first + k) == MHD_OK);
    }
    for (int pass = 0; pass < 2; ++pass)
        for (int k = 0; k < n; ++k) {
            double v = 0.0;
            mhd_run_info info{};
            CHECK(mhd_max_speed(ws[k], &g, &v) == MHD_OK && v == first + k);
            CHECK(mhd_clock_start(ws[k], &g, 0.4, 1.0) == MHD_OK);
            CHECK(mhd_clock_read(ws[k], &info) == MHD_OK && info.steps == 0 && info.t == 0.0);
            CHECK(mhd_synchronize(ws[k]) == MHD_OK);
        }
    for (int k = 0; k < n; ++k) CHECK(mhd_workspace_destroy(ws[k]) == MHD_OK);
}

static void slots() {
    fake::fail_host = true;
    read_back(3, 2.0);
    fake::fail_host = false;
    fake::host_allocs = 0;
    const mhd_grid g = shape();
    for (int k = 0; k < 20; ++k) {
        mhd_workspace* ws = nullptr;
        CHECK(mhd_workspace_create(&g, &ws) == MHD_OK && mhd_workspace_destroy(ws) == MHD_OK);
    }
    read_back(3, 2.0);
    CHECK(fake::host_allocs == 0);
    for (int k = 0; k < 100; ++k) read_back(2, 2.0);
    CHECK(fake::host_allocs == 1);
    read_back(700, 2.0);
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([t] {
            for (int k = 0; k < 50; ++k) read_back(100, 2.0 + 1000 * t);
        });
    for (auto& t : threads) t.join();
    CHECK(fake::host_allocs == 1 && fake::host.size() == 1);
    CHECK(fake::device.empty());
    // a device reset takes the block; slots of it that come back are not handed out again
    mhd_workspace *before = nullptr, *after[2] = {};
    double v = 0.0;
    CHECK(mhd_workspace_create(&g, &before) == MHD_OK && mhd_max_speed(before, &g, &v) == MHD_OK);
    std::free(fake::host.begin()->first);
    fake::host.clear();
    for (auto& w : after) CHECK(mhd_workspace_create(&g, &w) == MHD_OK);
    for (int k = 0; k < 300; ++k) CHECK(mhd_max_speed(after[0], &g, &v) == MHD_OK);
    CHECK(mhd_workspace_destroy(before) == MHD_OK);
    CHECK(mhd_max_speed(after[1], &g, &v) == MHD_OK);
    CHECK(fake::host_allocs == 2 && fake::host.size() == 1);
    for (auto& w : after) CHECK(mhd_workspace_destroy(w) == MHD_OK);
    read_back(600, 2.0);
}

int main() {
    slots();  // first: it counts the block's allocation
    order();
    std::printf("%d failures\n", failures);
    return failures ? 1 : 0;
}
