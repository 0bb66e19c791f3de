// Host-side checks of the workspace's scratch (csrc/capi.cu) on a fake runtime
// (fake_cuda.h; built and run by test_workspace.py, no GPU).
//   order: the CFL maximum's accumulator and arrival counter are zero before its
//   first launch, on a non-blocking stream, with work queued on the default stream.
#include <cstdio>

#include "../include/mhd_b200.h"
#include "fake_cuda.h"
#include "launch.h"

static int failures = 0;
#define CHECK(x) \
    do { if (!(x)) { ++failures; std::printf("line %d: %s\n", __LINE__, #x); } } while (0)

// The maximum: 1 for every state, delivered as the kernel's last CTA does.
namespace mhd {
cudaError_t launch_max_speed_f64(const DevGrid&, double, double, const MaxOut& out, cudaStream_t st) {
    fake::put(st, [=] {
        CHECK(*out.acc == 0 && *out.count == 0);
        const double one = 1.0;
        if (out.clock) {
            *out.clock = DevClock{};
            std::memcpy(&out.clock->maxbits[0], &one, 8);
        }
        if (out.host) {
            std::memcpy(&out.host[0], &one, 8);
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
    mhd_workspace* ws = nullptr;
    CHECK(mhd_workspace_create(&g, &ws) == MHD_OK);
    CHECK(mhd_workspace_set_stream(ws, (void*)16) == MHD_OK);
    double dt = 0.0;
    CHECK(mhd_compute_dt(ws, &g, 0.4, &dt) == MHD_OK && dt == 0.4 / 16);
    CHECK(mhd_workspace_destroy(ws) == MHD_OK);
    CHECK(fake::device.empty());
}

int main() {
    order();
    std::printf("%d failures\n", failures);
    return failures ? 1 : 0;
}
