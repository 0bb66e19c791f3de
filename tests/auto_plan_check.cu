// Host-side check of the size-aware task plans (x_plan_auto, y_plan_auto in
// mhd_gpu_acc_b200/csrc/sweep.cuh; built and run by test_auto_plans.py, no
// GPU).  For the extents given on the command line (nx ny) and both
// precisions' resident warps, factors and caps, every (row or strip, cell) must
// be covered exactly once by tasks no longer than the cap.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "sweep.cuh"

using namespace mhd;

static int check(const SweepPlan& pl, int total, int width, int cap) {
    std::vector<unsigned char> hit((size_t)total * width, 0);
    for (long long k = 0; k < plan_tasks(pl, width); ++k) {
        int idx = -1, start = -1, len = -1;
        if (!plan_task(pl, k, width, idx, start, len) || idx < 0 || idx >= width || start < 0 || len < 1 ||
            len > cap || start + len > total)
            return 1;
        for (int c = start; c < start + len; ++c) hit[(size_t)idx * total + c] += 1;
    }
    for (unsigned char h : hit)
        if (h != 1) return 1;
    return 0;
}

int main(int argc, char** argv) {
    int failures = 0;
    for (int a = 1; a + 1 < argc; a += 2) {
        const int nx = std::atoi(argv[a]), ny = std::atoi(argv[a + 1]), strips = (2 + nx + 31) / 32;
        for (int slots : {kSMs * 8, kSMs * 12, kSMs * 16})
            for (double c : {1.8, 2.2, 2.8}) {
                failures += check(x_plan_auto(nx, ny, slots, c, 64), nx, ny, x_seg_len(64));
                failures += check(y_plan_auto(ny, strips, slots, c, 56), ny, strips, 56);
            }
    }
    std::printf("%d failures\n", failures);
    return failures ? 1 : 0;
}
