// The branch-free quotient, reciprocal and square root of csrc/exact_div.cuh against
// the operators, bit for bit, over the whole of the ranges that the out_*
// functions let through: the exponents of numerator and denominator are drawn
// independently of each other, to the ranges' ends and past them, infinities, NaN
// and subnormal numbers among them (exact_div_check.cu holds the hardest
// roundings, at exponents near each other).  `host` or `device`; built and run by
// test_exact_range.py.
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "exact_div.cuh"

using namespace mhd::exact;
using u64 = unsigned long long;

struct Case {
    double a, b;
};

static std::vector<Case> cases(size_t n) {
    std::mt19937_64 r(17);
    auto value = [&](int lo, int hi) {
        const int kind = (int)(r() % 64);
        if (kind == 0) {
            const double odd[6] = {0.0, INFINITY, NAN, 5e-324, 2e-308, 1.7e308};
            return r() & 1 ? odd[r() % 6] : -odd[r() % 6];
        }
        // an exponent anywhere, or about an end of [2^lo, 2^hi)
        const int e = kind < 12 ? lo - 3 + (int)(r() % 6) : kind < 24 ? hi - 3 + (int)(r() % 6) : lo + (int)(r() % (hi - lo));
        u64 f = r() >> 12;
        if (r() % 4 == 0) f = ~(r() & 0xfff) & ((1ull << 52) - 1);
        if (r() % 4 == 0) f = r() & 0xfff;
        const u64 bits = ((r() & 1) << 63) | ((u64)(e + 1023) << 52) | f;
        double d;
        std::memcpy(&d, &bits, 8);
        return d;
    };
    std::vector<Case> out(n);
    for (Case& c : out) c = {value(-960, 900), value(-480, 60)};
    return out;
}

XD_HD bool same(double a, double b) { return hi_word(a) == hi_word(b) && lo_word(a) == lo_word(b); }
// 0 exact, 1 wrong, 2 out of range
XD_HD int check(const Case& c) {
    const double a = c.a, b = c.b;
    if (!out_rad(fabs(a)) && !same(root(fabs(a)), sqrt(fabs(a)))) return 1;
    if (out_den(b)) return 2;
    const Recip r = recip(b);
    if (!same(r.y, 1.0 / b)) return 1;
    if (out_num(a)) return 2;
    if (!same(quot(a, r), a / b) || !same(quot(a, recip_of(b, r.y)), a / b)) return 1;
    return a > 0.0 && b > 0.0 && !same(quot_pos(a, r), a / b) ? 1 : 0;
}

__global__ void kernel(const Case* c, int n, int* count) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(&count[check(c[i])], 1);
}

int main(int argc, char** argv) {
    const bool device = argc > 1 && !std::strcmp(argv[1], "device");
    const std::vector<Case> c = cases(device ? 20000000 : 4000000);
    int count[3] = {0};
    if (device) {
        Case* dc = nullptr;
        int* dn = nullptr;
        if (cudaMalloc(&dc, c.size() * sizeof(Case)) || cudaMalloc(&dn, sizeof count)) return 2;
        cudaMemcpy(dc, c.data(), c.size() * sizeof(Case), cudaMemcpyHostToDevice);
        cudaMemset(dn, 0, sizeof count);
        kernel<<<1184, 256>>>(dc, (int)c.size(), dn);
        if (cudaMemcpy(count, dn, sizeof count, cudaMemcpyDeviceToHost)) return 2;
    } else {
        for (const Case& k : c) {
            const int r = check(k);
            if (r == 1 && count[1] < 10) std::printf("wrong: %a / %a: %a, operator %a\n", k.a, k.b, quot(k.a, recip(k.b)), k.a / k.b);
            ++count[r];
        }
    }
    std::printf("%d exact, %d wrong, %d out of range\n", count[0], count[1], count[2]);
    return count[1] || count[0] < (int)c.size() / 4 ? 1 : 0;
}
