// Compares the branch-free quotient, reciprocal and square root of
// csrc/exact_div.cuh with the operators, bit for bit (built and run by
// test_exact_div.py).  `host`: with std::fma and the host's seeds; `device`: on
// the GPU, with the hardware's.  Operands: random significands over the declared
// exponents, significands near all ones and near powers of two, quotients whose
// exact value lies next to a rounding midpoint (a nearest to b m for a 54-bit
// m), and every root whose radicand lies within 64 quarter-units of a midpoint's
// square (found by lifting k^2 + k + c = 0 modulo powers of two), which covers
// every root that is closer to a midpoint than the iteration's error.
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "exact_div.cuh"

using namespace mhd::exact;
using u64 = unsigned long long;
using u128 = unsigned __int128;

struct Case {
    double a, b;
};

static double make(u64 sig53, int e, bool neg) {  // sig53 in [2^52, 2^53), value sig53 * 2^(e - 52)
    const u64 bits = ((u64)neg << 63) | ((u64)(e + 1023) << 52) | (sig53 & ((1ull << 52) - 1));
    double d;
    std::memcpy(&d, &bits, 8);
    return d;
}

static void quotients(std::vector<Case>& out, size_t n) {
    std::mt19937_64 r(11);
    auto sig = [&](int kind) -> u64 {
        const u64 s = (r() >> 11) | (1ull << 52);
        if (kind == 1) return ((1ull << 53) - 1 - (r() & 0xfff)) | (1ull << 52);  // near all ones
        if (kind == 2) return (1ull << 52) + (r() & 0xfff);                       // near a power of two
        return s & ((1ull << 53) - 1);
    };
    for (size_t i = 0; i < n; ++i) {
        const int kind = (int)(i % 4);
        const u64 b = sig(kind < 3 ? kind : 0);
        const int eb = (int)(r() % 540) - 480;
        u64 a;
        int ea = eb + (int)(r() % 200) - 100;
        if (kind == 3) {  // next to a midpoint: a = the 53 leading bits of b (2 k + 1), rounded down or up
            const u128 p = (u128)b * (2 * ((r() >> 12) | (1ull << 51)) + 1);
            int sh = 0;
            u128 q = p;
            while (q >> 53) { q >>= 1; ++sh; }
            a = (u64)q + (r() & 1);
            if (a >> 53) a = 1ull << 52;
        } else {
            a = sig((int)(r() % 3));
        }
        if (ea < -950) ea = -950;
        if (ea > 890) ea = 890;
        out.push_back({make(a, ea, r() & 1), make(b, eb, r() & 1)});
    }
    for (double z : {0.0, -0.0})
        for (double b : {3.0, -3.0, 1.0 / 3.0}) out.push_back({z, b});
}

// k in [2^52, 2^53) (and [2^53, 2^54) for odd exponents) with X = k (k + 1) + c a 53-bit
// significand times a power of two: the low `low` bits of X vanish.
static void roots(std::vector<double>& out, size_t n) {
    std::mt19937_64 r(13);
    for (size_t i = 0; i < n; ++i) {
        const u64 s = i % 3 == 1 ? (1ull << 53) - 1 - (r() & 0xfff) : i % 3 == 2 ? (1ull << 52) + (r() & 0xfff)
                                                                                  : (r() >> 11) | (1ull << 52);
        out.push_back(make(s & ((1ull << 53) - 1), (int)(r() % 1700) - 850, false));
    }
    // sqrt(X) against the midpoint k + 1/2: X - (k + 1/2)^2 = c - 1/4 with X = k^2 + k + c
    for (int low : {52, 53})
        for (int c = -64; c <= 64; ++c) {
            std::vector<u64> sol;  // k modulo 2^bits with k^2 + k + c = 0 modulo 2^bits
            for (u64 k = 0; k < 2; ++k)
                if (((k * k + k + (u64)(long long)c) & 1) == 0) sol.push_back(k);
            for (int bits = 2; bits <= low && !sol.empty(); ++bits) {
                std::vector<u64> next;
                const u64 mask = (1ull << bits) - 1;
                for (u64 s : sol)
                    for (u64 t : {s, s + (1ull << (bits - 1))})
                        if ((((u128)t * t + t + (u128)(__int128)c) & mask) == 0) next.push_back(t);
                sol.swap(next);
            }
            for (u64 s : sol)
                for (u64 k = s; k < (1ull << 53); k += 1ull << low) {
                    if (k < (1ull << 52)) continue;
                    const u128 X = (u128)k * k + k + (u128)(__int128)c;  // in [2^104, 2^106)
                    for (int e : {0, 1}) {
                        const int width = 104 + e;  // leading bit
                        if ((X >> width) != 1) continue;
                        const int drop = width - 52;
                        if (X & (((u128)1 << drop) - 1)) continue;
                        for (int p : {-400, 0, 300}) out.push_back(make((u64)(X >> drop), e + 2 * p, false));
                    }
                }
        }
    out.push_back(0.0);
}

XD_HD bool same(double a, double b) { return hi_word(a) == hi_word(b) && lo_word(a) == lo_word(b); }
XD_HD int check_quotient(double a, double b) {
    if (out_den(b) || out_num(a)) return 2;
    const Recip r = recip(b);
    int bad = same(r.y, 1.0 / b) ? 0 : 1;
    if (!same(quot(a, r), a / b)) bad = 1;
    if (!same(quot(a, recip_of(b, r.y)), a / b)) bad = 1;
    if (a > 0.0 && b > 0.0 && !same(quot_pos(a, r), a / b)) bad = 1;
    return bad;
}
XD_HD int check_root(double x) { return out_rad(x) ? 2 : (same(root(x), sqrt(x)) ? 0 : 1); }

__global__ void quotients_kernel(const Case* c, int n, int* count) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(&count[check_quotient(c[i].a, c[i].b)], 1);
}
__global__ void roots_kernel(const double* x, int n, int* count) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(&count[3 + check_root(x[i])], 1);
}

int main(int argc, char** argv) {
    const bool device = argc > 1 && !std::strcmp(argv[1], "device");
    std::vector<Case> q;
    std::vector<double> x;
    quotients(q, device ? 40000000 : 4000000);
    const size_t plain = device ? 20000000 : 2000000;
    roots(x, plain);
    int count[6] = {0};
    if (device) {
        Case* dq = nullptr;
        double* dx = nullptr;
        int* dc = nullptr;
        if (cudaMalloc(&dq, q.size() * sizeof(Case)) || cudaMalloc(&dx, x.size() * 8) || cudaMalloc(&dc, sizeof count)) return 2;
        cudaMemcpy(dq, q.data(), q.size() * sizeof(Case), cudaMemcpyHostToDevice);
        cudaMemcpy(dx, x.data(), x.size() * 8, cudaMemcpyHostToDevice);
        cudaMemset(dc, 0, sizeof count);
        quotients_kernel<<<1184, 256>>>(dq, (int)q.size(), dc);
        roots_kernel<<<1184, 256>>>(dx, (int)x.size(), dc);
        if (cudaMemcpy(count, dc, sizeof count, cudaMemcpyDeviceToHost)) return 2;
    } else {
        for (const Case& c : q) count[check_quotient(c.a, c.b)]++;
        for (double v : x) count[3 + check_root(v)]++;
    }
    std::printf("quotients %d exact %d wrong %d out of range; roots %d exact %d wrong %d out of range (%zu hard)\n",
                count[0], count[1], count[2], count[3], count[4], count[5], x.size() - plain);
    return count[1] || count[4] || x.size() - plain < 100 || count[2] > count[0] / 100 ? 1 : 0;
}
