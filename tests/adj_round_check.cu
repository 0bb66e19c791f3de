// The adjoint's reciprocals and roots (rcp of csrc/adj_physics.cuh, root of
// csrc/adj_pair.cuh) on the GPU against the correctly rounded operations, bit for
// bit.  FP32: every significand at several exponents, and every bit pattern of a
// coarser raster, zeros, infinities, NaN and the ends of the range among them.
// FP64: random significands, all ones and near powers of two over all exponents.
// Built with the flags of the file of the sweeps it is compiled for, given by
// test_adjoint_rounding.py, which runs it.
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "adj_pair.cuh"

using namespace mhd::adj;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b)); }
__device__ bool same(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b) || (isnan(a) && isnan(b));
}

// count: 0 wrong reciprocals, 1 wrong roots, 2 operands
__global__ void check32(unsigned stride, unsigned first, int exponent, unsigned long long* count) {
    const unsigned n = exponent < 0 ? 0xffffffffu / stride : 1u << 23;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned bits = exponent < 0 ? first + i * stride : ((unsigned)exponent << 23) | i;
        const float x = __uint_as_float(bits);
        const float a = fabsf(x);
        const bool special = a == 0.0f || isinf(x) || isnan(x);
        if (special || (a >= 1.17549435e-38f && a < 8.50705917e37f))  // [2^-126, 2^126)
            if (!same(rcp(x), __fdiv_rn(1.0f, x))) atomicAdd(count, 1ull);
        float s, is;
        root(x, s, is);
        const float want = x > 0.0f ? __fsqrt_rn(x) : 0.0f;
        if (!same(s, want) || !same(is, x > 0.0f ? __fdiv_rn(1.0f, want) : 0.0f)) atomicAdd(count + 1, 1ull);
        atomicAdd(count + 2, 1ull);
    }
}
__global__ void check64(const double* v, int n, unsigned long long* count) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double x = v[i];
        if (!same(rcp(x), __ddiv_rn(1.0, x))) atomicAdd(count, 1ull);
        double s, is;
        root(x, s, is);
        const double want = x > 0.0 ? __dsqrt_rn(x) : 0.0;
        if (!same(s, want) || !same(is, x > 0.0 ? __ddiv_rn(1.0, want) : 0.0)) atomicAdd(count + 1, 1ull);
        atomicAdd(count + 2, 1ull);
    }
}

int main() {
    unsigned long long *dc = nullptr, c[3];
    if (cudaMalloc(&dc, sizeof c)) return 2;
    bool ok = true;
    auto report = [&](const char* what) {
        if (cudaMemcpy(c, dc, sizeof c, cudaMemcpyDeviceToHost)) ok = false;
        std::printf("%s: %llu operands, %llu wrong reciprocals, %llu wrong roots\n", what, c[2], c[0], c[1]);
        ok = ok && c[0] == 0 && c[1] == 0 && c[2] > 0;
    };
    cudaMemset(dc, 0, sizeof c);
    for (int e : {1, 2, 63, 64, 100, 126, 127, 128, 129, 190, 191, 252, 253, 254}) check32<<<1184, 256>>>(1, 0, e, dc);
    report("FP32, every significand");
    cudaMemset(dc, 0, sizeof c);
    check32<<<1184, 256>>>(61, 7, -1, dc);
    report("FP32, all exponents");
    std::vector<double> v;
    std::mt19937_64 r(3);
    for (int i = 0; i < 20000000; ++i) {
        unsigned long long f = r() >> 12;
        if (i % 8 == 1) f = ~(r() & 0xff) & ((1ull << 52) - 1);
        if (i % 8 == 2) f = r() & 0xff;
        if (i % 64 == 3) f = (1ull << 52) - 1;  // all ones
        const unsigned long long e = i % 4 ? r() % 2048 : 1023 - 4 + r() % 8, bits = (r() & 1) << 63 | e << 52 | f;
        double d;
        std::memcpy(&d, &bits, 8);
        v.push_back(d);
    }
    for (double d : {0.0, -0.0, HUGE_VAL, -HUGE_VAL, std::nan("")}) v.push_back(d);
    double* dv = nullptr;
    if (cudaMalloc(&dv, v.size() * 8)) return 2;
    cudaMemcpy(dv, v.data(), v.size() * 8, cudaMemcpyHostToDevice);
    cudaMemset(dc, 0, sizeof c);
    check64<<<1184, 256>>>(dv, (int)v.size(), dc);
    report("FP64");
    return ok ? 0 : 1;
}
