// A CUDA runtime on host memory for tests of the library's host code, which is
// compiled against the real headers and linked with this in the runtime's place
// (no GPU, no libcudart).  Device and page-locked memory are host memory filled
// with 0xab; what is queued on the default stream (null) stays queued until
// something waits for it, as behind earlier work, and other streams, which are
// non-blocking, do not wait for it; every allocation can be made to fail.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <vector>

namespace fake {
inline std::recursive_mutex lock;
inline std::vector<std::function<void()>> queued;  // on the default stream
inline std::map<char*, size_t> device, host;       // live allocations
inline int mallocs = 0, host_allocs = 0, fail_malloc_at = -1;
inline bool fail_host = false;
inline int default_waits = 0;  // of the host for the default stream
inline cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;  // of every stream asked about
inline std::function<void()> graph_launch;  // what a launch of the captured graph does
inline bool hollow = false;  // device blocks over 1 GB get a page only (their contents are not looked at)

inline void drain() {
    std::lock_guard<std::recursive_mutex> g(lock);
    for (auto& f : queued) f();
    queued.clear();
}
inline void put(cudaStream_t st, std::function<void()> f) {
    std::lock_guard<std::recursive_mutex> g(lock);
    if (st == nullptr) queued.push_back(f);
    else f();
}
// Whether [p, p + n) lies in a live allocation.
inline bool in(const std::map<char*, size_t>& m, const void* p, size_t n) {
    std::lock_guard<std::recursive_mutex> g(lock);
    auto it = m.upper_bound((char*)p);
    if (it == m.begin()) return false;
    --it;
    return (char*)p + n <= it->first + it->second;
}
inline cudaError_t alloc(std::map<char*, size_t>& m, void** p, size_t n) {
    std::lock_guard<std::recursive_mutex> g(lock);
    const size_t real = hollow && n > (1u << 30) ? 4096 : n;
    *p = std::malloc(real ? real : 1);
    std::memset(*p, 0xab, real);
    m[(char*)*p] = n;
    return cudaSuccess;
}
inline cudaError_t release(std::map<char*, size_t>& m, void* p) {
    if (!p) return cudaSuccess;
    drain();  // the runtime's free waits for the device
    std::lock_guard<std::recursive_mutex> g(lock);
    if (!m.erase((char*)p)) return cudaErrorInvalidValue;
    std::free(p);
    return cudaSuccess;
}
}  // namespace fake
