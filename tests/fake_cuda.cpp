// The runtime calls of fake_cuda.h.
#include "fake_cuda.h"

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::recursive_mutex> g(fake::lock);
    if (fake::mallocs++ == fake::fail_malloc_at) return cudaErrorMemoryAllocation;
    return fake::alloc(fake::device, p, n);
}
cudaError_t cudaFree(void* p) { return fake::release(fake::device, p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    std::lock_guard<std::recursive_mutex> g(fake::lock);
    ++fake::host_allocs;
    if (fake::fail_host) return cudaErrorMemoryAllocation;
    return fake::alloc(fake::host, p, n);
}
cudaError_t cudaFreeHost(void* p) { return fake::release(fake::host, p); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    a->type = fake::in(fake::host, p, 1) ? cudaMemoryTypeHost : fake::in(fake::device, p, 1) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
    fake::put(st, [=] { if (!fake::hollow || n <= (1u << 30)) std::memset(p, v, n); });
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return cudaMemsetAsync(p, v, n, nullptr); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    fake::put(st, [=] { std::memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
    cudaMemcpyAsync(d, s, n, k, nullptr);
    fake::drain();
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    if (st == nullptr) {
        ++fake::default_waits;
        fake::drain();
    }
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    fake::drain();
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)8; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)8; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)8; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
    if (fake::graph_launch) fake::graph_launch();
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)8; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = fake::capturing; return cudaSuccess; }
// events are recorded on the default stream only
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t, unsigned) {
    if (st != nullptr) fake::drain();
    return fake::capturing == cudaStreamCaptureStatusNone ? cudaSuccess : cudaErrorStreamCaptureIsolation;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)8; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    fake::drain();
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
}
