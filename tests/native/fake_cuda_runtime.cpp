// The CUDA runtime calls that the library makes, for launch_failure_test.cu:
// device memory is host memory, streams and events are nothing, a launch goes to
// the test's model of it.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>

#include "fake_cuda_runtime.h"

namespace fake {
int launches = 0, reject = -1;
bool capturing = false;
} // namespace fake

namespace {
thread_local cudaError_t g_last = cudaSuccess;

cudaError_t set(cudaError_t e)
{
    if (e != cudaSuccess) g_last = e;
    return e;
}
} // namespace

extern "C" {

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void** args)
{
    const int k = fake::launches++;
    if (k == fake::reject) return set(cudaErrorLaunchOutOfResources);
    fake::launched(k, args);
    return cudaSuccess;
}
cudaError_t cudaGetLastError()
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int)
{
    return *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1, cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned int, unsigned long long, cudaDriverEntryPointQueryResult*)
{
    return set(cudaErrorSymbolNotFound);  // no tensor maps: levels by plain loads
}
cudaError_t cudaMalloc(void** p, size_t n)
{
    *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
    return *p ? cudaSuccess : set(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemset(void* p, int v, size_t n) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return fake::capturing ? cudaSuccess : cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { return *n = 8, cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes*, const void*) { return set(cudaErrorInvalidValue); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s)
{
    return *s = fake::capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }

} // extern "C"
