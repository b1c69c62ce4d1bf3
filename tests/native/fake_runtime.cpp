// A fake of the CUDA runtime for server_failures.cu: device memory is host memory,
// and calls fail on request (the counters in fake.h).
#include "fake.h"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>

namespace fake {
std::atomic<int> live{0}, fail_malloc{0}, fail_host{0}, fail_scratch{0}, fail_sweeps{0};
std::atomic<bool> in_flight{false};
bool take(std::atomic<int> &n) { return n > 0 && n-- > 0; }
}  // namespace fake

using namespace fake;

static cudaError_t last = cudaSuccess;
static cudaError_t failed() { return last = cudaErrorMemoryAllocation; }

extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
char __cudaInitModule(void **) { return 1; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { in_flight = false; return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return take(fail_host) ? failed() : (*p = std::calloc(1, n), cudaSuccess); }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { return take(fail_malloc) ? failed() : (*p = std::calloc(1, n), ++live, cudaSuccess); }
cudaError_t cudaFree(void *p) { std::free(p); --live; return cudaSuccess; }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return take(fail_scratch) ? failed() : (*p = std::calloc(1, n), ++live, cudaSuccess); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { std::free(p); --live; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
}
