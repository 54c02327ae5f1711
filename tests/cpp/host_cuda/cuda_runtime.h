// The few names of the CUDA language that the headers under test need, for a
// host compiler: device code then is plain C++ run by host threads.
#pragma once

#define __host__
#define __device__
#define __shared__ static
#define __forceinline__ inline
#define __restrict__
#define __align__(n) alignas(n)

struct int2 {
    int x, y;
};
struct double2 {
    double x, y;
};
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dmul_rn(double a, double b) { return a * b; }

// The runtime calls of the host code under test; each test defines its own.
#include <cstddef>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaStreamCaptureMode { cudaStreamCaptureModeGlobal = 0, cudaStreamCaptureModeThreadLocal = 1, cudaStreamCaptureModeRelaxed = 2 };
enum { cudaHostAllocPortable = 1, cudaEventDisableTiming = 2 };
using cudaStream_t = struct FakeStream*;
using cudaEvent_t = struct FakeEvent*;
cudaError_t cudaHostAlloc(void**, size_t, unsigned);
cudaError_t cudaFreeHost(void*);
cudaError_t cudaGetLastError();
cudaError_t cudaSetDevice(int);
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned);
cudaError_t cudaEventDestroy(cudaEvent_t);
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t);
cudaError_t cudaEventSynchronize(cudaEvent_t);
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t);
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t);
cudaError_t cudaStreamSynchronize(cudaStream_t);
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*);
