// A stand-in for <cuda_runtime.h>: the host logic of the library's sources compiled by the
// host compiler, with runtime calls that a test defines itself (an error code from a fake
// of the failing call, a record of the order of calls).  Declarations only.
#pragma once
#include <stddef.h>
#include <stdint.h>

#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
struct fake_dim { unsigned x, y, z; };
static fake_dim threadIdx, blockIdx, blockDim, gridDim;
inline void __syncthreads() {}
template <typename T> T __shfl_up_sync(unsigned, T v, int) { return v; }
template <typename T> T __shfl_xor_sync(unsigned, T v, int) { return v; }

typedef int cudaError_t;
enum { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2, cudaErrorInvalidPitchValue = 12 };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone = 0 };
enum cudaMemcpyKind { cudaMemcpyDeviceToHost = 2 };
enum { cudaHostAllocPortable = 1, cudaEventDisableTiming = 2, cudaStreamNonBlocking = 1 };
typedef struct fake_stream* cudaStream_t;
typedef struct fake_event* cudaEvent_t;

cudaError_t cudaGetLastError();
const char* cudaGetErrorString(cudaError_t);
cudaError_t cudaStreamSynchronize(cudaStream_t);
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus*);
cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, unsigned);
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned);
cudaError_t cudaMalloc(void**, size_t);
cudaError_t cudaFree(void*);
cudaError_t cudaMallocHost(void**, size_t);
template <typename T> cudaError_t cudaMalloc(T** p, size_t n) { return cudaMalloc((void**)p, n); }
cudaError_t cudaHostAlloc(void**, size_t, unsigned);
cudaError_t cudaFreeHost(void*);
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t);
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t);
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t);
