// A host-side stand-in for the few runtime calls of transfer.cu, for a test without a GPU: "device" memory is host
// memory, copies on a stream are kept back until something waits for them, and calls can be made to fail.
#pragma once
#include <cstddef>

typedef int cudaError_t;
enum { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged };
struct cudaPointerAttributes {
	cudaMemoryType type;
};
typedef void* cudaStream_t;
typedef struct FakeEvent* cudaEvent_t;
enum { cudaHostAllocPortable = 1, cudaEventDisableTiming = 2 };

cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned flags);
cudaError_t cudaFreeHost(void* p);
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned flags);
cudaError_t cudaEventDestroy(cudaEvent_t e);
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s);
cudaError_t cudaEventSynchronize(cudaEvent_t e);
cudaError_t cudaStreamSynchronize(cudaStream_t s);
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t s);
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p);
cudaError_t cudaGetLastError();
cudaError_t cudaSetDevice(int device);
