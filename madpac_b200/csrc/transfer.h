// Copies between a caller's (pageable) host arrays and device buffers, through pinned chunks.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace mdgpu {

// Most molecules whose fields pass through a staging buffer that holds all of them at once (88 bytes per molecule,
// 369 MB). Of larger boxes one field after another does, in the room of the widest: a copy of 100 MB has nothing to
// gain from being queued with the next.
constexpr int64_t kStageWhole = int64_t(1) << 22;

struct CopySpan {
	void* host;
	void* dev;
	size_t bytes;
};

// Device -> host on stream s, after what is queued there; the host arrays are complete on return.
cudaError_t copy_to_host(int device, cudaStream_t s, const CopySpan* spans, int n);
// Host -> device on stream s; the host arrays have been read on return, except arrays of half a megabyte
// and more that the caller pinned: as with cudaMemcpyAsync, those are read in stream order.
cudaError_t copy_to_device(int device, cudaStream_t s, const CopySpan* spans, int n);

// The pinned chunks are shared by all contexts of the process: each context holds a reference while it
// lives, the last one to go frees them.
void transfer_retain();
void transfer_release();

}  // namespace mdgpu
