// transfer.cu against the stand-in runtime (fake_cuda/cuda_runtime.h).
#include <sched.h>
#include <sys/syscall.h>
#include <unistd.h>

#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <vector>

#include "cuda_runtime.h"

struct FakeEvent {
	size_t upto = 0;   // copies queued before it
};

namespace {
struct Op {
	void* dst;
	const void* src;
	size_t bytes;
	bool own;   // to or from the library's pinned chunks
};
std::mutex mu;
std::vector<Op> ops;
size_t done = 0;
std::map<const void*, cudaMemoryType> types;
std::set<void*> chunks;
std::set<long> threads;
int fail_alloc = -1, allocs = 0, fail_copy_at = -1, copies = 0, plain = 0, last = 0;

void run_to(size_t n) {
	for (; done < n && done < ops.size(); done++) std::memcpy(ops[done].dst, ops[done].src, ops[done].bytes);
}
bool own(const void* p) {
	for (void* c : chunks)
		if (p >= c && p < (char*) c + (512 << 10)) return true;
	return false;
}
}  // namespace

cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
	std::lock_guard<std::mutex> l(mu);
	if (fail_alloc >= 0 && allocs++ >= fail_alloc) return last = cudaErrorMemoryAllocation;
	*p = ::operator new(bytes);
	chunks.insert(*p);
	return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
	std::lock_guard<std::mutex> l(mu);
	chunks.erase(p);
	::operator delete(p);
	return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
	*e = new FakeEvent;
	return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
	delete e;
	return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
	std::lock_guard<std::mutex> l(mu);
	e->upto = ops.size();
	return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
	std::lock_guard<std::mutex> l(mu);
	run_to(e->upto);
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
	std::lock_guard<std::mutex> l(mu);
	run_to(ops.size());
	return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
	std::lock_guard<std::mutex> l(mu);
	if (copies++ == fail_copy_at) return last = cudaErrorInvalidValue;
	threads.insert(syscall(SYS_gettid));
	const bool mine = own(dst) || own(src);
	plain += mine ? 0 : 1;
	ops.push_back(Op{dst, src, bytes, mine});
	return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
	std::lock_guard<std::mutex> l(mu);
	auto it = types.find(p);
	a->type = it == types.end() ? cudaMemoryTypeUnregistered : it->second;
	return cudaSuccess;
}
cudaError_t cudaGetLastError() {
	const int e = last;
	last = 0;
	return e;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }

#include "transfer.cu"

extern "C" {
// alloc_fails: the first pinned allocation that fails, as do all after it (-1: none)
void fake_reset(int alloc_fails, int copy_fails_at) {
	std::lock_guard<std::mutex> l(mu);
	ops.clear();
	done = 0;
	types.clear();
	threads.clear();
	fail_alloc = alloc_fails;
	fail_copy_at = copy_fails_at;
	copies = plain = allocs = last = 0;
}
void fake_type(const void* p, int type) { types[p] = (cudaMemoryType) type; }
int fake_in_flight() { return (int) (ops.size() - done); }
int fake_plain() { return plain; }
int fake_last_error() { return last; }
int fake_threads() { return (int) threads.size(); }
int fake_chunks() { return (int) chunks.size(); }
void fake_finish() { cudaStreamSynchronize(nullptr); }
void retain() { mdgpu::transfer_retain(); }
void release() { mdgpu::transfer_release(); }
int copy_spans(int n, void** host, void** dev, const size_t* bytes, int to_host) {
	std::vector<mdgpu::CopySpan> s;
	for (int k = 0; k < n; k++) s.push_back(mdgpu::CopySpan{host[k], dev[k], bytes[k]});
	return to_host ? mdgpu::copy_to_host(0, nullptr, s.data(), n) : mdgpu::copy_to_device(0, nullptr, s.data(), n);
}
}
