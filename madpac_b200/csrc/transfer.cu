// Copies between a caller's pageable arrays and the device.
//
// A plain cudaMemcpyAsync to or from pageable memory is staged by the driver in one thread: 12 GB/s
// measured, and on arrays the caller has just allocated that thread also takes every page fault. Here the
// arrays are cut into chunks that go through pinned buffers: each host thread copies its chunks between
// the caller's memory and one of its two buffers while the other one's DMA runs. Large copies use several
// threads, which live for the call only; small ones the calling thread alone.
//
// Measured, state of 1,048,576 molecules on 16 cores: 88 MB out in 4.3 ms (13.4 by plain copies), into
// arrays just allocated in 7 ms (25), 50 MB in in 1.9 ms (3.8); four threads 9 ms into new arrays.
#include "transfer.h"

#include <sched.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace mdgpu {
namespace {

constexpr size_t kChunk = 512 * 1024;       // bytes per DMA: about 10 us on the link
constexpr size_t kPerThread = 1536 * 1024;  // bytes that pay for another thread (20 us to start one)
constexpr int kMaxThreads = 8;
constexpr size_t kMaxIdle = 2 * kMaxThreads;   // lanes kept for later calls: 16 MB of pinned memory

// One thread's pair of pinned chunks.
struct Lane {
	unsigned char* buf[2] = {nullptr, nullptr};
	cudaEvent_t done[2] = {nullptr, nullptr};   // the buffer's DMA
	int device = -1;                            // whose events these are
};

std::mutex g_mutex;
std::vector<Lane> g_idle;
int g_users = 0;

void free_lane(Lane& l) {
	for (int b = 0; b < 2; b++) {
		if (l.done[b]) cudaEventDestroy(l.done[b]);
		if (l.buf[b]) cudaFreeHost(l.buf[b]);
	}
	l = Lane{};
}

// A lane of the device from the idle ones, or a new one.
cudaError_t take_lane(int device, Lane& l) {
	{
		std::lock_guard<std::mutex> lock(g_mutex);
		for (size_t k = 0; k < g_idle.size(); k++)
			if (g_idle[k].device == device) {
				l = g_idle[k];
				g_idle.erase(g_idle.begin() + (std::ptrdiff_t) k);
				return cudaSuccess;
			}
	}
	l = Lane{};
	l.device = device;
	cudaError_t e = cudaSuccess;
	for (int b = 0; b < 2 && e == cudaSuccess; b++) {
		e = cudaHostAlloc((void**) &l.buf[b], kChunk, cudaHostAllocPortable);
		if (e == cudaSuccess) e = cudaEventCreateWithFlags(&l.done[b], cudaEventDisableTiming);
	}
	if (e != cudaSuccess) free_lane(l);
	return e;
}

// Back to the idle ones; every DMA of the lane has ended.
void give_lane(Lane& l) {
	try {
		std::lock_guard<std::mutex> lock(g_mutex);
		if (g_users > 0 && g_idle.size() < kMaxIdle) {
			g_idle.push_back(l);
			return;
		}
	} catch (...) {
	}
	free_lane(l);
}

cudaError_t queue(cudaStream_t s, const CopySpan& c, bool to_host) {
	return to_host ? cudaMemcpyAsync(c.host, c.dev, c.bytes, cudaMemcpyDeviceToHost, s)
	               : cudaMemcpyAsync(c.dev, c.host, c.bytes, cudaMemcpyHostToDevice, s);
}

struct Job {
	int device;
	cudaStream_t stream;
	std::vector<CopySpan> chunks;
	std::atomic<size_t> next{0};
	std::atomic<int> err{(int) cudaSuccess};

	bool ok() const { return err.load(std::memory_order_relaxed) == (int) cudaSuccess; }
	bool check(cudaError_t e) {
		if (e != cudaSuccess) err.store((int) e, std::memory_order_relaxed);
		return e == cudaSuccess;
	}
	const CopySpan* take() {
		const size_t k = next.fetch_add(1, std::memory_order_relaxed);
		return k < chunks.size() && ok() ? &chunks[k] : nullptr;
	}
};

// One thread's share of a copy. Never leaves with a DMA of its lane in flight.
void work(Job& job, Lane& l, bool to_host) {
	if (!job.check(cudaSetDevice(job.device))) return;
	const CopySpan* pending[2] = {nullptr, nullptr};   // the chunk in each buffer's DMA
	for (int b = 0;; b ^= 1) {
		// buffer b is free once its DMA has ended (and, on the way out, its chunk is copied)
		if (pending[b]) {
			if (job.check(cudaEventSynchronize(l.done[b])) && to_host)
				std::memcpy(pending[b]->host, l.buf[b], pending[b]->bytes);
			pending[b] = nullptr;
		}
		const CopySpan* c = job.take();
		if (!c) break;
		if (!to_host) std::memcpy(l.buf[b], c->host, c->bytes);
		if (!job.check(queue(job.stream, CopySpan{l.buf[b], c->dev, c->bytes}, to_host))) break;
		if (!job.check(cudaEventRecord(l.done[b], job.stream))) {
			cudaStreamSynchronize(job.stream);
			break;
		}
		pending[b] = c;
	}
	for (int b = 0; b < 2; b++)
		if (pending[b] && job.check(cudaEventSynchronize(l.done[b])) && to_host)
			std::memcpy(pending[b]->host, l.buf[b], pending[b]->bytes);
}

// Whether a span goes to the driver as it is: arrays that the caller pinned (the DMA runs at the link's rate by
// itself), and device or managed memory, which the driver judges.
bool plain_copy(const CopySpan& span) {
	cudaPointerAttributes a{};
	if (cudaPointerGetAttributes(&a, span.host) != cudaSuccess) {
		cudaGetLastError();
		return false;
	}
	return a.type != cudaMemoryTypeUnregistered && (a.type != cudaMemoryTypeHost || span.bytes >= kChunk);
}

// Processors that this thread may run on (containers and batch systems give a process a part of the machine's).
int processors() {
	cpu_set_t set;
	CPU_ZERO(&set);
	if (sched_getaffinity(0, sizeof(set), &set) == 0) return std::max(1, CPU_COUNT(&set));
	return std::max(1, (int) std::thread::hardware_concurrency());
}

// The lanes of one copy, given back at its end.
struct Lanes {
	std::vector<Lane> all;
	~Lanes() {
		for (Lane& l : all) give_lane(l);
	}
};

// The copy; `direct` is set once one is queued that reads or writes the caller's memory by itself.
cudaError_t copy_spans(int device, cudaStream_t s, const CopySpan* spans, int n, bool to_host, bool& direct) {
	Job job;
	job.device = device;
	job.stream = s;
	size_t total = 0;
	for (int k = 0; k < n; k++) {
		if (!spans[k].host || spans[k].bytes == 0) continue;
		if (plain_copy(spans[k])) {
			const cudaError_t e = queue(s, spans[k], to_host);
			if (e != cudaSuccess) return e;
			direct = true;
			continue;
		}
		for (size_t o = 0; o < spans[k].bytes; o += kChunk)
			job.chunks.push_back(CopySpan{(unsigned char*) spans[k].host + o, (unsigned char*) spans[k].dev + o,
			                              std::min(kChunk, spans[k].bytes - o)});
		total += spans[k].bytes;
	}
	if (job.chunks.empty()) return cudaSuccess;
	const int want = std::max(1, std::min({kMaxThreads, processors() / 2, (int) (total / kPerThread)}));
	Lanes lanes;
	lanes.all.reserve((size_t) want);
	std::vector<std::thread> threads;
	threads.reserve((size_t) want);
	for (int t = 0; t < want; t++) {
		Lane l;
		if (take_lane(device, l) != cudaSuccess) {
			cudaGetLastError();   // fewer lanes do as well: not an error of this call
			break;
		}
		lanes.all.push_back(l);
	}
	if (lanes.all.empty()) {
		// no pinned memory to be had: the driver stages the copies
		for (const CopySpan& c : job.chunks) {
			const cudaError_t e = queue(s, c, to_host);
			if (e != cudaSuccess) return e;
			direct = true;
		}
		return cudaSuccess;
	}
	try {
		for (size_t t = 1; t < lanes.all.size(); t++)
			threads.emplace_back([&job, &lanes, t, to_host] { work(job, lanes.all[t], to_host); });
	} catch (...) {   // no more threads: those that run take all chunks
	}
	work(job, lanes.all[0], to_host);
	for (auto& t : threads) t.join();
	return (cudaError_t) job.err.load();
}

cudaError_t copy(int device, cudaStream_t s, const CopySpan* spans, int n, bool to_host) {
	bool direct = false;
	cudaError_t e;
	try {
		e = copy_spans(device, s, spans, n, to_host, direct);
	} catch (const std::bad_alloc&) {
		e = cudaErrorMemoryAllocation;
	}
	// what comes back is complete on return, and an error leaves no copy of the caller's memory in flight
	if (direct && (to_host || e != cudaSuccess)) {
		const cudaError_t es = cudaStreamSynchronize(s);
		if (e == cudaSuccess) e = es;
	}
	return e;
}

}  // namespace

cudaError_t copy_to_host(int device, cudaStream_t s, const CopySpan* spans, int n) {
	return copy(device, s, spans, n, true);
}

cudaError_t copy_to_device(int device, cudaStream_t s, const CopySpan* spans, int n) {
	return copy(device, s, spans, n, false);
}

void transfer_retain() {
	std::lock_guard<std::mutex> lock(g_mutex);
	g_users++;
}

void transfer_release() {
	std::vector<Lane> old;
	{
		std::lock_guard<std::mutex> lock(g_mutex);
		if (--g_users == 0) old.swap(g_idle);
	}
	for (Lane& l : old) free_lane(l);
}

}  // namespace mdgpu
