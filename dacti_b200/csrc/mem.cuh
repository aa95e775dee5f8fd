// Device memory of the solvers: one stream-ordered pool per device, owned by the library.
//
// cudaMalloc and cudaFree wait for the whole device. A solver makes about fifteen allocations, a growing
// tree replaces its pool, lists and scratch every few steps, and while many solvers step side by side each
// such call waits for every other solver's kernels. Allocations from the pool are ordered with the solver's
// own stream instead. While solvers live the pool keeps up to KEEP bytes that nothing uses; when the last
// one is gone it gives back all but KEEP_IDLE. CUDA's release threshold counts what the pool holds, used or not, so it
// follows what is in use: a fixed one of KEEP let a synchronisation unmap everything unused, which the next growth
// mapped again, as soon as solvers used more than that.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

namespace dg {

struct DeviceMemory {
	static constexpr size_t KEEP      = size_t(4) << 30;
	static constexpr size_t KEEP_IDLE = size_t(512) << 20;
	static constexpr size_t LARGE     = size_t(16) << 20;  // allocations after which the release threshold is looked at

	cudaMemPool_t pool  = nullptr;
	cudaStream_t stream = nullptr;  // of frees whose last use the host has waited for
	size_t total        = 0;        // the device's memory
	size_t threshold    = KEEP;     // the pool's release threshold as last set
	int users           = 0;

	static std::mutex &lock() {
		static std::mutex m;
		return m;
	}

	// The current device's memory, made at its first use; null with the error in `e`.
	static DeviceMemory *of_device(cudaError_t &e) {
		static DeviceMemory all[64];
		int dev = 0;
		if ((e = cudaGetDevice(&dev)) != cudaSuccess) return nullptr;
		if (dev < 0 || dev >= 64) {
			e = cudaErrorInvalidDevice;
			return nullptr;
		}
		DeviceMemory &d = all[dev];
		std::lock_guard<std::mutex> l(lock());
		if (!d.pool) {
			cudaMemPoolProps p{};
			p.allocType     = cudaMemAllocationTypePinned;
			p.handleTypes   = cudaMemHandleTypeNone;
			p.location.type = cudaMemLocationTypeDevice;
			p.location.id   = dev;
			cudaMemPool_t pool  = nullptr;
			cudaStream_t stream = nullptr;
			if ((e = cudaMemPoolCreate(&pool, &p)) != cudaSuccess) return nullptr;
			unsigned long long keep = KEEP;
			e                       = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
			size_t free_now = 0, total = 0;
			if (e == cudaSuccess) e = cudaMemGetInfo(&free_now, &total);
			if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
			if (e != cudaSuccess) {
				cudaMemPoolDestroy(pool);
				return nullptr;
			}
			d.pool   = pool;
			d.stream = stream;
			d.total  = total;
		}
		return &d;
	}

	size_t in_use() const {
		unsigned long long used = 0;
		return cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess ? (size_t) used : 0;
	}
	// The release threshold at KEEP above what is in use; set where it is off by an eighth of KEEP.
	void follow() {
		const size_t want = in_use() + KEEP;
		std::lock_guard<std::mutex> l(lock());
		if (want < threshold + KEEP / 8 && threshold < want + KEEP / 8) return;
		unsigned long long keep = want;
		if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess) threshold = want;
	}
};

// `bytes` of device memory for work on stream `st`, from its order on.
inline cudaError_t mem_alloc(void **p, size_t bytes, cudaStream_t st) {
	cudaError_t e;
	DeviceMemory *d = DeviceMemory::of_device(e);
	if (!d) return e;
	e = cudaMallocFromPoolAsync(p, bytes > 0 ? bytes : 1, d->pool, st);
	if (e != cudaErrorMemoryAllocation) {
		if (bytes >= DeviceMemory::LARGE) d->follow();
		return e;
	}
	// blocks freed before, of other sizes, may hold the room: give them back and ask once more
	cudaGetLastError();
	if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
	cudaMemPoolTrimTo(d->pool, 0);
	return cudaMallocFromPoolAsync(p, bytes > 0 ? bytes : 1, d->pool, st);
}
// Gives memory back once the work queued on `st` so far is done with it.
inline void mem_free(void *p, cudaStream_t st) {
	if (p) cudaFreeAsync(p, st);
}
// Gives back memory that nothing queued uses any more, whatever became of the stream it was used on.
inline void mem_free_idle(void *p) {
	cudaError_t e;
	DeviceMemory *d = p ? DeviceMemory::of_device(e) : nullptr;
	if (d) cudaFreeAsync(p, d->stream);
}
// Bytes that the pool holds and nothing uses.
inline size_t mem_unused() {
	cudaError_t e;
	DeviceMemory *d             = DeviceMemory::of_device(e);
	unsigned long long reserved = 0, used = 0;
	if (!d || cudaMemPoolGetAttribute(d->pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
	    cudaMemPoolGetAttribute(d->pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
		return 0;
	return reserved > used ? (size_t) (reserved - used) : 0;
}
// Whether more than half of the device's memory is in use by solvers.
inline bool mem_tight() {
	cudaError_t e;
	DeviceMemory *d = DeviceMemory::of_device(e);
	return !d || d->in_use() > d->total / 2;
}
// A user of the current device's pool, as long as it lives.
class MemoryUser {
	DeviceMemory *d_;

public:
	MemoryUser() {
		cudaError_t e;
		d_ = DeviceMemory::of_device(e);
		std::lock_guard<std::mutex> l(DeviceMemory::lock());
		if (d_) ++d_->users;
	}
	MemoryUser(const MemoryUser &)            = delete;
	MemoryUser &operator=(const MemoryUser &) = delete;
	~MemoryUser() {
		if (!d_) return;
		// what the user held has been given back on `stream` (mem_free_idle)
		cudaStreamSynchronize(d_->stream);
		d_->follow();
		std::lock_guard<std::mutex> l(DeviceMemory::lock());
		cudaMemPoolTrimTo(d_->pool, --d_->users > 0 ? d_->threshold : DeviceMemory::KEEP_IDLE);
	}
};

// Held by the one launch that takes every SM of the current device and whose blocks wait for one another.
inline std::mutex &whole_gpu() {
	static std::mutex m[64];
	int dev = 0;
	cudaGetDevice(&dev);
	return m[dev >= 0 && dev < 64 ? dev : 0];
}

// A pinned host block of PINNED_BYTES; up to PINNED_KEEP of them wait for the next solver, since pinning a page
// costs as much as building a small one.
constexpr size_t PINNED_BYTES = 2048;
constexpr size_t PINNED_KEEP  = 64;
inline std::vector<void *> &pinned_free() {
	static std::vector<void *> v;
	return v;
}
inline cudaError_t pinned_alloc(void **p) {
	{
		std::lock_guard<std::mutex> l(DeviceMemory::lock());
		if (!pinned_free().empty()) {
			*p = pinned_free().back();
			pinned_free().pop_back();
			return cudaSuccess;
		}
	}
	return cudaHostAlloc(p, PINNED_BYTES, cudaHostAllocPortable);
}
inline void pinned_release(void *p) {
	if (!p) return;
	{
		std::lock_guard<std::mutex> l(DeviceMemory::lock());
		if (pinned_free().size() < PINNED_KEEP) {
			pinned_free().push_back(p);
			return;
		}
	}
	cudaFreeHost(p);
}

}  // namespace dg
