// Device memory of the solvers: small blocks from one stream-ordered pool per device, owned by the library, large
// ones from cudaMalloc.
//
// cudaMalloc and cudaFree wait for the whole device. A solver makes about fifteen allocations, a growing
// tree replaces its pool, lists and scratch every few steps, and while many solvers step side by side each
// such call waits for every other solver's kernels. Allocations from the pool are ordered with the solver's
// own stream instead. But the pool maps and unmaps memory at 6.5 ms a GiB each way, with stalls of a second and more
// on a shared host, where cudaMalloc takes 1 to 2 ms and cudaFree 0.5 ms a GiB whatever the size: a tree that grows from 2 to
// 36 GiB takes 0.15 s with the one and 0.7 to 4.7 s with the other. So blocks of LARGE bytes on do not come from the pool.
// A large block that is given back waits in a list for the next moment that waits for the device anyway: an allocation that
// does not fit, the end of a user, or KEEP bytes of them.
//
// While solvers live the pool keeps up to KEEP bytes that nothing uses; when the last one is gone it gives
// back all but KEEP_IDLE. CUDA's release threshold counts what the pool holds, used or not, so it follows what is in
// use: a fixed one let a synchronisation unmap everything unused, which the next growth mapped again, as soon as solvers
// used more than that.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <unordered_map>
#include <vector>

namespace dg {

struct DeviceMemory {
	static constexpr size_t KEEP      = size_t(2) << 30;
	static constexpr size_t KEEP_IDLE = size_t(512) << 20;
	static constexpr size_t LARGE     = size_t(64) << 20;  // a mapping of this size takes as long as cudaMalloc
	static constexpr size_t NOTICE    = size_t(4) << 20;   // allocations after which the release threshold is looked at

	cudaMemPool_t pool  = nullptr;
	cudaStream_t stream = nullptr;  // of frees whose last use the host has waited for
	size_t total        = 0;        // the device's memory
	size_t threshold    = KEEP;     // the pool's release threshold as last set
	int users           = 0;
	std::unordered_map<void *, size_t> large;  // blocks from cudaMalloc
	std::vector<void *> retired;               // the same, given back
	size_t large_bytes = 0, retired_bytes = 0;

	static std::mutex &lock() {
		static std::mutex m;
		return m;
	}

	// The current device's memory, made at its first use; null with the error in `e`.
	static DeviceMemory *of_device(cudaError_t &e) {
		static DeviceMemory *all = new DeviceMemory[64];  // outlives every user, at the process's end too
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

	size_t pool_in_use() const {
		unsigned long long used = 0;
		return cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess ? (size_t) used : 0;
	}
	// The release threshold at KEEP above what is in use; set where it is off by an eighth of KEEP.
	void follow() {
		const size_t want = pool_in_use() + KEEP;
		std::lock_guard<std::mutex> l(lock());
		if (want < threshold + KEEP / 8 && threshold < want + KEEP / 8) return;
		unsigned long long keep = want;
		if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess) threshold = want;
	}
	cudaError_t alloc(void **p, size_t bytes, cudaStream_t st) {
		if (bytes < LARGE) {
			const cudaError_t e = cudaMallocFromPoolAsync(p, bytes > 0 ? bytes : 1, pool, st);
			if (e == cudaSuccess && bytes >= NOTICE) follow();
			return e;
		}
		const cudaError_t e = cudaMalloc(p, bytes);
		if (e != cudaSuccess) return e;
		std::lock_guard<std::mutex> l(lock());
		large[*p] = bytes;
		large_bytes += bytes;
		return cudaSuccess;
	}
	// Takes back a large block, which work already queued may still use; false for a block of the pool.
	bool retire(void *p) {
		{
			std::lock_guard<std::mutex> l(lock());
			const auto it = large.find(p);
			if (it == large.end()) return false;
			large_bytes -= it->second;
			retired_bytes += it->second;
			large.erase(it);
			retired.push_back(p);
			if (retired_bytes <= KEEP) return true;
		}
		reclaim();
		return true;
	}
	// Frees the retired blocks once nothing uses them.
	void reclaim() {
		std::vector<void *> gone;
		{
			std::lock_guard<std::mutex> l(lock());
			gone.swap(retired);
			retired_bytes = 0;
		}
		if (gone.empty()) return;
		cudaDeviceSynchronize();
		for (void *p: gone) cudaFree(p);
	}
};

// `bytes` of device memory for work on stream `st`, from its order on.
inline cudaError_t mem_alloc(void **p, size_t bytes, cudaStream_t st) {
	cudaError_t e;
	DeviceMemory *d = DeviceMemory::of_device(e);
	if (!d) return e;
	e = d->alloc(p, bytes, st);
	if (e != cudaErrorMemoryAllocation) return e;
	// blocks given back before may hold the room: free them and ask once more
	cudaGetLastError();
	if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
	d->reclaim();
	cudaMemPoolTrimTo(d->pool, 0);
	return d->alloc(p, bytes, st);
}
// Gives memory back once the work queued on `st` so far is done with it.
inline void mem_free(void *p, cudaStream_t st) {
	cudaError_t e;
	DeviceMemory *d = p ? DeviceMemory::of_device(e) : nullptr;
	if (d && !d->retire(p)) cudaFreeAsync(p, st);
}
// Gives back memory that nothing queued uses any more, whatever became of the stream it was used on.
inline void mem_free_idle(void *p) {
	cudaError_t e;
	DeviceMemory *d = p ? DeviceMemory::of_device(e) : nullptr;
	if (d && !d->retire(p)) cudaFreeAsync(p, d->stream);
}
// Bytes that the library holds and nothing uses.
inline size_t mem_unused() {
	cudaError_t e;
	DeviceMemory *d             = DeviceMemory::of_device(e);
	unsigned long long reserved = 0, used = 0;
	if (!d || cudaMemPoolGetAttribute(d->pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
	    cudaMemPoolGetAttribute(d->pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
		return 0;
	std::lock_guard<std::mutex> l(DeviceMemory::lock());
	return (reserved > used ? (size_t) (reserved - used) : 0) + d->retired_bytes;
}
// Whether more than half of the device's memory is in use by solvers, or would nearly be (45%) with `more`: what is taken
// below the one line is not given up again at once above the other.
inline bool mem_tight(size_t more = 0) {
	cudaError_t e;
	DeviceMemory *d = DeviceMemory::of_device(e);
	if (!d) return true;
	const size_t used = d->pool_in_use();
	std::lock_guard<std::mutex> l(DeviceMemory::lock());
	return used + d->large_bytes + more > (more > 0 ? d->total / 20 * 9 : d->total / 2);
}
// A user of the current device's memory, as long as it lives.
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
		// what the user held has been given back (mem_free_idle)
		d_->reclaim();
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
