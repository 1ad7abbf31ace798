// Host-side CUDA helpers shared by the engine's translation units: error
// reporting, device check, allocation and the bounded stream wait.
#pragma once
#include "qpc_internal.h"
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdlib>
#include <time.h>

namespace qpc {

#define QPC_CUDA(call) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) { \
	set_error("%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); return QPC_ERR_CUDA; } } while (0)

// the current device, if it is Blackwell-class (sm_100 or later)
inline int check_device(int* dev)
{
	int n = 0;
	cudaError_t e = cudaGetDeviceCount(&n);
	if (e != cudaSuccess || n == 0) { set_error("no CUDA device: %s", cudaGetErrorString(e)); return QPC_ERR_NODEVICE; }
	QPC_CUDA(cudaGetDevice(dev));
	cudaDeviceProp prop;
	QPC_CUDA(cudaGetDeviceProperties(&prop, *dev));
	if (prop.major * 10 + prop.minor < 100) { set_error("device %s (sm_%d%d) is not Blackwell-class", prop.name, prop.major, prop.minor); return QPC_ERR_NODEVICE; }
	return QPC_OK;
}

// QPC_ALLOC_MAX: device allocations above this many bytes fail, as they would on a full card (for tests of what happens then)
inline bool alloc_refused(size_t bytes)
{
	const char* e = std::getenv("QPC_ALLOC_MAX");
	return e && bytes > (size_t)std::atoll(e);
}

// a failure leaves no error behind for the next cudaGetLastError: some callers go on with less memory
template <class T> inline int dalloc(T** p, size_t n)
{
	const size_t bytes = sizeof(T) * std::max<size_t>(n, 1);
	cudaError_t e = alloc_refused(bytes) ? cudaErrorMemoryAllocation : cudaMalloc((void**)p, bytes);
	if (e != cudaSuccess) { cudaGetLastError(); *p = nullptr; set_error("cudaMalloc(%zu bytes): %s", sizeof(T) * n, cudaGetErrorString(e)); return QPC_ERR_NOMEM; }
	return QPC_OK;
}

inline size_t free_bytes()
{
	size_t f = 0, total = 0;
	if (cudaMemGetInfo(&f, &total) != cudaSuccess) { cudaGetLastError(); return 0; }
	return f;
}

// bounded wait: poll the stream until its work is done, give up after
// wait_limit_s() seconds of wall time with QPC_ERR_TIMEOUT (the work stays
// queued; a later call on the same stream waits for it again)
inline int wait_on(cudaStream_t st)
{
	struct timespec t0, now;
	clock_gettime(CLOCK_MONOTONIC, &t0);
	const double limit = wait_limit_s();
	for (;;) {
		cudaError_t e = cudaStreamQuery(st);
		if (e == cudaSuccess) return QPC_OK;
		if (e != cudaErrorNotReady) { set_error("stream error: %s", cudaGetErrorString(e)); return QPC_ERR_CUDA; }
		clock_gettime(CLOCK_MONOTONIC, &now);
		const double waited = (double)(now.tv_sec - t0.tv_sec) + 1e-9 * (double)(now.tv_nsec - t0.tv_nsec);
		if (waited > limit) {
			set_error("timed out after %.3g s waiting for the device", limit);
			return QPC_ERR_TIMEOUT;
		}
		// a sleep of any length takes ~55 us (the kernel's timer slack): poll without one for the first half millisecond
		// (a single step is 30-100 us), then sleep between polls
		if (waited < 5e-4) continue;
		struct timespec ts = {0, waited < 0.05 ? 20000L : 100000L};
		nanosleep(&ts, nullptr);
	}
}

// Copies to the device and fills go through the stream of the work that reads them (cudaMemcpyAsync, cudaMemsetAsync):
// a plain cudaMemcpy or cudaMemset belongs to the legacy stream, may return before the transfer has reached the device,
// and the library's streams, which do not block on that one, would not wait for it.  The host side of such a copy is
// kept until the stream has been waited for.

// device -> host copy of a result: wait (bounded) for the work queued before it, then
// copy.  Waiting first means the copy never blocks on queued work (a copy into pageable
// memory may block inside the driver until the stream reaches it, without a bound), and a
// wait that runs out leaves no copy pending into a host buffer the caller may free.
inline int copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t st)
{
	if (int rc = wait_on(st)) return rc;
	QPC_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
	return wait_on(st);
}

} // namespace qpc
