// How much dynamic shared memory a kernel may use is set per device: one of these beside every launch of a kernel that
// needs more than 48 KB, so that a process that uses a second device sets it there too.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <mutex>

namespace flsgpu {

class SmemLimit {
	std::mutex mu;
	uint32_t   set[64] {}; // bytes, by device ordinal

public:
	// Let fn use `bytes` on the current device; asks the runtime only when it may not do so yet.
	cudaError_t need(const void* fn, uint32_t bytes) {
		int               dev = 0;
		const cudaError_t g   = cudaGetDevice(&dev);
		if (g != cudaSuccess) { return g; }
		if (dev < 0 || dev >= 64) { return cudaErrorInvalidDevice; }
		std::lock_guard<std::mutex> lk(mu);
		if (bytes <= set[dev]) { return cudaSuccess; }
		const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
		if (e == cudaSuccess) { set[dev] = bytes; }
		return e;
	}
};

} // namespace flsgpu
