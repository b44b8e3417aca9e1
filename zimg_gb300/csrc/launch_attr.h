// A kernel's dynamic shared memory above 48 KB, admitted once per device: the
// attribute call costs about a microsecond of a launch.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace zg {

// `devices`: one bit per device that has admitted it; a static of the caller,
// one per kernel.
inline cudaError_t allow_shared_memory(const void *kernel, int bytes, std::atomic<unsigned long long> &devices)
{
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess)
		return e;
	const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
	if (devices.load(std::memory_order_acquire) & bit)
		return cudaSuccess;
	e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
	if (e == cudaSuccess)
		devices.fetch_or(bit, std::memory_order_release);
	return e;
}

} // namespace zg
