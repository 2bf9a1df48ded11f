// Host launch helpers shared by the passes' translation units.
#pragma once
#include <atomic>
#include <utility>
#include <cuda_runtime.h>

namespace ab
{

// The dynamic shared-memory limit of a kernel is a per-device setting: set it
// once for each device a process launches on (bit d of `done` = device d).
template <typename Kernel>
static cudaError_t allow_dynamic_smem(Kernel kernel, size_t smem, std::atomic<unsigned long long> & done)
{
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess) return e;
	const unsigned long long bit = 1ull << (dev & 63);
	if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
	e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_acq_rel);
	return e;
}

// Launch with programmatic stream serialization (see griddep_wait).
template <typename... P, typename... A>
static cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&... args)
{
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = grid;
	cfg.blockDim = block;
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

} // namespace ab
