// Host-side launch sizing: persistent grids = (#SMs x resident CTAs per SM), capped by the task count.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

namespace yalm {

struct DeviceInfo {
	int device = -1;
	int sms = 0;
	int max_smem_optin = 0;
};

inline const DeviceInfo &device_info() {
	static thread_local DeviceInfo info;
	int dev = 0;
	cudaGetDevice(&dev);
	if (info.device != dev) {
		info.device = dev;
		cudaDeviceGetAttribute(&info.sms, cudaDevAttrMultiProcessorCount, dev);
		cudaDeviceGetAttribute(&info.max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
	}
	return info;
}

// Launch whose beginning - scheduling, barriers, tensor memory - overlaps the end of the kernel before it in the stream; the kernel calls
// chain_wait() (common.cuh) before it touches global memory.  Back to back, launch and prologue were up to half of the small kernels' time
// (decode attention at 37 positions 6.2 -> 3.8 us, first prompt portion's attention 16.4 -> 13.7 us, four scored layers 1.36 -> 1.25 ms).  Not for persistent
// grids of several CTAs per SM: these would settle where the kernel before left room first, unevenly (the row kernels of ops_gemv.cu, feed-forward of a token
// 75 -> 87 us); one CTA per SM, by its shared memory, has no choice (stream_rows.cuh).
template <typename... P, typename... A>
inline int launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster, A &&...args) {
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = st;
	cudaLaunchAttribute at[2];
	at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[0].val.programmaticStreamSerializationAllowed = 1;
	at[1].id = cudaLaunchAttributeClusterDimension;
	at[1].val.clusterDim.x = cluster, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
	cfg.attrs = at, cfg.numAttrs = cluster > 1 ? 2 : 1;
	return (int)cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// Lets a kernel use that much dynamic shared memory on the current device: more than 48 KB has to be asked for, on each device.
inline cudaError_t allow_smem(const void *kernel, size_t smem) {
	static std::mutex mu;
	static std::map<std::pair<int, const void *>, size_t> limits;
	if (smem <= 48 * 1024) return cudaSuccess;
	std::lock_guard<std::mutex> lock(mu);
	size_t &limit = limits[{device_info().device, kernel}];
	if (smem <= limit) return cudaSuccess;
	const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (err == cudaSuccess) limit = smem;
	return err;
}

// Resident CTAs per SM for (kernel, block, smem); raises the kernel's dynamic-smem limit on demand.
// Results are cached: the occupancy query is not free and this sits on the per-token path when the
// ops are used outside a CUDA graph.
inline int resident_ctas(const void *kernel, int block, size_t smem, cudaError_t *err) {
	static std::mutex mu;
	static std::map<std::pair<const void *, std::pair<int, size_t>>, int> cache;
	std::lock_guard<std::mutex> lock(mu);
	*err = allow_smem(kernel, smem);
	if (*err != cudaSuccess) return 0;
	auto key = std::make_pair(kernel, std::make_pair(block, smem));
	auto it = cache.find(key);
	if (it != cache.end()) return it->second;
	int occ = 0;
	*err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, block, smem);
	if (*err != cudaSuccess) return 0;
	cache[key] = occ;
	return occ;
}

// Grid for `tasks` warp-tasks with `warps_per_cta` warps per CTA.
inline int persistent_grid(const void *kernel, int block, size_t smem, long tasks, cudaError_t *err) {
	int occ = resident_ctas(kernel, block, smem, err);
	if (*err != cudaSuccess) return 0;
	if (occ < 1) {
		*err = cudaErrorLaunchOutOfResources;
		return 0;
	}
	const int warps_per_cta = block / 32;
	long need = (tasks + warps_per_cta - 1) / warps_per_cta;
	long cap = (long)device_info().sms * occ;
	return (int)std::max(1L, std::min(need, cap));
}

} // namespace yalm
