// One launch of the kernel for few rays with a given bound of its first wait for the upper nodes' copy, at the grid
// that the library takes for it. Returns a CUDA error code.
#include <algorithm>

#include "runtime.cuh"
#include "small_cast.cuh"

using namespace phe_gb300;

extern "C" int small_cast_once(const phe_scene* scene, const phe_ray_in* rays, void* out, const uint32_t* scatter, uint32_t n, int any,
                               uint32_t raysPerWarp, uint32_t copyWaits)
{
	const uint32_t warps = (n - 1) / raysPerWarp + 1, grid = std::min(warps, 152u), perBlock = (warps - 1) / grid + 1;
	if (perBlock > (uint32_t)kSmallMaxWarps) return cudaErrorInvalidConfiguration;
	const size_t smem = (size_t)scene->dev.numTop * 64u;
	auto kernel = any ? small_cast_kernel<true> : small_cast_kernel<false>;
	cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kTopNodes * 64u));
	if (e != cudaSuccess) return e;
	kernel<<<grid, 32 * perBlock, smem>>>(scene->dev, rays, out, scatter, n, scene->dev.numTop, raysPerWarp, copyWaits, scene->status);
	if ((e = cudaGetLastError()) != cudaSuccess) return e;
	return cudaDeviceSynchronize();
}
