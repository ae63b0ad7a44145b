// Primary-ray generation (genPrimaryRaysKernel + calculatePrimaryRayDir,
// cuda_ray_tracer/kernels/RayCastKernel.cu:891-919) with a sub-pixel jitter offset added to the
// pixel location, as the TAA camera offset does (screens/GameScreen.cpp:187-203).

#include "raygen.cuh"
#include "runtime.cuh"

namespace phe_gb300 {

// One thread a ray, in the order of the output: a warp writes 1 KB in one go (32-byte stores where the buffer is
// aligned to them). With the closest hits
// of its 512x512 rays 40.6 us; 42.6 in blocks of 8x8 pixels with two 16-byte stores a ray.
constexpr int kGenBlock = 256;
__global__ void __launch_bounds__(kGenBlock) gen_primary_kernel(phe_ray_in* __restrict__ rays, phe_camera_def cam, uint32_t n,
                                                                uint32_t resX, uint32_t resY, float jx, float jy, int order,
                                                                bool aligned32)
{
	const uint32_t id = blockIdx.x * kGenBlock + threadIdx.x;
	if (id >= n) return;
	uint32_t x, y;
	if (order == 0) {
		y = id / resX;
		x = id - y * resX;
	} else {   // 8x8 tiles (getRayIdx, CudaDeviceHelpers.cuh:49-62)
		const uint32_t tile = id >> 6, tilesX = resX >> 3, tileY = tile / tilesX;
		y = tileY * 8u + ((id >> 3) & 7u);
		x = (tile - tileY * tilesX) * 8u + (id & 7u);
	}
	const f3 d = primary_dir(cam, x, y, resX, resY, jx, jy);
	float4* p = reinterpret_cast<float4*>(rays + id);
	if (aligned32) {
		asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(pack2(cam.origin[0], cam.origin[1])),
		             "l"(pack2(cam.origin[2], 0.0001f)), "l"(pack2(d.x, d.y)), "l"(pack2(d.z, 3.402823466e+38f))
		             : "memory");
	} else {
		p[0] = make_float4(cam.origin[0], cam.origin[1], cam.origin[2], 0.0001f);
		p[1] = make_float4(d.x, d.y, d.z, 3.402823466e+38f);
	}
}

} // namespace phe_gb300

using namespace phe_gb300;

extern "C" phe_status phe_gen_primary_rays(phe_ray_in* rays, const phe_camera_def* cam, uint32_t resX, uint32_t resY,
                                           float jitterX, float jitterY, int order, void* stream)
{
	if (!rays || !cam) return fail(PHE_ERR_INVALID_ARGUMENT, "phe_gen_primary_rays: null argument");
	if (order != 0 && order != 1) return fail(PHE_ERR_INVALID_ARGUMENT, "phe_gen_primary_rays: order must be 0 or 1");
	if (order == 1 && ((resX % 8u) != 0 || (resY % 8u) != 0))
		return fail(PHE_ERR_INVALID_ARGUMENT, "phe_gen_primary_rays: 8x8 order needs a resolution multiple of 8");
	if ((uint64_t)resX * resY > 0xFFFFFFFFull) return fail(PHE_ERR_TOO_LARGE, "phe_gen_primary_rays: too many pixels");
	if (resX == 0 || resY == 0) return PHE_OK;
	const uint32_t n = resX * resY, grid = (uint32_t)(((uint64_t)n + kGenBlock - 1) / kGenBlock);
	gen_primary_kernel<<<grid, kGenBlock, 0, (cudaStream_t)stream>>>(rays, *cam, n, resX, resY, jitterX, jitterY, order,
	                                                                ((uintptr_t)rays & 31u) == 0);
	PHE_CUDA_TRY(cudaGetLastError(), "gen_primary_kernel launch");
	return PHE_OK;
}
