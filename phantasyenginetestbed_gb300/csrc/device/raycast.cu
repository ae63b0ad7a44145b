// Ray-cast kernels and their C-ABI launchers: closest hit (plain and persistent) and any hit.
// Replaces rayCastKernel / rayCastNoPersistenceKernel / shadowRayCastKernel and their launchers
// (cuda_ray_tracer/kernels/RayCastKernel.cu:179-886).
//
// Differences in the launch model: every launch is asynchronous on the caller's stream (the
// reference synchronises the whole device after each launch, RayCastKernel.cu:831-832), and the
// persistent kernels take their work counter from a per-launch slot zeroed on the same stream
// instead of a file-static global reset by a second kernel (RayCastKernel.cu:172-177), so launches
// on different streams do not share state.

#include <algorithm>
#include <atomic>

#include "runtime.cuh"
#include "traverse.cuh"

namespace phe_gb300 {

constexpr int kPlainBlock = 128;
constexpr int kPersistentBlock = 128;
// 10 resident blocks of 128 per SM (48 registers): 9 (the compiler's 52 registers) and 8 made 1M diffuse rays
// 1% and 4% slower, 12 (40 registers, spills) 12%.
constexpr int kCastMinBlocks = 10;
constexpr int cast_min_blocks(bool wide) { return wide ? kWideMinBlocks : kCastMinBlocks; }

template <bool WIDE>
__global__ void __launch_bounds__(kPlainBlock, cast_min_blocks(WIDE)) closest_plain_kernel(DeviceScene s, const phe_ray_in* __restrict__ rays,
                                                                    phe_ray_hit* __restrict__ hits, uint32_t n,
                                                                    uint32_t* __restrict__ status)
{
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	RayState r = load_ray(rays, i);
	HitRecord h = empty_hit(r);
	uint32_t err = trace<false, WIDE>(s, r, h);
	if (err) atomicOr(status, err);
	store_hit(hits, i, r, h);
}

// Persistent warps: a warp starts with the 32 rays of its own index and then takes 32 consecutive rays per atomic
// fetch behind the grid's (one atomic per warp, lane 0 fetches and broadcasts) until the batch is exhausted. With the
// first rays from the counter as well, its 6,080 warps began with as many atomics on one word: 200,000 shadow rays
// on 10K triangles 25.7 -> 22.9 us, 1M diffuse rays 297 -> 293 us, 4M rays 0.3-1.4%. Without a counter the grid covers
// the rays: a launch of one wave needs none cleared before it (2-3 us).
__device__ __forceinline__ uint32_t next_rays(uint32_t* __restrict__ counter)
{
	if (!counter) return 0xFFFFFFFFu;
	wait_for_previous();   // the counter is cleared
	uint32_t base = 0;
	if ((threadIdx.x & 31u) == 0) base = gridDim.x * blockDim.x + atomicAdd(counter, 32u);
	return __shfl_sync(0xffffffffu, base, 0);
}

template <bool WIDE>
__global__ void __launch_bounds__(kPersistentBlock, cast_min_blocks(WIDE)) closest_persistent_kernel(DeviceScene s,
                                                                              const phe_ray_in* __restrict__ rays,
                                                                              phe_ray_hit* __restrict__ hits, uint32_t n,
                                                                              uint32_t* __restrict__ counter,
                                                                              uint32_t* __restrict__ status)
{
	const uint32_t lane = threadIdx.x & 31u;
	uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u;
	while (base < n) {
		uint32_t i = base + lane;
		if (i < n) {
			RayState r = load_ray(rays, i);
			HitRecord h = empty_hit(r);
			uint32_t err = trace<false, WIDE>(s, r, h);
			if (err) atomicOr(status, err);
			store_hit(hits, i, r, h);
		}
		__syncwarp();
		base = next_rays(counter);
	}
}

template <bool WIDE>
__global__ void __launch_bounds__(kPersistentBlock, cast_min_blocks(WIDE)) any_persistent_kernel(DeviceScene s,
                                                                          const phe_ray_in* __restrict__ rays,
                                                                          uint8_t* __restrict__ inLight,
                                                                          const uint32_t* __restrict__ scatter, uint32_t n,
                                                                          uint32_t* __restrict__ counter,
                                                                          uint32_t* __restrict__ status)
{
	const uint32_t lane = threadIdx.x & 31u;
	uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u;
	while (base < n) {
		uint32_t i = base + lane;
		if (i < n) {
			RayState r = load_ray(rays, i);
			HitRecord h = empty_hit(r);
			uint32_t err = trace<true, WIDE>(s, r, h);
			if (err) atomicOr(status, err);
			uint32_t o = scatter ? __ldg(scatter + i) : i;
			inLight[o] = h.slot == ~0u ? 1 : 0;
		}
		__syncwarp();
		base = next_rays(counter);
	}
}

// Any hit of few rays: a warp takes 4 to 32 of them, so that fewer lanes wait for one another, and loads three triangles of a
// leaf at a time, since no other warp hides its loads. (Which rays share a warp changes no answer of an any hit; a closest hit
// reports the slot of a duplicated triangle that its warp comes to first, and keeps 32 consecutive rays.)
//
// Few rays a warp cost instructions that the launches of other streams could issue, so they are taken while the launch makes
// at most kSmallWarps warps an SM, and a block is one warp without shared memory. 155K triangles, us a cast, this / 32 rays a
// warp in blocks of 128: 4,096 rays alone 36.9 / 54.9, on 16 streams at once 4.5 / 4.6 (both bound by the host's launches);
// 8,192 47.7 / 58.9 and 6.2 / 5.9; 16,384 47.8 / 68.3 and 7.2 / 6.8; 40,000 64.2 / 69.6 and 12.4 / 11.9. 4 rays a warp at
// 16,384: 51.9 alone but 16.9 on 16 streams. The upper nodes copied to shared memory (128 KB a block, one block an SM) made
// 4,096 closest hits on 10K triangles 45.7 us alone instead of 49.8 and gained nothing on 155K, but launches of several
// streams waited for one another: on 16 streams 36 us a cast on 155K instead of 5.
constexpr int kSmallLeaf = 3;
constexpr uint32_t kSmallWarps = 7, kSmallMaxWarps = 16;   // of a launch, an SM: with fewer than 32 rays each; with 32
__global__ void __launch_bounds__(32) small_any_kernel(DeviceScene s, const phe_ray_in* __restrict__ rays, uint8_t* __restrict__ inLight,
                                                       const uint32_t* __restrict__ scatter, uint32_t n, uint32_t raysPerWarp,
                                                       uint32_t* __restrict__ status)
{
	const uint32_t i = blockIdx.x * raysPerWarp + threadIdx.x;
	if (threadIdx.x >= raysPerWarp || i >= n) return;
	const RayState r = load_ray(rays, i);
	HitRecord h = empty_hit(r);
	const TraversalBounds bd{s.numNodes, s.numSlots};
	const uint32_t err = fast_ray(r, s.dirLimit) ? traverse<true, true, 0, kSmallLeaf>(s.nodes, s.tris, bd, r, h)
	                                             : traverse<false, true, 0, kSmallLeaf>(s.nodes, s.tris, bd, r, h);
	if (err) atomicOr(status, err);
	inLight[scatter ? __ldg(scatter + i) : i] = h.slot == ~0u ? 1 : 0;
}

// [closest, any] x [binary, wide]; filled on first use (threads that race store the same value)
static std::atomic<int> g_persistentBlocksPerSM[4] = {};

static phe_status persistent_grid(int which, const void* kernel, int* grid)
{
	DeviceInfo* d = nullptr;
	phe_status st = device_info(&d);
	if (st) return st;
	int blocks = g_persistentBlocksPerSM[which].load(std::memory_order_relaxed);
	if (blocks == 0) {
		int b = 0;
		PHE_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, kPersistentBlock,
		                                                           stack_smem_bytes(kPersistentBlock)), "occupancy");
		blocks = b > 0 ? b : 1;
		g_persistentBlocksPerSM[which].store(blocks, std::memory_order_relaxed);
	}
	*grid = blocks * d->numSMs;
	return PHE_OK;
}

static phe_status check_cast_args(const phe_scene* scene, const void* rays, const void* out)
{
	if (!scene) return fail(PHE_ERR_INVALID_ARGUMENT, "scene is null");
	if (!rays || !out) return fail(PHE_ERR_INVALID_ARGUMENT, "ray or result buffer is null");
	if (((uintptr_t)rays & 15u) != 0) return fail(PHE_ERR_INVALID_ARGUMENT, "ray buffer must be 16-byte aligned");
	return PHE_OK;
}

// Queues an any-hit launch of few rays on binary nodes (*done) or leaves it to the caller.
static phe_status small_any(const phe_scene* scene, const phe_ray_in* rays, uint8_t* inLight, const uint32_t* scatter, uint32_t n,
                            cudaStream_t stream, bool* done)
{
	*done = false;
	if (scene->dev.nodes4 || scene->dev.nodes8) return PHE_OK;
	DeviceInfo* d = nullptr;
	if (phe_status st = device_info(&d)) return st;
	uint32_t perWarp = 4;
	while (perWarp < 32u && (n - 1) / perWarp >= (uint32_t)d->numSMs * kSmallWarps) perWarp *= 2;
	const uint32_t warps = (n - 1) / perWarp + 1;
	if (warps > (uint32_t)d->numSMs * kSmallMaxWarps) return PHE_OK;
	small_any_kernel<<<warps, 32, 0, stream>>>(scene->dev, rays, inLight, scatter, n, perWarp, scene->status);
	PHE_CUDA_TRY(cudaGetLastError(), "small_any_kernel launch");
	*done = true;
	return PHE_OK;
}

} // namespace phe_gb300

using namespace phe_gb300;

extern "C" phe_status phe_cast_closest_plain(const phe_scene* scene, const phe_ray_in* rays, phe_ray_hit* hits, uint32_t n,
                                             void* stream)
{
	phe_status st = check_cast_args(scene, rays, hits);
	if (st) return st;
	if (((uintptr_t)hits & 15u) != 0) return fail(PHE_ERR_INVALID_ARGUMENT, "hit buffer must be 16-byte aligned");
	if (n == 0) return PHE_OK;
	uint32_t grid = (n + kPlainBlock - 1) / kPlainBlock;
	auto kernel = (scene->dev.nodes4 || scene->dev.nodes8) ? closest_plain_kernel<true> : closest_plain_kernel<false>;
	kernel<<<grid, kPlainBlock, stack_smem_bytes(kPlainBlock), (cudaStream_t)stream>>>(scene->dev, rays, hits, n,
	                                                                                   scene->status);
	PHE_CUDA_TRY(cudaGetLastError(), "closest_plain_kernel launch");
	return PHE_OK;
}

extern "C" phe_status phe_cast_closest(const phe_scene* scene, const phe_ray_in* rays, phe_ray_hit* hits, uint32_t n,
                                       void* stream)
{
	phe_status st = check_cast_args(scene, rays, hits);
	if (st) return st;
	if (((uintptr_t)hits & 15u) != 0) return fail(PHE_ERR_INVALID_ARGUMENT, "hit buffer must be 16-byte aligned");
	if (n == 0) return PHE_OK;
	if (n > kMaxPersistentRays) return fail(PHE_ERR_TOO_LARGE, "phe_cast_closest: at most %u rays per launch", kMaxPersistentRays);
	const bool wide = scene->dev.nodes4 || scene->dev.nodes8;
	auto kernel = wide ? closest_persistent_kernel<true> : closest_persistent_kernel<false>;
	int grid = 0;
	if ((st = persistent_grid(wide ? 2 : 0, (const void*)kernel, &grid))) return st;
	uint32_t maxGrid = (n + kPersistentBlock - 1) / kPersistentBlock;
	uint32_t* counter = nullptr;
	bool early = false;
	if ((uint32_t)grid >= maxGrid) grid = (int)maxGrid;   // one wave: no counter
	else if ((st = acquire_counter((cudaStream_t)stream, &counter, &early))) return st;
	PHE_CUDA_TRY(launch_early(early, kernel, grid, kPersistentBlock, stack_smem_bytes(kPersistentBlock), (cudaStream_t)stream,
	                          scene->dev, rays, hits, n, counter, scene->status), "closest_persistent_kernel launch");
	return PHE_OK;
}

extern "C" phe_status phe_cast_any(const phe_scene* scene, const phe_ray_in* rays, uint8_t* inLight, uint32_t n,
                                   const uint32_t* scatter, void* stream)
{
	phe_status st = check_cast_args(scene, rays, inLight);
	if (st) return st;
	if (n == 0) return PHE_OK;
	if (n > kMaxPersistentRays) return fail(PHE_ERR_TOO_LARGE, "phe_cast_any: at most %u rays per launch", kMaxPersistentRays);
	bool done = false;
	if ((st = small_any(scene, rays, inLight, scatter, n, (cudaStream_t)stream, &done)) || done) return st;
	const bool wide = scene->dev.nodes4 || scene->dev.nodes8;
	auto kernel = wide ? any_persistent_kernel<true> : any_persistent_kernel<false>;
	int grid = 0;
	if ((st = persistent_grid(wide ? 3 : 1, (const void*)kernel, &grid))) return st;
	uint32_t maxGrid = (n + kPersistentBlock - 1) / kPersistentBlock;
	uint32_t* counter = nullptr;
	bool early = false;
	if ((uint32_t)grid >= maxGrid) grid = (int)maxGrid;   // one wave: no counter
	else if ((st = acquire_counter((cudaStream_t)stream, &counter, &early))) return st;
	PHE_CUDA_TRY(launch_early(early, kernel, grid, kPersistentBlock, stack_smem_bytes(kPersistentBlock), (cudaStream_t)stream,
	                          scene->dev, rays, inLight, scatter, n, counter, scene->status), "any_persistent_kernel launch");
	return PHE_OK;
}
