// The ray-cast kernel for launches of few rays.
#pragma once

#include "traverse.cuh"

namespace phe_gb300 {

// Launches of few rays: every chunk of rays has a warp from the start, so there is no
// work counter to clear, and one block an SM spreads the warps over the chip.
//
// Such a launch lasts as long as its slowest warp, whose loads no other warp hides: the tree's upper
// nodes (numTop of them, at most 128 KB) come to shared memory in bulk copies while the rays load, a
// leaf's triangles are loaded three at a time, and registers are plentiful. 4,096 rays on 10K
// triangles: closest hit 58 -> 52 us; any hit 51.5 -> 34 us, with 4 rays a warp (raycast.cu).
constexpr int kSmallMaxWarps = 16;
constexpr int kSmallLeaf = 3;
constexpr uint32_t kCopyWaits = 1u << 20;   // bound of a wait for the copy (each try waits some time itself)

__device__ __forceinline__ bool wait_copy(uint32_t barrier, uint32_t tries)
{
	uint32_t done = 0;
	for (uint32_t k = 0; k < tries && !done; k++)
		asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
		             : "=r"(done) : "r"(barrier) : "memory");
	return done != 0;
}

// A copy that has not arrived after `copyWaits` tries: the thread reads global memory instead, says so (kErrTopCopy),
// and waits again before it ends. kErrCopyPending: it ended all the same while the copy was under way.
template <bool ANY>
__global__ void __launch_bounds__(32 * kSmallMaxWarps, 1)
small_cast_kernel(DeviceScene s, const phe_ray_in* __restrict__ rays, void* __restrict__ out, const uint32_t* __restrict__ scatter,
                  uint32_t n, uint32_t numTop, uint32_t raysPerWarp, uint32_t copyWaits, uint32_t* __restrict__ status)
{
	extern __shared__ ulonglong2 topNodes[];
	__shared__ alignas(8) unsigned long long barrierWord;
	const uint32_t barrier = (uint32_t)__cvta_generic_to_shared(&barrierWord);
	if (threadIdx.x == 0) {
		const uint32_t bytes = numTop * 64u, dst = (uint32_t)__cvta_generic_to_shared(topNodes);
		asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(barrier));
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
		asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(barrier), "r"(bytes) : "memory");
		for (uint32_t at = 0; at < bytes; at += 16384u)
			asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst + at),
			             "l"((const char*)s.nodes + at), "r"(min(16384u, bytes - at)), "r"(barrier)
			             : "memory");
	}
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t i = (blockIdx.x + gridDim.x * (threadIdx.x >> 5)) * raysPerWarp + lane;
	const bool active = lane < raysPerWarp && i < n;
	RayState r;
	if (active) r = load_ray(rays, i);
	__syncthreads();   // the barrier is initialised
	const bool copied = wait_copy(barrier, copyWaits);   // this thread's: others of its block may see the copy arrive
	if (active) {
		HitRecord h = empty_hit(r);
		const TraversalBounds bd{s.numNodes, s.numSlots};
		const TopNodes nodes{s.nodes, topNodes, copied ? numTop : 0u};
		const uint32_t err = fast_ray(r, s.dirLimit) ? traverse<true, ANY, 0, kSmallLeaf>(nodes, s.tris, bd, r, h)
		                                             : traverse<false, ANY, 0, kSmallLeaf>(nodes, s.tris, bd, r, h);
		if (err) atomicOr(status, err);
		if (ANY) ((uint8_t*)out)[scatter ? __ldg(scatter + i) : i] = h.slot == ~0u ? 1 : 0;
		else store_hit((phe_ray_hit*)out, i, r, h);
	}
	if (!copied)   // the copy may still write this block's shared memory
		atomicOr(status, wait_copy(barrier, kCopyWaits) ? kErrTopCopy : kErrTopCopy | kErrCopyPending);
}

} // namespace phe_gb300
