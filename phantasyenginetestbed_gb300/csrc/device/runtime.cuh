// Per-device runtime state of the library: device properties, kernel occupancy and the pool of
// per-launch work counters used by the persistent kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../host/common.hpp"
#include "common.cuh"

struct phe_scene {
	phe_gb300::DeviceScene dev;         // dev.nodes4 / dev.nodes8 are set only while that layout is selected
	const float4* nodes4 = nullptr;     // 4-wide nodes, when the tree allows them (else null)
	const uint4* nodes8 = nullptr;      // 8-wide compressed nodes and their leaf records, when the tree
	const float4* leaves8 = nullptr;    // allows them (else null)
	uint32_t numNodes8 = 0, numLeaves8 = 0, maxDepth8 = 0;
	void* allocation = nullptr;   // one cudaMalloc holding nodes, 4-wide nodes, tris, datas, status
	void* shading = nullptr;      // one cudaMalloc holding materials, texture table, sRGB table, texels
	uint64_t bytes = 0, shadingBytes = 0;
	uint64_t generation = 0;      // bumped whenever `dev` changes (layout, materials): graphs re-capture
	int64_t maxMaterialIndex = -1; // largest materialIndex of the triangle data (-1 without data)
	uint32_t* status = nullptr;   // device word: OR of error bits raised by kernels on this scene
	uint32_t maxDepth = 0, maxDepth4 = 0;   // deepest leaf level of the binary and 4-wide trees
	int device = 0;               // ordinal of the device holding the scene
};

namespace phe_gb300 {

struct DeviceInfo {
	int device = -1;
	int numSMs = 0;
	int maxThreadsPerSM = 0;
	uint32_t* counterPool = nullptr; // kCounterPool words
};

constexpr int kMaxDevices = 64;   // device ordinals that the library takes
constexpr uint32_t kCounterPool = 4096;
// Largest ray count of one persistent launch. Every resident warp fetches 32 rays past the end before
// it stops, so the 32-bit work counter needs headroom above the count (2^26 covers 2M resident warps).
constexpr uint32_t kMaxPersistentRays = PHE_MAX_PERSISTENT_RAYS;

// Returns the runtime state of the current device, initialising it on first use.
phe_status device_info(DeviceInfo** out);
// A zeroed work counter for one persistent launch on `stream`. It is cleared by work queued on the stream: a memset
// in a stream that is being captured (*early false), else a kernel that lets the next one start beside it (*early
// true): launch_early the persistent kernel, which waits (wait_for_previous) before it first uses the counter.
phe_status acquire_counter(cudaStream_t stream, uint32_t** counter, bool* early);

// Programmatic launches: a kernel queued with launch_early starts as soon as every block of the kernel before it on
// the stream has left or has said let_next_start, so its launch is not waited for; what that kernel wrote may be read
// after wait_for_previous (a no-op in a kernel launched otherwise). The kernel before it never waits for this one.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Whether launches on `stream` go into a graph (or may not be made now: the launch itself then reports why).
inline bool stream_captures(cudaStream_t stream)
{
	cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
	if (cudaStreamIsCapturing(stream, &c) == cudaSuccess) return c != cudaStreamCaptureStatusNone;
	cudaGetLastError();
	return true;
}

template <class... P, class... A>
cudaError_t launch_early(bool early, void (*kernel)(P...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t stream, A... args)
{
	cudaLaunchAttribute at = {};
	at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at.val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t c = {};
	c.gridDim = dim3(grid);
	c.blockDim = dim3(block);
	c.dynamicSmemBytes = smem;
	c.stream = stream;
	c.attrs = &at;
	c.numAttrs = early ? 1 : 0;
	cudaLaunchKernelEx(&c, kernel, P(args)...);
	return cudaGetLastError();
}

inline phe_status cuda_fail(cudaError_t e, const char* what)
{
	return fail(e == cudaErrorMemoryAllocation ? PHE_ERR_OUT_OF_MEMORY : PHE_ERR_CUDA, "%s: %s", what,
	            cudaGetErrorString(e));
}

#define PHE_CUDA_TRY(call, what)                                  \
	do {                                                          \
		cudaError_t e_ = (call);                                  \
		if (e_ != cudaSuccess) return ::phe_gb300::cuda_fail(e_, what); \
	} while (0)

// Set-up uploads (cudaMemcpy from pageable host memory, cudaMemset of device memory) run on the legacy
// default stream and may return before the bytes reach the device, and launches on streams created
// non-blocking are not ordered after that stream. Waiting for it makes such uploads complete before the
// call that made them returns, so the next launch on any stream reads them.
inline phe_status finish_uploads(const char* what)
{
	cudaError_t e = cudaStreamSynchronize(cudaStreamLegacy);
	return e == cudaSuccess ? PHE_OK : cuda_fail(e, what);
}

} // namespace phe_gb300
