// The CUDA runtime calls that this library's host code makes, on host memory and without a device: linked with the
// library's own objects, it runs their host code (scene upload, launch sequences) on a machine that has no GPU. Kernels
// are recorded, not run; what is not needed for that is left undefined (lazy binding).
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <string>
#include <vector>

namespace {

struct Launch {
	std::string kernel;
	dim3 grid, block;
	size_t smem;
	std::string scene;   // the bytes of a scene passed by value as the first argument
	bool early;   // with the programmatic-serialization attribute
};
struct Config {
	dim3 grid, block;
	size_t smem;
	cudaStream_t stream;
};

int g_device = 0;
int g_occupancy[2] = {4, 4};   // resident blocks of every kernel, by device
uintptr_t g_handles = 16;      // streams and events are numbers
std::vector<Launch> g_launches;
std::vector<std::pair<void*, size_t>> g_allocations;   // in order of allocation
std::vector<Config> g_configs;
int g_live = 0;                // allocations not freed
thread_local long g_newsLeft = -1;   // host allocations until one fails (-1: none does)

std::map<const void*, std::string>& kernel_names()
{
	static std::map<const void*, std::string> names;
	return names;
}
cudaError_t g_lastError = cudaSuccess;

cudaError_t record(const void* f, dim3 grid, dim3 block, size_t smem, void** args, bool early)
{
	if (!grid.x || !grid.y || !grid.z || grid.x > 0x7FFFFFFFu || grid.y > 65535u || grid.z > 65535u)
		return g_lastError = cudaErrorInvalidConfiguration;
	const std::string& name = kernel_names()[f];
	const bool scene = name.find("EvNS_11DeviceScene") != std::string::npos;
	g_launches.push_back({name, grid, block, smem, scene ? std::string((const char*)args[0], 128) : "", early});
	return cudaSuccess;
}

} // namespace

// The library's host allocations, of which one can be made to fail.
void* operator new(size_t n)
{
	if (g_newsLeft >= 0 && g_newsLeft-- == 0) throw std::bad_alloc();
	if (void* p = std::malloc(n ? n : 1)) return p;
	throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {

// What the tests set and read.
void fake_fail_new(long after) { g_newsLeft = after; }
int fake_live_allocations() { return g_live; }
void fake_set_device(int device) { g_device = device; }
void fake_set_occupancy(int device, int blocks) { g_occupancy[device] = blocks; }
int fake_num_launches() { return (int)g_launches.size(); }
const char* fake_launch(int i, uint32_t grid[3], uint32_t block[3], size_t* smem, int* early)
{
	const Launch& l = g_launches[i];
	grid[0] = l.grid.x, grid[1] = l.grid.y, grid[2] = l.grid.z;
	block[0] = l.block.x, block[1] = l.block.y, block[2] = l.block.z;
	*smem = l.smem;
	*early = l.early;
	return l.kernel.c_str();
}
const char* fake_launch_scene(int i) { return g_launches[i].scene.size() == 128 ? g_launches[i].scene.data() : nullptr; }
int fake_num_allocations() { return (int)g_allocations.size(); }
void* fake_allocation(int i, size_t* bytes)
{
	*bytes = g_allocations[i].second;
	return g_allocations[i].first;
}

// Registration and launches.
static void* g_module;
void** __cudaRegisterFatBinary(void*) { return &g_module; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) { kernel_names()[host] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream)
{
	g_configs.push_back({grid, block, smem, (cudaStream_t)stream});
	return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream)
{
	const Config c = g_configs.back();
	g_configs.pop_back();
	*grid = c.grid, *block = c.block, *smem = c.smem, *(cudaStream_t*)stream = c.stream;
	return cudaSuccess;
}
cudaError_t __cudaGetKernel(void** handle, const void* f)
{
	*handle = const_cast<void*>(f);
	return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(void* handle, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t)
{
	return record(handle, grid, block, smem, args, false);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args)
{
	bool early = false;
	for (unsigned i = 0; i < c->numAttrs; i++)
		early = early || (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization &&
		                  c->attrs[i].val.programmaticStreamSerializationAllowed);
	return record(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, args, early);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t)
{
	*n = g_occupancy[g_device];
	return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int block, size_t smem, unsigned)
{
	return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, block, smem);
}

// Devices, memory, streams and events.
cudaError_t cudaGetDevice(int* d) { return *d = g_device, cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int)
{
	std::memset(p, 0, sizeof(*p));
	p->multiProcessorCount = 152;
	p->maxThreadsPerMultiProcessor = 2048;
	return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError()
{
	const cudaError_t e = g_lastError;
	g_lastError = cudaSuccess;
	return e;
}
cudaError_t cudaMalloc(void** p, size_t n)
{
	const size_t size = (n + 255) & ~size_t(255);
	*p = std::aligned_alloc(256, size);
	if (!*p) return cudaErrorMemoryAllocation;
	std::memset(*p, 0xCD, size);
	g_allocations.push_back({*p, n});
	g_live++;
	return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
	g_live -= p != nullptr;
	std::free(p);
	return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = std::calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)g_handles++, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { return *c = cudaStreamCaptureStatusNone, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) { return *g = (cudaGraphExec_t)g_handles++, cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)g_handles++, cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)g_handles++, cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }

} // extern "C"
