// Compares the texels and the weight of one axis of a GL_LINEAR fetch (linear_axis, csrc/device/sampling.cuh) with the
// same in 64-bit integers, over sizes up to 2^32 - 1 and positions up to beyond them. Prints the count of
// differing results; exits 0 when there are none.
#include <cstdio>
#include <vector>

#include "common.cuh"
#include "sampling.cuh"

__global__ void compare(const float* ps, uint32_t numP, const uint32_t* ns, uint32_t numN, unsigned long long* bad)
{
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= numP * numN) return;
	const float p = ps[i % numP];
	const uint32_t n = ns[i / numP];
	const phe_gb300::LinearAxis got = phe_gb300::linear_axis(p, n);
	const float f = __fsub_rn(p, 0.5f), f0 = floorf(f), a = __fsub_rn(f, f0);
	const long long m = (long long)n - 1, x0 = f0 < -1e18f ? -1 : f0 > 1e18f ? m : (long long)f0, x1 = x0 + 1;
	const long long i0 = x0 < 0 ? 0 : x0 > m ? m : x0, i1 = x1 < 0 ? 0 : x1 > m ? m : x1;
	if (got.i0 != i0 || got.i1 != i1 || (__float_as_uint(got.a) != __float_as_uint(a) && !isnan(a))) atomicAdd(bad, 1ull);
}

int main()
{
	const std::vector<uint32_t> ns = {1, 2, 3, 97, 1920, 65536, 65537, 16777217, 0x7FFFFFFFu, 0x80000000u, 0x80000001u, 0xFFFFFFFFu};
	std::vector<float> ps = {0.0f, -0.0f, 1e-30f, 0.49999997f, 0.5f, 0.50000006f, -INFINITY, INFINITY, 3.4e38f, -3.4e38f};
	for (float x = 0.25f; x < 1e11f; x *= 1.00037f)
		for (float y : {x, -x, floorf(x), floorf(x) + 0.5f, -floorf(x)}) ps.push_back(y);
	for (uint32_t n : ns)
		for (float y : {(float)n, (float)n - 0.5f, nextafterf((float)n, 0.0f), nextafterf((float)n, 1e20f), (float)n - 1.0f}) ps.push_back(y);
	float* dp = nullptr;
	uint32_t* dn = nullptr;
	unsigned long long *bad = nullptr, count = ~0ull;
	if (cudaMalloc(&dp, ps.size() * 4) != cudaSuccess || cudaMalloc(&dn, ns.size() * 4) != cudaSuccess ||
	    cudaMalloc(&bad, sizeof(count)) != cudaSuccess || cudaMemset(bad, 0, sizeof(count)) != cudaSuccess ||
	    cudaMemcpy(dp, ps.data(), ps.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
	    cudaMemcpy(dn, ns.data(), ns.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess)
		return 2;
	const uint32_t work = (uint32_t)(ps.size() * ns.size());
	compare<<<(work + 255) / 256, 256>>>(dp, (uint32_t)ps.size(), dn, (uint32_t)ns.size(), bad);
	if (cudaMemcpy(&count, bad, sizeof(count), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
	std::printf("%llu values differ\n", count);
	return count == 0 ? 0 : 1;
}
