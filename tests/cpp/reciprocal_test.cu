// Compares the traversal's reciprocal (reciprocal_in_range, csrc/device/common.cuh) with __frcp_rn on every float
// whose magnitude a determinant can have there: from the rejection epsilon to 2^126. Prints the count of
// differing values; exits 0 when there are none.
#include <cstdio>

#include "common.cuh"

__global__ void compare(unsigned long long* bad)
{
	const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
	for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += stride) {
		const float x = __uint_as_float((uint32_t)i);
		if (!(fabsf(x) >= 1e-5f && fabsf(x) < 0x1p126f)) continue;
		if (__float_as_uint(phe_gb300::reciprocal_in_range(x)) != __float_as_uint(__frcp_rn(x))) atomicAdd(bad, 1ull);
	}
}

int main()
{
	unsigned long long* bad = nullptr;
	unsigned long long n = ~0ull;
	if (cudaMalloc(&bad, sizeof(n)) != cudaSuccess || cudaMemset(bad, 0, sizeof(n)) != cudaSuccess) return 2;
	compare<<<1024, 256>>>(bad);
	if (cudaMemcpy(&n, bad, sizeof(n), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
	std::printf("%llu values differ\n", n);
	return n == 0 ? 0 : 1;
}
