// GL-style sampling of float images in device memory, restated with explicit rounding so that the
// oracle reproduces it: GLSL mix() and GL_LINEAR filtering with clamp-to-edge addressing (the
// framebuffer textures of the reference's post-process passes, sfz/gl/Framebuffer.cpp:292-304).
#pragma once

#include <cstdint>

namespace phe_gb300 {

// GLSL mix(a, b, t) = a * (1 - t) + b * t
__device__ __forceinline__ float glsl_mix(float a, float b, float t)
{
	return __fadd_rn(__fmul_rn(a, __fsub_rn(1.0f, t)), __fmul_rn(b, t));
}

// One axis of GL_LINEAR with clamp to edge: the two texels around pixel-space position p (texel centres at
// integer + 0.5) of n (1 to 2^32 - 1), and the weight of the second.
struct LinearAxis {
	uint32_t i0, i1;
	float a;
};
__device__ __forceinline__ LinearAxis linear_axis(float p, uint32_t n)
{
	const float f = __fsub_rn(p, 0.5f), f0 = floorf(f);
	const uint32_t m = n - 1;
	LinearAxis r;
	r.a = __fsub_rn(f, f0);
	r.i0 = min(__float2uint_rz(f0), m);   // the conversion saturates: 0 below the first texel
	r.i1 = min(r.i0 + (f0 >= 0.0f ? 1u : 0u), m);
	return r;
}

__device__ __forceinline__ float2 glsl_mix(float2 a, float2 b, float t) { return make_float2(glsl_mix(a.x, b.x, t), glsl_mix(a.y, b.y, t)); }
__device__ __forceinline__ float4 glsl_mix(float4 a, float4 b, float t)
{
	return make_float4(glsl_mix(a.x, b.x, t), glsl_mix(a.y, b.y, t), glsl_mix(a.z, b.z, t), glsl_mix(a.w, b.w, t));
}

// One texel of a float2 or float4 image: one load when the image is aligned to its texels (VEC), one per
// channel for an image that is only aligned to floats.
template <bool VEC>
__device__ __forceinline__ float4 ld_texel(const float4* p)
{
	if constexpr (VEC) return __ldg(p);
	const float* f = reinterpret_cast<const float*>(p);
	return make_float4(__ldg(f), __ldg(f + 1), __ldg(f + 2), __ldg(f + 3));
}
template <bool VEC>
__device__ __forceinline__ float2 ld_texel(const float2* p)
{
	if constexpr (VEC) return __ldg(p);
	const float* f = reinterpret_cast<const float*>(p);
	return make_float2(__ldg(f), __ldg(f + 1));
}

// The four texels of a GL_LINEAR fetch of a float2 or float4 image W texels wide.
template <bool VEC, class T>
struct LinearTexels {
	T t00, t10, t01, t11;
	__device__ __forceinline__ LinearTexels(const T* __restrict__ tex, uint32_t W, const LinearAxis& x, const LinearAxis& y)
	{
		const T *r0 = tex + (size_t)y.i0 * W, *r1 = tex + (size_t)y.i1 * W;
		t00 = ld_texel<VEC>(r0 + x.i0);
		t10 = ld_texel<VEC>(r0 + x.i1);
		t01 = ld_texel<VEC>(r1 + x.i0);
		t11 = ld_texel<VEC>(r1 + x.i1);
	}
	__device__ __forceinline__ T mix(float ax, float ay) const
	{
		return glsl_mix(glsl_mix(t00, t10, ax), glsl_mix(t01, t11, ax), ay);
	}
};

} // namespace phe_gb300
