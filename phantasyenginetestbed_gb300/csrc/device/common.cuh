// Device helpers shared by the kernels: explicitly rounded FP32 arithmetic in the reference's
// operation order (sfz vector math, externals/sfzCore/include/sfz/math/Vector.inl), the device-side
// scene layout, PCG32 and the sampling sine/cosine. Every float operation that decides a hit or a
// sampled direction goes through __fadd_rn/__fsub_rn/__fmul_rn/__fdiv_rn/__fsqrt_rn, which the
// compiler never fuses, so results equal the host's IEEE single-precision results bit for bit.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "phe_gb300.h"

namespace phe_gb300 {

// ------------------------------------------------------------------------------------------------
// Device scene layout (built on upload from the reference arrays)
//
// nodes: 64 B per node, two 32-byte halves — (lo.x, lo.y, hi.x, hi.y) of child 0, then of child 1;
//        (lo.z, hi.z) of child 0, of child 1, then (child0, child1, count0, count1) with inner children
//        as node indices >= 0 and leaf children as ~firstSlot (< 0); count is 0 for inner children. The
//        box planes come in the pairs that the packed slab test consumes (traverse.cuh).
// tris:  48 B per slot, 3 x float4 — (p0.xyz, endMarker), (e2.x, e1.x, e2.y, e1.y), (e2.z, e1.z, 0, 0):
//        e1 = p1 - p0 and e2 = p2 - p0 interleaved, the operand pairs of the packed triangle test. e1
//        and e2 are the exact float subtractions Moller-Trumbore performs first, so storing them changes
//        no result bit. endMarker is -1 on the last slot of each leaf, else 0. (64 B with two 32-byte
//        loads took 1% longer: more sectors a leaf.)
// ------------------------------------------------------------------------------------------------

// nodes4 (optional): the same tree collapsed to 4-wide nodes, 128 B each — 6 float4 of child bounds
//        in SoA order (lo.x[4], lo.y[4], lo.z[4], hi.x[4], hi.y[4], hi.z[4]), one int4 of child refs
//        (4-wide node index >= 0, leaf ~firstSlot < 0, kEmptyChild for an unused slot) and one float4
//        of padding. Every child box is a box of the binary tree (a grandchild when the binary child
//        is inner), and it is built only when each grandchild box lies inside its parent box, so the
//        4-wide test of a grandchild passes only if the skipped binary test of its parent would pass.
// nodes8 / leaves8 (optional): the 8-wide compressed layout, 80 B per node and 32 B per leaf record
//        (format in host/wide8.hpp, traversal in traverse8.cuh).
// Textures of a scene: texels of texture k start at texels + offset (rows rowBytes apart, tightly
// packed); srgb[b] = powf(b / 255, 2.2) correctly rounded.
struct DeviceTexture {
	uint64_t offset;
	int32_t width, height;
	uint32_t bytesPerPixel, rowBytes;
};
static_assert(sizeof(DeviceTexture) == 24, "DeviceTexture is 24 bytes");

struct DeviceScene {
	const float4* nodes;
	const float4* tris;
	const phe_triangle_data* datas;
	const phe_material* materials;
	uint32_t numNodes, numSlots, numMaterials, numNodes4;
	const float4* nodes4;
	uint32_t* status;   // device word: OR of the error bits any kernel raised on this scene
	const DeviceTexture* textures;
	const uint8_t* texels;
	const float* srgb;
	uint32_t numTextures, pad;
	const uint4* nodes8;    // set only while the 8-wide layout is selected (host/wide8.hpp)
	const float4* leaves8;  // its leaf records
	uint32_t numNodes8, numLeaves8;
	float dirLimit;   // a ray direction with components up to this keeps every |det| below 2^126
	uint32_t pad2;
};
static_assert(sizeof(DeviceScene) == 128, "DeviceScene is 128 bytes");

constexpr int32_t kEmptyChild = 0x7FFFFFFE;

// Traversal stack depth: leaves of a valid scene are at most 64 levels deep, and a node pushes at
// most one entry per inner level, plus the sentinel.
constexpr int kStackSize = 68;
// 4-wide traversal: a node pushes up to 3 entries; a binary tree of depth <= 64 collapses to <= 32 levels.
constexpr int kStackSize4 = 100;
constexpr int32_t kSentinel = 0x7FFFFFFF;

// Error bits written to the per-launch status word.
constexpr uint32_t kErrStackOverflow = 1u;   // tested in the checked build (binary nodes), and in the wide traversals
constexpr uint32_t kErrBadIndex = 2u;   // checked build: a node or slot index outside its array

// The checked build (-DPHE_DEVICE_CHECKS=1, libphe_gb300_checked.so) tests every node and slot index a
// traversal is about to read against the array sizes; an index outside sets kErrBadIndex and ends that
// ray (no trap, no out-of-bounds access). The normal build relies on the host validation of the tree
// done at upload, and these tests compile away.
#ifndef PHE_DEVICE_CHECKS
#define PHE_DEVICE_CHECKS 0
#endif
constexpr bool kDeviceChecks = PHE_DEVICE_CHECKS != 0;
struct TraversalBounds {
	uint32_t numNodes;   // nodes of the layout being traversed (binary or 4-wide)
	uint32_t numSlots;
};

// Cache hints for data that is read or written once per launch (rays in, hits out, the frame's queues
// and contributions): with kStreamHints they use the evict-first ("streaming") cache policy, so these
// streams do not push scene nodes and triangles out of L2. Plain loads through the read-only path and
// plain stores otherwise.
#ifndef PHE_STREAM_HINTS
#define PHE_STREAM_HINTS 1
#endif
constexpr bool kStreamHints = PHE_STREAM_HINTS != 0;
template <class T>
__device__ __forceinline__ T ld_stream(const T* p)
{
	if constexpr (kStreamHints) return __ldcs(p);
	else return __ldg(p);
}
template <class T>
__device__ __forceinline__ void st_stream(T* p, T v)
{
	if constexpr (kStreamHints) __stcs(p, v);
	else *p = v;
}

struct f3 { float x, y, z; };

__device__ __forceinline__ f3 mk3(float x, float y, float z) { return f3{x, y, z}; }
__device__ __forceinline__ f3 add3(f3 a, f3 b) { return mk3(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)); }
__device__ __forceinline__ f3 sub3(f3 a, f3 b) { return mk3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)); }
__device__ __forceinline__ f3 mul3(f3 a, f3 b) { return mk3(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z)); }
__device__ __forceinline__ f3 muls3(f3 a, float s) { return mk3(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s)); }
__device__ __forceinline__ f3 divs3(f3 a, float s) { return mk3(__fdiv_rn(a.x, s), __fdiv_rn(a.y, s), __fdiv_rn(a.z, s)); }
__device__ __forceinline__ float dot3(f3 a, f3 b)
{
	return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ f3 cross3(f3 a, f3 b)
{
	return mk3(__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)), __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
	           __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float length3(f3 a) { return __fsqrt_rn(dot3(a, a)); }
__device__ __forceinline__ f3 normalize3(f3 a) { return divs3(a, length3(a)); }
// std::min / std::max semantics (b < a ? b : a / a < b ? b : a), including NaN behaviour.
__device__ __forceinline__ float stdmin(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float stdmax(float a, float b) { return (a < b) ? b : a; }

// ------------------------------------------------------------------------------------------------
// Packed FP32 pairs (sm_100 and later): one instruction adds or multiplies two floats, each lane rounded
// to nearest exactly as the scalar operation. The traversal kernels are bound by instruction issue, so
// the slab test and the triangle test use them: 258 M against 326 M warp instructions for 1M diffuse
// rays on 155K triangles, with the loops of traverse.cuh (271 M with a scalar triangle test in them).
// Products are summed by scalar additions: ptxas contracts a packed product that feeds a packed sum into
// one fused operation with a single rounding, whatever the rounding modifiers say (measured; a packed
// sum that feeds a packed product, and a scalar sum of unpacked products, are left alone).
// ------------------------------------------------------------------------------------------------
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi)
{
	f32x2 r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
	return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
	f32x2 r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
	f32x2 r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
// (a * b - c * d) of both lanes, lanes swapped: one component of two cross products.
__device__ __forceinline__ f32x2 cross_swapped(f32x2 a, f32x2 b, f32x2 c, f32x2 d)
{
	float p0, p1, n0, n1;
	unpack2(mul2(a, b), p0, p1);
	unpack2(mul2(c, d), n0, n1);
	return pack2(__fsub_rn(p1, n1), __fsub_rn(p0, n0));
}
// (ax * bx + ay * by) + az * bz of both lanes.
__device__ __forceinline__ void dot2(f32x2 ax, f32x2 bx, f32x2 ay, f32x2 by, f32x2 az, f32x2 bz, float& lo, float& hi)
{
	float x0, x1, y0, y1, z0, z1;
	unpack2(mul2(ax, bx), x0, x1);
	unpack2(mul2(ay, by), y0, y1);
	unpack2(mul2(az, bz), z0, z1);
	lo = __fadd_rn(__fadd_rn(x0, y0), z0);
	hi = __fadd_rn(__fadd_rn(x1, y1), z1);
}
// 32 bytes (aligned to 32) of data that no kernel writes, in one load.
__device__ __forceinline__ void ld32(const void* p, f32x2& a, f32x2& b, f32x2& c, f32x2& d)
{
	asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
}

// Slots allocated past the last one, so that a leaf's triangles can be loaded several at a time.
constexpr int kTriPadding = 3;

// One slot of `tris` as loaded.
struct TriSlot {
	float4 p0;          // p0.xyz, end marker
	f32x2 ex, ey, ez;   // (e2, e1) per axis
	__device__ __forceinline__ bool last() const { return p0.w < 0.0f; }
};
__device__ __forceinline__ TriSlot load_tri(const float4* __restrict__ tris, uint32_t slot)
{
	const float4* p = tris + 3 * (size_t)slot;
	TriSlot t;
	t.p0 = __ldg(p);
	asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(t.ex), "=l"(t.ey) : "l"(p + 1));
	asm("ld.global.nc.b64 %0, [%1];" : "=l"(t.ez) : "l"(p + 2));
	return t;
}

// ------------------------------------------------------------------------------------------------
// Moller-Trumbore with the reference's absolute determinant epsilon (Intersection.hpp:24-67,
// RayCastKernel.cu:96-131), on a slot stored as (p0, e1, e2). Returns true on a hit.
//
// Every quantity is computed with the reference's operations and rounding; only the control flow
// differs. The reference returns early after the determinant, u and v tests; here all of u, v and t
// are computed and the same three tests are combined into one predicate, so a rejected triangle gives
// the same answer. In a warp the early returns saved little (the warp runs until its last lane
// rejects), while the straight-line form has no branches and overlaps the reciprocal with the other
// products. f = rn(1 / det) is taken as the correctly rounded reciprocal, the same value as the
// correctly rounded quotient 1.0f / det.
//
// FAST: |det| < 2^126 is known (DeviceScene::dirLimit), so the reciprocal needs no range check: the
// hardware approximation and one Newton-Raphson step with fused residual, which Markstein (IBM J. Res.
// Dev. 34, 1990) shows to round correctly up to cases that enumeration settles; all 2^32 floats were
// compared with __frcp_rn (tests/cpp/reciprocal_test.cu). A |det| below the epsilon is rejected whatever f is.
// 1M diffuse rays on 155K triangles take 314 us with it, 326 with __frcp_rn.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ float reciprocal_in_range(float x)
{
	float r;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
	return __fmaf_rn(r, __fmaf_rn(-x, r, 1.0f), r);
}

template <bool FAST>
__device__ __forceinline__ bool intersect_tri(const TriSlot& tri, f3 o, f3 d, float& t, float& u, float& v)
{
	const float EPS = 0.00001f;
	const f3 s = mk3(__fsub_rn(o.x, tri.p0.x), __fsub_rn(o.y, tri.p0.y), __fsub_rn(o.z, tri.p0.z));
	// (r, q) = (s x e1, d x e2), then their products with e and with (d, s)
	const f32x2 dsx = pack2(d.x, s.x), dsy = pack2(d.y, s.y), dsz = pack2(d.z, s.z);
	const f32x2 rqx = cross_swapped(dsy, tri.ez, dsz, tri.ey);
	const f32x2 rqy = cross_swapped(dsz, tri.ex, dsx, tri.ez);
	const f32x2 rqz = cross_swapped(dsx, tri.ey, dsy, tri.ex);
	float det, tt, su, dv;
	dot2(tri.ex, rqx, tri.ey, rqy, tri.ez, rqz, tt, det);   // e2 . r, e1 . q
	dot2(dsx, rqx, dsy, rqy, dsz, rqz, dv, su);             // d . r, s . q
	const float f = FAST ? reciprocal_in_range(det) : __frcp_rn(det);
	u = __fmul_rn(f, su);
	v = __fmul_rn(f, dv);
	t = __fmul_rn(f, tt);
	return !(fabsf(det) < EPS) && !(u < 0.0f) && !(v < 0.0f || __fadd_rn(u, v) > 1.0f);
}

// ------------------------------------------------------------------------------------------------
// PCG32 (O'Neill 2014), identical to the host generator (host/pcg.hpp).
// ------------------------------------------------------------------------------------------------
struct DevPcg {
	uint64_t state, inc;
	__device__ __forceinline__ uint32_t next()
	{
		uint64_t old = state;
		state = old * 6364136223846793005ull + inc;
		uint32_t xorshifted = (uint32_t)(((old >> 18u) ^ old) >> 27u);
		uint32_t rot = (uint32_t)(old >> 59u);
		return (xorshifted >> rot) | (xorshifted << ((32u - rot) & 31u));
	}
	__device__ __forceinline__ void seed(uint64_t initstate, uint64_t initseq)
	{
		state = 0u;
		inc = (initseq << 1u) | 1u;
		next();
		state += initstate;
		next();
	}
	__device__ __forceinline__ float uniform() { return __fmul_rn((float)(next() >> 8), 0x1.0p-24f); }
};

// Stream of pixel `pixel` for shading stage `stage` of frame `frame`.
__device__ __forceinline__ void pixel_stream(DevPcg& r, uint64_t seed, uint32_t frame, uint32_t pixel, uint32_t stage)
{
	uint64_t initstate = seed ^ ((uint64_t)frame * 0x9E3779B97F4A7C15ull);
	uint64_t initseq = ((uint64_t)pixel << 2) | (uint64_t)(stage & 3u);
	r.seed(initstate, initseq);
}

// sin(2 pi r), cos(2 pi r) for r in [0, 1): exact quadrant reduction, then Taylor polynomials of
// degree 9 (sine) and 10 (cosine) on [0, pi/4] evaluated in Horner form with single roundings.
// Truncation error below 2e-9; the host restatement performs the same operations.
__device__ __forceinline__ void sincos_2pi(float r, float& s, float& c)
{
	float q = __fmul_rn(r, 4.0f);
	int k = (int)q;
	k = k > 3 ? 3 : (k < 0 ? 0 : k);
	float f = __fsub_rn(q, (float)k);
	bool swap = f > 0.5f;
	float g = swap ? __fsub_rn(1.0f, f) : f;
	float x = __fmul_rn(g, 0x1.921fb6p+0f);
	float x2 = __fmul_rn(x, x);
	float sp = __fmul_rn(x, __fadd_rn(1.0f, __fmul_rn(x2, __fadd_rn(-0x1.555556p-3f, __fmul_rn(x2, __fadd_rn(0x1.111112p-7f,
	                         __fmul_rn(x2, __fadd_rn(-0x1.a01a02p-13f, __fmul_rn(x2, 0x1.71de3ap-19f)))))))));
	float cp = __fadd_rn(1.0f, __fmul_rn(x2, __fadd_rn(-0x1.0p-1f, __fmul_rn(x2, __fadd_rn(0x1.555556p-5f,
	                         __fmul_rn(x2, __fadd_rn(-0x1.6c16c2p-10f, __fmul_rn(x2, __fsub_rn(0x1.a01a02p-16f,
	                         __fmul_rn(x2, 0x1.27e4fcp-22f))))))))));
	float sq = swap ? cp : sp;
	float cq = swap ? sp : cp;
	switch (k) {
	case 0: s = sq; c = cq; break;
	case 1: s = cq; c = -sq; break;
	case 2: s = -sq; c = -cq; break;
	default: s = -cq; c = sq; break;
	}
}

} // namespace phe_gb300
