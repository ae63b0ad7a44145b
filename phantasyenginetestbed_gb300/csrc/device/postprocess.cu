// Display post-process for headless image dumps: the Uncharted 2 filmic tonemap followed by gamma
// correction (resources/shaders/gamma_correction.frag:20-74, the combination its main() selects), from
// a linear float RGBA image to display-referred float RGBA and/or 8-bit RGBA. The GL pass drew into a
// window; here the result is a device buffer the caller copies out (or writes to a file).

#include "filmic.cuh"
#include "runtime.cuh"
#include "sampling.cuh"

namespace phe_gb300 {

__device__ __forceinline__ unsigned char to_byte(float v)
{
	return (unsigned char)__float2int_rn(__fmul_rn(fminf(fmaxf(v, 0.0f), 1.0f), 255.0f));
}

// Bound by instruction issue, most of it powf (337 warp instructions for 32 pixels at 3.5 of 4 per cycle, 23 us at
// 1080p; 378 and 26 us with the compiler's divisions), not by its 16 + 16 bytes a pixel.
__global__ void postprocess_kernel(uint32_t n, const float4* __restrict__ linear, float invGamma,
                                   float4* __restrict__ display, uchar4* __restrict__ rgba8)
{
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	float4 c = linear[i];
	const float BLACK_CRUSH = 0.0015f, exposureBias = 2.0f;
	float v[3] = {c.x, c.y, c.z};
	for (int k = 0; k < 3; k++) {
		float x = __fmul_rn(exposureBias, fmaxf(0.0f, __fsub_rn(v[k], BLACK_CRUSH)));
		v[k] = powf(filmic_over_white(x), invGamma);
	}
	if (display) display[i] = make_float4(v[0], v[1], v[2], c.w);
	if (rgba8) {
		unsigned char q[4];
		float a[4] = {v[0], v[1], v[2], c.w};
		for (int k = 0; k < 4; k++) q[k] = to_byte(a[k]);
		rgba8[i] = make_uchar4(q[0], q[1], q[2], q[3]);
	}
}

// scaling.frag:19-35 for destination pixel (x, y): uv at the pixel centre, coord = uv * viewport / src,
// four GL_LINEAR taps at +-1/4 destination pixel, averaged; alpha 1.
//
// The four taps are two columns by two rows of positions, and down a destination column the rows' source
// texels never go back. So a warp takes 32 columns and walks ROWS rows: a thread keeps the source
// rows of the current tap, each already filtered along x at both columns, and loads and filters a source
// row once for all the taps and destination rows that use it, instead of 16 texels a pixel; the rows'
// and the columns' positions come from tables that the block computes once, and the filters run on pairs of
// floats. 1920x1080 to 2560x1440: 64 us (56.7 M warp instructions, 16 x 4 one-float loads a pixel) before, 31 (22.4 M)
// with scalar filters and the columns computed by every warp, 28 (17.5 M) now, with 8 rows a warp (4: 2 us longer, 16: the same).
//
// A small image has too few warps at 8 rows each: a warp takes 1, 2, 4 or 8 rows, as many as leave 20 warps an SM.
// Tonemap and scaling of 640x360 to 300x200 / 640x360 / 901x503 / 1280x720 at 1, 2, 4 and 8 rows: 10.4 12.4 13.3 16.5 /
// 12.5 12.4 12.4 14.5 / 14.5 13.6 12.4 14.5 / 18.6 16.5 14.5 14.8 us (12.4 / 15.5 / 18.6 / 28.8 with 16 loads a pixel).
constexpr int kScaleWarps = 8, kScaleWarpsPerSM = 20;

struct ScaledRow {   // a source row filtered along x at the left and the right column: (x, y) of each, both z
	f32x2 l, r, z;
};
// glsl_mix of both lanes, with the weights (w1, w1) = 1 - t and (w2, w2) = t.
__device__ __forceinline__ f32x2 mix2(f32x2 a, f32x2 b, f32x2 w1, f32x2 w2)
{
	float a0, a1, b0, b1;
	unpack2(mul2(a, w1), a0, a1);
	unpack2(mul2(b, w2), b0, b1);
	return pack2(__fadd_rn(a0, b0), __fadd_rn(a1, b1));
}
template <bool VEC>
__device__ __forceinline__ ScaledRow scaled_row(const float4* __restrict__ src, uint32_t W, uint32_t row, const LinearAxis& xl,
                                                const LinearAxis& xr)
{
	const float4* p = src + (size_t)row * W;
	const float4 a = ld_texel<VEC>(p + xl.i0), b = ld_texel<VEC>(p + xl.i1);
	const float4 c = ld_texel<VEC>(p + xr.i0), d = ld_texel<VEC>(p + xr.i1);
	const float wl = __fsub_rn(1.0f, xl.a), wr = __fsub_rn(1.0f, xr.a);
	ScaledRow o;
	o.l = mix2(pack2(a.x, a.y), pack2(b.x, b.y), pack2(wl, wl), pack2(xl.a, xl.a));
	o.r = mix2(pack2(c.x, c.y), pack2(d.x, d.y), pack2(wr, wr), pack2(xr.a, xr.a));
	o.z = pack2(glsl_mix(a.z, b.z, xl.a), glsl_mix(c.z, d.z, xr.a));
	return o;
}

template <bool VEC, int ROWS>
__global__ void __launch_bounds__(32 * kScaleWarps)
scale_kernel(uint32_t srcW, uint32_t srcH, const float4* __restrict__ src, float vpW, float vpH, uint32_t dstW, uint32_t dstH,
             float4* __restrict__ dst, uchar4* __restrict__ rgba8)
{
	constexpr int kTile = ROWS * kScaleWarps;   // rows of a block
	static_assert(kTile <= 32 * (kScaleWarps - 1), "the last warp fills the columns' table");
	// the taps of the block's rows and columns, each computed once
	__shared__ LinearAxis rowTop[kTile], rowBottom[kTile], colLeft[32], colRight[32];
	const uint32_t x = blockIdx.x * 32u + threadIdx.x;
	const uint32_t yBlock = blockIdx.y * kTile, yFirst = yBlock + threadIdx.y * ROWS;
	const uint32_t yEnd = min(dstH, yFirst + ROWS);
	const uint32_t t = threadIdx.y * 32u + threadIdx.x;
	if (t < kTile) {
		const float dh = (float)dstH, sh = (float)srcH, oy = __fmul_rn(__fdiv_rn(1.0f, dh), 0.25f);
		const float cy = __fdiv_rn(__fmul_rn(__fdiv_rn(__fadd_rn((float)(yBlock + t), 0.5f), dh), vpH), sh);
		rowTop[t] = linear_axis(__fmul_rn(__fadd_rn(cy, -oy), sh), srcH);
		rowBottom[t] = linear_axis(__fmul_rn(__fadd_rn(cy, oy), sh), srcH);
	} else if (threadIdx.y == kScaleWarps - 1) {
		// columns beyond the last repeat it, so that the warps stay whole; their lanes store nothing
		const float dw = (float)dstW, sw = (float)srcW, ox = __fmul_rn(__fdiv_rn(1.0f, dw), 0.25f);
		const float cx = __fdiv_rn(__fmul_rn(__fdiv_rn(__fadd_rn((float)min(x, dstW - 1), 0.5f), dw), vpW), sw);
		colLeft[threadIdx.x] = linear_axis(__fmul_rn(__fadd_rn(cx, -ox), sw), srcW);
		colRight[threadIdx.x] = linear_axis(__fmul_rn(__fadd_rn(cx, ox), sw), srcW);
	}
	__syncthreads();
	const LinearAxis xl = colLeft[threadIdx.x], xr = colRight[threadIdx.x];
	// source rows held in r0 and r1 (none yet)
	uint32_t have0 = 0xFFFFFFFFu, have1 = 0xFFFFFFFFu;
	ScaledRow r0{}, r1{};
	auto need = [&](uint32_t y0, uint32_t y1) {   // the same for every lane
		if (have0 != y0) {
			r0 = have1 == y0 ? r1 : scaled_row<VEC>(src, srcW, y0, xl, xr);
			have0 = y0;
		}
		if (have1 != y1) {
			r1 = y1 == y0 ? r0 : scaled_row<VEC>(src, srcW, y1, xl, xr);
			have1 = y1;
		}
	};
	for (uint32_t y = yFirst; y < yEnd; y++) {
		const LinearAxis yt = rowTop[y - yBlock], yb = rowBottom[y - yBlock];
		f3 acc;
		auto tap = [&](float t, bool first) {
			const float u = __fsub_rn(1.0f, t);
			const f32x2 w1 = pack2(u, u), w2 = pack2(t, t);
			float lx, ly, rx, ry, lz, rz;
			unpack2(mix2(r0.l, r1.l, w1, w2), lx, ly);
			unpack2(mix2(r0.r, r1.r, w1, w2), rx, ry);
			unpack2(mix2(r0.z, r1.z, w1, w2), lz, rz);
			const f3 l = mk3(lx, ly, lz);
			acc = add3(first ? l : add3(acc, l), mk3(rx, ry, rz));
		};
		need(yt.i0, yt.i1);
		tap(yt.a, true);
		need(yb.i0, yb.i1);
		tap(yb.a, false);
		const float4 o = make_float4(__fmul_rn(acc.x, 0.25f), __fmul_rn(acc.y, 0.25f), __fmul_rn(acc.z, 0.25f), 1.0f);
		if (x >= dstW) continue;
		const size_t p = (size_t)y * dstW + x;
		if (dst) dst[p] = o;
		if (rgba8) rgba8[p] = make_uchar4(to_byte(o.x), to_byte(o.y), to_byte(o.z), 255);
	}
}

} // namespace phe_gb300

using namespace phe_gb300;

extern "C" phe_status phe_scale(uint32_t srcW, uint32_t srcH, const float* src, uint32_t viewportW, uint32_t viewportH,
                                uint32_t dstW, uint32_t dstH, float* dst, uint8_t* dstRgba8, void* stream)
{
	if (!src || (!dst && !dstRgba8)) return fail(PHE_ERR_INVALID_ARGUMENT, "phe_scale: null buffer");
	if (!srcW || !srcH || !viewportW || !viewportH || viewportW > srcW || viewportH > srcH)
		return fail(PHE_ERR_INVALID_ARGUMENT, "phe_scale: viewport must be a non-empty part of the source");
	if (srcW > 65536 || srcH > 65536 || dstW > 65536 || dstH > 65536)
		return fail(PHE_ERR_TOO_LARGE, "phe_scale: images are limited to 65536 x 65536");
	if (!dstW || !dstH) return PHE_OK;
	int dev = 0, numSMs = 0;
	PHE_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
	PHE_CUDA_TRY(cudaDeviceGetAttribute(&numSMs, cudaDevAttrMultiProcessorCount, dev), "SM count");
	// rows of a warp: as many as leave kScaleWarpsPerSM warps an SM
	const uint64_t strips = (uint64_t)((dstW + 31) / 32) * dstH;   // rows of 32 columns
	int k = 0;
	while (k < 3 && strips >> (k + 1) >= (uint64_t)kScaleWarpsPerSM * (uint32_t)numSMs) k++;
	const bool vec = !((uintptr_t)src & 15u);   // src may be aligned to floats only
	using Kernel = decltype(&scale_kernel<true, 1>);
	static constexpr Kernel kernels[2][4] = {
		{scale_kernel<false, 1>, scale_kernel<false, 2>, scale_kernel<false, 4>, scale_kernel<false, 8>},
		{scale_kernel<true, 1>, scale_kernel<true, 2>, scale_kernel<true, 4>, scale_kernel<true, 8>}};
	const uint32_t tile = (uint32_t)kScaleWarps << k;
	kernels[vec][k]<<<dim3((dstW + 31) / 32, (dstH + tile - 1) / tile), dim3(32, kScaleWarps), 0, (cudaStream_t)stream>>>(
		srcW, srcH, (const float4*)src, (float)viewportW, (float)viewportH, dstW, dstH, (float4*)dst, (uchar4*)dstRgba8);
	PHE_CUDA_TRY(cudaGetLastError(), "scale_kernel launch");
	return PHE_OK;
}

extern "C" phe_status phe_postprocess(uint32_t resX, uint32_t resY, const float* linear, float gamma, float* display,
                                      uint8_t* rgba8, void* stream)
{
	if (!linear || (!display && !rgba8)) return fail(PHE_ERR_INVALID_ARGUMENT, "phe_postprocess: null buffer");
	if (!(gamma > 0.0f)) return fail(PHE_ERR_INVALID_ARGUMENT, "phe_postprocess: gamma must be positive");
	uint64_t n = (uint64_t)resX * resY;
	if (n == 0) return PHE_OK;
	if (n > 0xFFFFFFFFull) return fail(PHE_ERR_TOO_LARGE, "phe_postprocess: too many pixels");
	uint32_t grid = (uint32_t)((n + 255) / 256);
	postprocess_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((uint32_t)n, (const float4*)linear, 1.0f / gamma,
	                                                          (float4*)display, (uchar4*)rgba8);
	PHE_CUDA_TRY(cudaGetLastError(), "postprocess_kernel launch");
	return PHE_OK;
}
