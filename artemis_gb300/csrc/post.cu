/*
 * post.cu -- what follows the accumulated frame: HDR -> LDR tonemapping and
 * an AOV-guided denoiser.
 *
 * Tonemapping follows include/cuda/color.cuh of the reference: aces()
 * (:33-39), srgb() (:13-30), quantize_unsigned_8_bits() (:42-55),
 * make_color() (:57-66) and cast.cuh to_ui32() (:16-20), with the vertical
 * flip of hdr_to_ldr_kernel (:84-103).  ACES is plain IEEE arithmetic and
 * matches the reference bit for bit; sRGB calls powf, whose last bit can
 * differ from the host C library's.
 *
 * The reference denoises with the OptiX AI denoiser (source/layers/
 * denoiser.cu:9-149), a closed library; this is a filter of its own: the
 * edge-avoiding a-trous wavelet transform (Dammertz et al., "Edge-Avoiding
 * A-Trous Wavelet Transform for fast Global Illumination Filtering", HPG
 * 2010).  Pass i (i = 0 .. iterations-1) convolves with the 5 x 5 B3-spline
 * kernel (1/16, 1/4, 3/8, 1/4, 1/16 in each direction) spread by a step of
 * 2^i pixels, each tap weighted by three edge-stopping functions between the
 * centre p and the tap q:
 *   colour    exp(-|l_p - l_q| / (sigma_color 2^-i (l_p + l_q) / 2 + 1e-4)),
 *             l = luminance of the demodulated value (relative, so HDR
 *             radiance of any scale filters the same way)
 *   normal    max(0, n_p . n_q) ^ normal_power
 *   position  exp(-d / sigma_position), d = |n_p . (x_q - x_p)| / |x_q - x_p|,
 *             the distance of q off p's tangent plane per unit of separation
 *             (scale free)
 * With the albedo guide the filter works on colour / albedo' (albedo'
 * = albedo where a channel exceeds 1e-3, else 1) and multiplies back at the
 * end, so texture and material detail is not blurred.  Pixels without a hit
 * (zero normal) only average among themselves.
 */
#include <float.h>

#include "kgr_post.h"

namespace kgr {

namespace {

__device__ __forceinline__ float clamp_ref(float f, float a, float b) { return fmaxf(a, fminf(f, b)); }

/* aces (color.cuh:33-39) */
__device__ __forceinline__ float aces1(float c)
{
	float a = c * (c * 2.51f + 0.03f);
	float b = c * (c * 2.43f + 0.59f) + 0.14f;
	return clamp_ref(a / b, 0.0f, 1.0f);
}

/* srgb (color.cuh:13-30) */
__device__ __forceinline__ float srgb1(float c)
{
	float powed = powf(c, 1.0f / 2.4f);
	float s = c < 0.0031308f ? 12.92f * c : 1.055f * powed - 0.055f;
	return clamp_ref(s, 0.0f, 1.0f);
}

/* quantize_unsigned_8_bits (color.cuh:42-55) */
__device__ __forceinline__ uint32_t quantize8(float x)
{
	x = clamp_ref(x, 0.0f, 1.0f);
	uint32_t q = (uint32_t)(x * 256.0f);
	return q < 255u ? q : 255u;
}

__global__ void tonemap_kernel(const float4 *__restrict__ hdr, uint32_t *__restrict__ ldr, uint32_t width,
		uint32_t height, int mode)
{
	uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
	uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
	if (x >= width || y >= height)
		return;
	float4 c = hdr[(size_t)y * width + x];
	float r, g, b;
	if (mode == KGR_TONEMAP_ACES) {
		r = aces1(c.x);
		g = aces1(c.y);
		b = aces1(c.z);
	} else {
		r = srgb1(c.x);
		g = srgb1(c.y);
		b = srgb1(c.z);
	}
	/* to_ui32 (cast.cuh:16-20): alpha 255 in the top byte, red in the lowest */
	uint32_t v = (255u << 24) | (quantize8(b) << 16) | (quantize8(g) << 8) | quantize8(r);
	ldr[(size_t)(height - y - 1) * width + x] = v;
}

__device__ __forceinline__ float lum(float3 c) { return 0.2126f * c.x + 0.7152f * c.y + 0.0722f * c.z; }

__device__ __forceinline__ float3 f3of(float4 v) { return make_float3(v.x, v.y, v.z); }

__device__ __forceinline__ float dot3(float3 a, float3 b)
{
	return __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, a.z * b.z));
}

/* 1 / x to an ulp, over the whole range (__fdividef gives 0 above 2^126) */
__device__ __forceinline__ float rcp(float x)
{
	float r;
	asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
	return r;
}

/* a / b, within an ulp: the product with the reciprocal and what its residual
 * a - b q (exact in a fused operation; Markstein 1990) adds to it.  Where the
 * residual is not a number the product is 0 or infinite already, as the
 * quotient is. */
__device__ __forceinline__ float quotient(float a, float b)
{
	const float r = rcp(b), q = a * r;
	const float t = __fmaf_rn(__fmaf_rn(-b, q, a), r, q);
	return t == t ? t : q;
}

/* a / sqrt(x), within two ulp, x > 0: a step of Newton's iteration on the
 * reciprocal root.  A residual that is not a number (x infinite, r 0) counts
 * as 1. */
__device__ __forceinline__ float over_root(float a, float x)
{
	const float r = rsqrtf(x), q = a * r;
	const float h = fminf(__fmaf_rn(-x * r, r, 1.0f), 1.0f);
	return __fmaf_rn(q * 0.5f, h, q);
}

__device__ __forceinline__ float3 albedo_div(float4 a)
{
	return make_float3(a.x > 1e-3f ? a.x : 1.0f, a.y > 1e-3f ? a.y : 1.0f, a.z > 1e-3f ? a.z : 1.0f);
}

/* c ^ (2 ^ n) to within an ulp, c >= 0: each squaring keeps its rounding error,
 * and the last rounds once (into the denormal numbers too).  Above the largest
 * float the errors are not numbers: infinity then. */
__device__ __forceinline__ float squared(float c, int n)
{
	float lo = 0.0f;
#pragma unroll
	for (int q = 1; q < n; q++) {
		const float sq = c * c, e = __fmaf_rn(c, c, -sq);
		lo = q == 1 ? e : __fmaf_rn(c + c, lo, e);
		c = sq;
	}
	return n ? fminf(__fmaf_rn(c, c, (c + c) * lo), INFINITY) : c;
}

/* 3/8, 1/4, 1/16 at 0, 1, 2 */
__device__ __forceinline__ float spline(int d)
{
	return d == 0 ? 0.375f : (d == 1 || d == -1 ? 0.25f : 0.0625f);
}

/* colour / albedo' before the first pass.  in and out may be the same buffer:
 * a thread reads and writes its own pixel only. */
__global__ void demodulate_kernel(const float4 *in, const float4 *__restrict__ albedo, float4 *out, uint32_t n)
{
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	float4 c = in[i];
	float3 d = albedo_div(albedo[i]);
	out[i] = make_float4(c.x / d.x, c.y / d.y, c.z / d.z, c.w);
}

/* How a pass raises the normal cosine to its power: the default 64 and other
 * powers of two by squaring (the default's chain unrolled), anything else by
 * powf. */
enum { POWER_NONE = 0, POWER_SQUARES = 1, POWER_ANY = 2, POWER_64 = 3 };

struct AtrousPass {
	uint32_t width, height;
	int step;
	float half_sigma;    /* sigma_color 2^-i / 2 */
	float position_rate; /* 1 / sigma_position, finite */
	float normal_power;
	int squarings;       /* POWER_64, POWER_SQUARES: normal_power = 2^squarings */
	int remodulate;      /* the last pass of an albedo-guided filter */
};

/* The centre of a filter and its sums. */
struct AtrousPixel {
	int x, y;
	bool hit;
	float3 n, pos, sum;
	float l, wsum;
};

/* The 25 taps of one pixel.  No branch on a loaded value lies between a row's
 * loads and its sums, so that they go out together. */
template <int POWER, bool POSITION>
__device__ __forceinline__ void atrous_taps(AtrousPixel &p, const float4 *__restrict__ in,
		const float4 *__restrict__ normal, const float4 *__restrict__ position, const AtrousPass &ps)
{
	const int width = (int)ps.width, height = (int)ps.height, step = ps.step;
#pragma unroll 1
	for (int dy = -2; dy <= 2; dy++) {
		const int qy = p.y + dy * step;
		if (qy < 0 || qy >= height)
			continue;
#pragma unroll
		for (int dx = -2; dx <= 2; dx++) {
			const int qx = p.x + dx * step;
			if (qx < 0 || qx >= width)
				continue;
			const size_t iq = (size_t)qy * width + qx;
			const float3 cq = f3of(in[iq]);
			const float3 nq = f3of(normal[iq]);
			const float3 xq = POSITION ? f3of(position[iq]) : p.pos;
			/* not all zero (of either sign) */
			const bool hit_q = ((__float_as_uint(nq.x) | __float_as_uint(nq.y) | __float_as_uint(nq.z)) << 1) != 0u;
			const float lq = lum(cq);
			float w = spline(dx) * spline(dy) *
				expf(-quotient(fabsf(p.l - lq), __fmaf_rn(ps.half_sigma, p.l + lq, 1e-4f)));
			if (p.hit) {
				if (POWER != POWER_NONE) {
					float c = fmaxf(p.n.x * nq.x + p.n.y * nq.y + p.n.z * nq.z, 0.0f);
					w *= POWER == POWER_ANY ? powf(c, ps.normal_power) : squared(c, POWER == POWER_64 ? 6 : ps.squarings);
				}
				if (POSITION && (dx != 0 || dy != 0)) {
					float3 v = make_float3(xq.x - p.pos.x, xq.y - p.pos.y, xq.z - p.pos.z);
					float len2 = dot3(v, v);
					float d = len2 > 0.0f ? over_root(fabsf(dot3(p.n, v)), len2) : 0.0f;
					w *= expf(-d * ps.position_rate);
				}
			}
			/* a tap of the other kind adds nothing, whatever its colour */
			if (p.hit == hit_q) {
				p.sum.x = __fmaf_rn(w, cq.x, p.sum.x);
				p.sum.y = __fmaf_rn(w, cq.y, p.sum.y);
				p.sum.z = __fmaf_rn(w, cq.z, p.sum.z);
				p.wsum += w;
			}
		}
	}
}

/* One a-trous pass, one pixel a thread.
 *
 * Bound by the arithmetic of a tap (issue slots 87% busy, L1 39%, DRAM 12%).  Every step of a weight is good to an ulp or two, but cheaper than
 * its general form: quotients from the MUFU's reciprocal and a residual, a
 * Newton step on the reciprocal root, squarings that carry their error for the
 * power of two, fused sums.  One loop for every pixel: normals that are means
 * of several samples' give weights down to the denormal numbers, whose result
 * hangs on the roundings, and the three weights are multiplied in this order
 * because the power may leave only a few bits of one.
 *
 * 1080p, five passes, every guide, behind 1 and 4 samples a pixel on the
 * terrain, then on the box scene: 1785, 1722, 2350, 2146 us with divisions,
 * powf and a demodulation of every tap (demodulate_kernel has taken that out),
 * now 847, 851, 1030, 1030; the error against 64 bits is 0.96 to 1.00 of what
 * it was.  Bare MUFU results, plain squarings (32 ulp) and a second loop for
 * averaged normals took 781, 1553, 908, 2332 us and left a weight several
 * times the error.  Two pixels of a column a thread, which halves the loads, were no
 * faster; packed operations on two taps (f32x2) 15% slower; all 25 taps
 * unrolled 840 to 930 us where this loop took 781, waiting for instructions; a
 * branch past the loads of a tap of the other kind 900; 8, 9, 11 and 12 blocks
 * an SM 1 to 5% slower. */
template <int POWER, bool POSITION>
__global__ void __launch_bounds__(128, 10) atrous_kernel(const float4 *__restrict__ in, float4 *__restrict__ out,
		const float4 *__restrict__ normal, const float4 *__restrict__ albedo, const float4 *__restrict__ position,
		AtrousPass ps)
{
	AtrousPixel p;
	p.x = (int)(blockIdx.x * 32 + threadIdx.x);
	p.y = (int)((blockIdx.z * gridDim.y + blockIdx.y) * 4 + threadIdx.y);
	if (p.x >= (int)ps.width || p.y >= (int)ps.height)
		return;
	const size_t ip = (size_t)p.y * ps.width + p.x;
	p.n = f3of(normal[ip]);
	p.hit = p.n.x != 0.0f || p.n.y != 0.0f || p.n.z != 0.0f;
	p.pos = POSITION ? f3of(position[ip]) : make_float3(0.0f, 0.0f, 0.0f);
	const float4 c = in[ip];
	p.l = lum(f3of(c));
	p.sum = make_float3(0.0f, 0.0f, 0.0f);
	p.wsum = 0.0f;
	atrous_taps<POWER, POSITION>(p, in, normal, position, ps);
	float3 r = p.wsum > 0.0f ? make_float3(p.sum.x / p.wsum, p.sum.y / p.wsum, p.sum.z / p.wsum) : f3of(c);
	if (ps.remodulate) {
		float3 d = albedo_div(albedo[ip]);
		r = make_float3(r.x * d.x, r.y * d.y, r.z * d.z);
	}
	out[ip] = make_float4(r.x, r.y, r.z, c.w);
}

template <int POWER>
void launch_atrous(dim3 grid, const float4 *in, float4 *out, const float4 *normal, const float4 *albedo,
		const float4 *position, const AtrousPass &ps, bool use_position, cudaStream_t st)
{
	if (use_position)
		atrous_kernel<POWER, true><<<grid, dim3(32, 4), 0, st>>>(in, out, normal, albedo, position, ps);
	else
		atrous_kernel<POWER, false><<<grid, dim3(32, 4), 0, st>>>(in, out, normal, albedo, position, ps);
	KGR_CUDA(cudaGetLastError());
}

} /* namespace */

void tonemap(const float4 *hdr, uint32_t *ldr, uint32_t width, uint32_t height, int mode, cudaStream_t st)
{
	dim3 block(16, 16);
	dim3 grid((width + 15) / 16, (height + 15) / 16);
	tonemap_kernel<<<grid, block, 0, st>>>(hdr, ldr, width, height, mode);
	KGR_CUDA(cudaGetLastError());
}

void denoise(const float4 *color, const float4 *normal, const float4 *albedo, const float4 *position, float4 *out,
		float4 *scratch, uint32_t width, uint32_t height, const kgr_denoise_params &p, int guides, cudaStream_t st)
{
	const bool use_albedo = (guides & KGR_DENOISE_ALBEDO) != 0;
	AtrousPass ps;
	ps.width = width;
	ps.height = height;
	/* not infinite for a denormal sigma: a distance of 0 weighs 1 */
	ps.position_rate = fminf(1.0f / p.sigma_position, FLT_MAX);
	ps.normal_power = p.normal_power;
	ps.squarings = 0;
	int power = POWER_NONE;
	if (guides & KGR_DENOISE_NORMAL) {
		/* 1, 2, 4, ... 1024 by squaring (the default is 64); any other
		 * exponent by powf, a quarter of a tap's time */
		power = POWER_ANY;
		for (int k = 0; k <= 10; k++)
			if (p.normal_power == (float)(1 << k)) {
				power = k == 6 ? POWER_64 : POWER_SQUARES;
				ps.squarings = k;
			}
	}
	/* passes alternate between out and scratch so that the last one lands in
	 * out; the demodulated image goes where the first pass does not write */
	auto target = [&](int i) { return (p.iterations - 1 - i) % 2 == 0 ? out : scratch; };
	const float4 *src = color;
	if (use_albedo) {
		float4 *first = target(0) == out ? scratch : out;
		uint32_t n = width * height;
		demodulate_kernel<<<(n + 255) / 256, 256, 0, st>>>(color, albedo, first, n);
		KGR_CUDA(cudaGetLastError());
		src = first;
	}
	for (int i = 0; i < p.iterations; i++) {
		ps.step = 1 << i;
		ps.half_sigma = p.sigma_color * (1.0f / (float)(1 << i)) * 0.5f;
		ps.remodulate = use_albedo && i == p.iterations - 1;
		/* four rows a block: an image of more than 262,140 rows takes
		 * several layers of the grid (65,535 is the most in y) */
		const uint32_t rows = (height + 3) / 4, layer = 65535u;
		dim3 grid((width + 31) / 32, rows < layer ? rows : layer, (rows + layer - 1) / layer);
		float4 *dst = target(i);
		const bool use_position = (guides & KGR_DENOISE_POSITION) != 0;
		if (power == POWER_64)
			launch_atrous<POWER_64>(grid, src, dst, normal, albedo, position, ps, use_position, st);
		else if (power == POWER_SQUARES)
			launch_atrous<POWER_SQUARES>(grid, src, dst, normal, albedo, position, ps, use_position, st);
		else if (power == POWER_ANY)
			launch_atrous<POWER_ANY>(grid, src, dst, normal, albedo, position, ps, use_position, st);
		else
			launch_atrous<POWER_NONE>(grid, src, dst, normal, albedo, position, ps, use_position, st);
		src = dst;
	}
}

} /* namespace kgr */
