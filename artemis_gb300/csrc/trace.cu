/*
 * trace.cu -- ray-buffer traversal kernels behind kgr_trace_closest and
 * kgr_trace_any: rays read as two 16-byte loads {o, unused} {d, tmax}, hits
 * written as one 16-byte store.  One ray per thread, or, by the number of
 * rays, eight lanes a ray or lanes that refill (launch_trace_persistent).
 */
#include "kgr_device.cuh"
#include "kgr_wavefront.h"

namespace kgr {

namespace {

#define TRACE_BLOCK 128
#define TRACE_COHERENT 0.9f

/* Whether the rays are coherent: whether, in the 32 consecutive ones at each of
 * four places of the buffer, all but one or two head the way of the one before
 * (within 18 degrees).  An image's row may end in one of the places: its first
 * and last rays are far apart, but only two neighbours are.  Every thread of a
 * block of TRACE_BLOCK takes part; n >= 256. */
__device__ __forceinline__ bool rays_agree(const float4 *__restrict__ rays, uint32_t n)
{
	const uint32_t at = (2u * (threadIdx.x >> 5) + 1u) * (n / 8u) + (threadIdx.x & 31u);
	const float4 d = __ldg(&rays[2 * (size_t)at + 1]);
	const float x = __shfl_up_sync(0xffffffffu, d.x, 1), y = __shfl_up_sync(0xffffffffu, d.y, 1),
		z = __shfl_up_sync(0xffffffffu, d.z, 1);
	const float c = d.x * x + d.y * y + d.z * z;
	const bool close = c > 0.0f &&
		c * c >= TRACE_COHERENT * (d.x * d.x + d.y * d.y + d.z * d.z) * (x * x + y * y + z * z);
	return __syncthreads_and(__popc(__ballot_sync(0xffffffffu, close)) >= 30) != 0;
}

/* One ray per thread, grid-stride. */
template <bool ANY, int LAYOUT>
__device__ __forceinline__ void trace_each(const DeviceScene &s, const float4 *__restrict__ rays, uint32_t n,
		kgr_hit *__restrict__ hits, uint32_t *__restrict__ occluded)
{
	uint32_t stride = gridDim.x * blockDim.x;
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
		float4 a = __ldg(&rays[2 * (size_t)i]);
		float4 b = __ldg(&rays[2 * (size_t)i + 1]);
		f3 o = mk(a.x, a.y, a.z), d = mk(b.x, b.y, b.z);
		kgr_hit h;
		bool r;
		if (LAYOUT == KGR_LAYOUT_THREADED)
			r = trace_threaded<ANY, false>(s, o, d, b.w, h);
		else
			r = trace_fast<ANY, false, LAYOUT>(s, o, d, b.w, h);
		if (ANY) {
			occluded[i] = r ? 1u : 0u;
		} else {
			reinterpret_cast<float4 *>(hits)[i] = make_float4(__int_as_float(h.prim), h.t, h.b1, h.b2);
		}
	}
}

template <bool ANY, int LAYOUT>
__global__ void __launch_bounds__(TRACE_BLOCK) trace_rays_kernel(DeviceScene s, const float4 *__restrict__ rays,
		uint32_t n, kgr_hit *__restrict__ hits, uint32_t *__restrict__ occluded)
{
	trace_each<ANY, LAYOUT>(s, rays, n, hits, occluded);
}

#define TRACE_CHUNK 64u
/* between a bounce's best (31) and a mixed buffer's (8 to 20) */
#define TRACE_REFILL 24

/* The k-th ray of one of `blocks` blocks: it owns the chunks blockIdx, blockIdx
 * + blocks, blockIdx + 2 blocks, ... of `chunk` consecutive rays.  Grows with
 * k. */
__device__ __forceinline__ uint64_t block_ray(uint32_t k, uint32_t chunk, uint32_t blocks)
{
	uint32_t c = k / chunk;
	return ((uint64_t)c * blocks + blockIdx.x) * chunk + (k - c * chunk);
}

/* Lanes that take the next rays of their block when at most `refill` of their
 * warp still walk (persistent_walk). */
template <bool ANY, int LAYOUT>
__device__ __forceinline__ void trace_refill(const DeviceScene &s, const float4 *__restrict__ rays, uint32_t n,
		kgr_hit *__restrict__ hits, uint32_t *__restrict__ occluded, uint32_t *taken, int refill, uint32_t blocks)
{
	const int lane = threadIdx.x & 31;
	int32_t entries[KGR_STACK_DEPTH];
	LocalStack stack(nullptr, entries);
	uint32_t i = 0;
	persistent_walk<ANY, false, LAYOUT>(s, stack, refill, nullptr,
		[&](bool need, unsigned m, float4 &a, float4 &b) {
			int leader = __ffs(m) - 1;
			uint32_t base = 0;
			if (lane == leader)
				base = atomicAdd(taken, (uint32_t)__popc(m));
			base = __shfl_sync(0xffffffffu, base, leader);
			uint64_t at = block_ray(base + (uint32_t)__popc(m & ((1u << lane) - 1u)), TRACE_CHUNK, blocks);
			if (!need || at >= n)
				return false;
			i = (uint32_t)at;
			a = __ldg(&rays[2 * at]);
			b = __ldg(&rays[2 * at + 1]);
			return true;
		},
		[&](const kgr_hit &h, bool occ) {
			if (ANY)
				occluded[i] = occ ? 1u : 0u;
			else
				reinterpret_cast<float4 *>(hits)[i] = make_float4(__int_as_float(h.prim), h.t, h.b1, h.b2);
		});
}

/* Bound by the latency of the node fetches (L2 and L1) and by the lanes of a
 * warp waiting for its longest walk.  The fast and wide layouts with many rays:
 * the first `resident` blocks, all that the GPU holds at once, whose lanes take
 * the rays of their block as they finish, handed out in order by a counter in
 * shared memory, so the call needs no device memory of its own and calls may
 * overlap on any streams.
 * Against one ray per thread over a grid-stride loop, 2,073,600 rays on the
 * box scene, the 0.26M- and the 1.16M-triangle terrain: bounce rays 1096, 861,
 * 1089 -> 912, 719, 879 us, shadow rays 808, 546, 694 -> 584, 449, 573, camera
 * rays 513, 387, 550 -> 497, 357, 478.
 *
 * Camera rays end together, so refilling only mixes warps that belong together,
 * and what they lose is balance: a block keeps its share to the end, where the
 * hardware would have put a new block on an SM that is done.  So every block
 * looks at the rays (rays_agree), and coherent ones go one ray per thread over
 * all the grid's blocks, or (MANY) are taken a whole warp at a time by four
 * times the blocks the GPU holds.  For the others the blocks past the resident
 * ones return.  Camera rays, one ray per thread throughout / the refilling walk
 * throughout / this: box scene, 400,000 139, 158, 140 us, 600,000 194, 217, 195;
 * the larger terrain 171, 162, 172 and 199, 205, 199.  (Two launches, of which
 * one returned at once, cost every buffer 3 to 5 us: 600,000 bounce rays on the
 * box scene 305 and now 297.) */
template <bool ANY, int LAYOUT, bool MANY>
__global__ void __launch_bounds__(TRACE_BLOCK) trace_many_kernel(DeviceScene s, const float4 *__restrict__ rays,
		uint32_t n, kgr_hit *__restrict__ hits, uint32_t *__restrict__ occluded, uint32_t resident)
{
	__shared__ uint32_t taken;
	if (threadIdx.x == 0)
		taken = 0;
	const bool coherent = rays_agree(rays, n); /* a barrier too */
	if (coherent && !MANY) {
		trace_each<ANY, LAYOUT>(s, rays, n, hits, occluded);
		return;
	}
	if (!coherent && blockIdx.x >= resident)
		return;
	trace_refill<ANY, LAYOUT>(s, rays, n, hits, occluded, &taken, coherent ? 0 : TRACE_REFILL,
		coherent ? gridDim.x : resident);
}

/* The cooperative walk, eight lanes a ray; rays as above. */
template <bool ANY>
__global__ void __launch_bounds__(TRACE_BLOCK) trace_coop_kernel(DeviceScene s, const float4 *__restrict__ rays,
		uint32_t n, kgr_hit *__restrict__ hits, uint32_t *__restrict__ occluded)
{
	__shared__ uint32_t taken;
	if (threadIdx.x == 0)
		taken = 0;
	__syncthreads();
	const int lane = threadIdx.x & 31, group = lane >> 3;
	const uint32_t chunk = TRACE_BLOCK / 8;
	uint32_t i = 0;
	coop_walk<ANY>(s,
		[&](bool need, float4 &a, float4 &b) {
			/* one bit per group that needs a ray */
			unsigned m = __ballot_sync(0xffffffffu, need) & 0x01010101u;
			uint32_t base = 0;
			if (lane == 0)
				base = atomicAdd(&taken, (uint32_t)__popc(m));
			base = __shfl_sync(0xffffffffu, base, 0);
			uint64_t at = block_ray(base + (uint32_t)__popc(m & ((1u << (8 * group)) - 1u)), chunk, gridDim.x);
			if (!need || at >= n)
				return false;
			i = (uint32_t)at;
			a = __ldg(&rays[2 * at]);
			b = __ldg(&rays[2 * at + 1]);
			return true;
		},
		[&](const kgr_hit &h, bool occ) {
			if (ANY)
				occluded[i] = occ ? 1u : 0u;
			else
				reinterpret_cast<float4 *>(hits)[i] = make_float4(__int_as_float(h.prim), h.t, h.b1, h.b2);
		});
}

int grid_for(uint32_t n, int block)
{
	int dev = 0, sms = 152;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	long long blocks = ((long long)n + block - 1) / block;
	long long cap = (long long)sms * 16;
	return (int)(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

template <bool ANY, int LAYOUT>
void launch_trace_persistent(const DeviceScene &s, const float4 *rays, uint32_t n, kgr_hit *hits, uint32_t *occluded,
		cudaStream_t st)
{
	/* what the GPU holds of either variant at once */
	static const uint32_t resident = (uint32_t)resident_blocks(trace_many_kernel<ANY, LAYOUT, false>, TRACE_BLOCK);
	static const uint32_t resident_many = (uint32_t)resident_blocks(trace_many_kernel<ANY, LAYOUT, true>, TRACE_BLOCK);
	if (LAYOUT == KGR_LAYOUT_FAST && s.coop_nodes) {
		/* up to KGR_COOP_ROUNDS_RAYS rays for each of the resident groups */
		static const int coop = resident_blocks(trace_coop_kernel<ANY>, TRACE_BLOCK);
		const uint32_t groups = (uint32_t)coop * (TRACE_BLOCK / 8);
		if (n <= KGR_COOP_ROUNDS_RAYS * groups) {
			const uint32_t blocks = (n + TRACE_BLOCK / 8 - 1) / (TRACE_BLOCK / 8);
			trace_coop_kernel<ANY><<<blocks < (uint32_t)coop ? blocks : (uint32_t)coop, TRACE_BLOCK, 0, st>>>(s, rays,
				n, hits, occluded);
			return;
		}
	}
	/* Coherent rays are MANY past three rounds of the per-thread grid (933,888
	 * rays): its fourth round is mostly empty, 990,000 camera rays 293, 243, 322
	 * us on the three scenes and 275, 209, 290 by whole warps; at 900,000 257,
	 * 201, 296 one ray per thread.  A fourth round that is nearly full makes up
	 * for it (1.2M rays 320, 243, 333 and 326, 249, 341). */
	/* Few rays a lane: one ray per thread, as many blocks as it takes.  The
	 * lanes hardly refill then, and the persistent walk's bookkeeping is 2 to
	 * 7% of 77,000 to 200,000 rays (box scene and both terrains). */
	if (n <= KGR_REFILL_ROUNDS * resident_many * TRACE_BLOCK) {
		trace_rays_kernel<ANY, LAYOUT><<<grid_for(n, TRACE_BLOCK), TRACE_BLOCK, 0, st>>>(s, rays, n, hits, occluded);
		return;
	}
	if (n > 3u * (uint32_t)grid_for(n, TRACE_BLOCK) * TRACE_BLOCK) {
		trace_many_kernel<ANY, LAYOUT, true><<<4 * resident_many, TRACE_BLOCK, 0, st>>>(s, rays, n, hits, occluded,
			resident_many);
	} else {
		const uint32_t each = (uint32_t)grid_for(n, TRACE_BLOCK);
		trace_many_kernel<ANY, LAYOUT, false><<<each > resident ? each : resident, TRACE_BLOCK, 0, st>>>(s, rays, n, hits,
			occluded, resident);
	}
}

template <bool ANY>
__global__ void __launch_bounds__(128) trace_stats_kernel(DeviceScene s, const float4 *__restrict__ rays,
		uint32_t n, unsigned long long *counters)
{
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	TraceCounters tf = {0, 0}, tt = {0, 0};
	if (i < n) {
		float4 a = __ldg(&rays[2 * (size_t)i]);
		float4 b = __ldg(&rays[2 * (size_t)i + 1]);
		f3 o = mk(a.x, a.y, a.z), d = mk(b.x, b.y, b.z);
		kgr_hit h;
		trace_fast<ANY, true>(s, o, d, b.w, h, &tf);
		trace_threaded<ANY, true>(s, o, d, b.w, h, &tt);
	}
	unsigned long long v[4] = {tf.nodes, tf.tris, tt.nodes, tt.tris};
	for (int k = 0; k < 4; k++) {
		unsigned long long x = v[k];
		for (int off = 16; off > 0; off >>= 1)
			x += __shfl_down_sync(0xffffffffu, x, off);
		if ((threadIdx.x & 31) == 0)
			atomicAdd(&counters[k], x);
	}
}

__global__ void read_probe_kernel(const float4 *__restrict__ buf, size_t n, float4 *sink, int iters)
{
	float acc = 0.0f;
	size_t stride = (size_t)gridDim.x * blockDim.x;
	for (int it = 0; it < iters; it++)
		for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
			float4 v = __ldcg(&buf[i]);
			acc += (v.x + v.y) + (v.z + v.w);
		}
	if (acc == 1234.5678f)
		sink[0] = make_float4(acc, 0.0f, 0.0f, 0.0f);
}

} /* namespace */

void launch_read_probe(const float4 *buf, size_t n, float4 *sink, int iters, cudaStream_t st)
{
	int dev = 0, sms = 152;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	read_probe_kernel<<<sms * 8, 256, 0, st>>>(buf, n, sink, iters);
	KGR_CUDA(cudaGetLastError());
}

void launch_trace_closest(const DeviceScene &s, const float4 *rays, uint32_t n, kgr_hit *hits,
		int layout, cudaStream_t stream)
{
	if (n == 0)
		return;
	int grid = grid_for(n, 128);
	if (layout == KGR_LAYOUT_THREADED)
		trace_rays_kernel<false, KGR_LAYOUT_THREADED><<<grid, 128, 0, stream>>>(s, rays, n, hits, nullptr);
	else if (layout == KGR_LAYOUT_WIDE)
		launch_trace_persistent<false, KGR_LAYOUT_WIDE>(s, rays, n, hits, nullptr, stream);
	else if (layout == KGR_LAYOUT_CW8)
		trace_rays_kernel<false, KGR_LAYOUT_CW8><<<grid, 128, 0, stream>>>(s, rays, n, hits, nullptr);
	else
		launch_trace_persistent<false, KGR_LAYOUT_FAST>(s, rays, n, hits, nullptr, stream);
	KGR_CUDA(cudaGetLastError());
}

void launch_trace_any(const DeviceScene &s, const float4 *rays, uint32_t n, uint32_t *occluded,
		int layout, cudaStream_t stream)
{
	if (n == 0)
		return;
	int grid = grid_for(n, 128);
	if (layout == KGR_LAYOUT_THREADED)
		trace_rays_kernel<true, KGR_LAYOUT_THREADED><<<grid, 128, 0, stream>>>(s, rays, n, nullptr, occluded);
	else if (layout == KGR_LAYOUT_WIDE)
		launch_trace_persistent<true, KGR_LAYOUT_WIDE>(s, rays, n, nullptr, occluded, stream);
	else if (layout == KGR_LAYOUT_CW8)
		trace_rays_kernel<true, KGR_LAYOUT_CW8><<<grid, 128, 0, stream>>>(s, rays, n, nullptr, occluded);
	else
		launch_trace_persistent<true, KGR_LAYOUT_FAST>(s, rays, n, nullptr, occluded, stream);
	KGR_CUDA(cudaGetLastError());
}

void launch_trace_stats(const DeviceScene &s, const float4 *rays, uint32_t n, int any,
		unsigned long long *counters, cudaStream_t stream)
{
	if (n == 0)
		return;
	int grid = (int)((n + 127) / 128);
	if (any)
		trace_stats_kernel<true><<<grid, 128, 0, stream>>>(s, rays, n, counters);
	else
		trace_stats_kernel<false><<<grid, 128, 0, stream>>>(s, rays, n, counters);
	KGR_CUDA(cudaGetLastError());
}

} /* namespace kgr */
