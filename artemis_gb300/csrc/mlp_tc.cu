/*
 * mlp_tc.cu -- radiance-cache network inference on the fifth-generation
 * tensor cores: tcgen05.mma with the accumulator in tensor memory (TMEM).
 *
 * The network is the one of mlp.cu (64 inputs -> 5 x 64 ReLU -> 3 outputs,
 * BF16 or FP16 weights and activations, FP32 accumulation); this kernel is
 * an alternative to its mma.sync inference and computes the same function.
 *
 * A CTA of five warpgroups (640 threads), one an SM, holds the weights once and
 * runs five independent chains, one a warpgroup, each walking tiles of 128 rows
 * (the MMA's M) with its own input buffer, barriers and accumulator:
 *   weights        the six layers (B operands, N x K) in shared memory in
 *                  the canonical K-major layout without swizzle: 8 x 8 core
 *                  matrices of 128 contiguous bytes, K neighbours 128 bytes
 *                  apart (leading byte offset), 8-row groups 1024 bytes apart
 *                  (stride byte offset);
 *   input          one 128 x 64 tile (the first layer's A operand) a chain in
 *                  the K-major layout with the 128-byte swizzle: row r at r x
 *                  128 bytes, its 16-byte chunk c at chunk c ^ (r mod 8).  A
 *                  tile arrives by one TMA load (cp.async.bulk.tensor.2d, the
 *                  tensor map's 128-byte swizzle writes exactly this layout;
 *                  rows past the end read as zero); the chain's next tile is
 *                  loaded into the same buffer as soon as the first layer's
 *                  MMA has read it, and arrives under the other five layers;
 *   TMEM           96 columns a chain: the activations (32 columns, two halves
 *                  a column, row i in lane i: the A operand of every layer
 *                  after the first) and the FP32 accumulator (64 columns); a
 *                  warp reads and writes lanes 32 (warp mod 4) .. +31;
 *   per layer      one thread of the chain issues four tcgen05.mma (K = 16
 *                  each) and a tcgen05.commit to the chain's mbarrier; after it
 *                  every warp of the chain reads its 32 lanes with tcgen05.ld,
 *                  rounds to half precision, applies ReLU and writes the next
 *                  layer's A operand with tcgen05.st; the chain's 128 threads
 *                  meet at a named barrier (1 + chain).
 *
 * Activations in TMEM are what the five chains buy: written back to shared
 * memory they cost a tile 16 KB of stores and 16 KB of operand reads a layer
 * beside the weights' 8 KB, and that bandwidth was the limit (four chains in
 * each of two CTAs an SM: 129 us for 2.07M rows; this kernel 81 us, 0.54 of the
 * measured BF16 peak).  What is left is the latency of a layer (issue, MMA,
 * commit, read, write, barrier), so every instruction on that path counts: a
 * ReLU of its own beside the conversion 106 against 93 us, the six layers
 * unrolled 102 -> 81 us; four chains 93 us.  Two MMAs of N = 32 a layer, the
 * first half's epilogue under the second's MMA: 139 us.
 *
 * Every wait on an mbarrier is bounded.  A wait that runs out sets bit 0 of
 * the error word; the chain stops at the next layer boundary (the barrier there
 * takes the decision for all its threads together), waits (bounded) for its TMA
 * load in flight, and the block frees its TMEM and returns; the host reads the
 * word with kgr_mlp_check.  kgr_mlp_test_wait_timeout exercises that path: its launch
 * withholds each block's first load, so the wait on it runs out (after
 * TC_WAIT_TEST_LIMIT polls) before any MMA was issued.
 */
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cuda.h>

#include <mutex>
#include <type_traits>

#include "kgr_mlp.h"

namespace kgr {

namespace {

#define TC_ROWS 128                 /* rows per tile: the MMA's M */
#define TC_W 64                     /* hidden width and input width */
#define TC_OUT 16                   /* N of the last layer (3 outputs used) */
#define TC_LAYERS 6
#define TC_LBO 128u                 /* bytes between K-neighbour core matrices */
#define TC_SBO 1024u                /* bytes between 8-row groups (64-wide K) */
#define TC_LAYER_BYTES 8192u        /* 64 x 64 half-precision weights */
#define TC_W_BYTES (5u * TC_LAYER_BYTES + 2048u)
#define TC_CHAINS 5                 /* warpgroups a CTA, each walking tiles of its own */
#define TC_THREADS (128 * TC_CHAINS)
#define TC_X_OFF 43008u             /* = TC_W_BYTES, a multiple of 1024 (swizzle atom) */
#define TC_X_BYTES (TC_ROWS * TC_W * 2u)
#define TC_BAR_OFF (TC_X_OFF + TC_CHAINS * TC_X_BYTES)  /* per chain: MMA barrier, TMA barrier */
#define TC_SLOT_OFF (TC_BAR_OFF + TC_CHAINS * 16u)
#define TC_SMEM (TC_SLOT_OFF + 8u)  /* 125,016 bytes: one CTA an SM */
#define TC_CHAIN_COLS 96u           /* 32 of activations, 64 of accumulator */
#define TC_TMEM_COLS 512u           /* 5 x 96, rounded up to a power of two */
#define TC_WAIT_LIMIT (1u << 24)    /* mbarrier polls before a wait gives up */
#define TC_WAIT_TEST_LIMIT (1u << 16) /* the same, in a launch that tests the give-up path */

/* Byte offset of element (r, k) of an R x 64 K-major operand without
 * swizzle (the weights). */
__device__ __forceinline__ uint32_t core_off(uint32_t r, uint32_t k)
{
	return (r >> 3) * TC_SBO + (k >> 3) * TC_LBO + (r & 7u) * 16u + (k & 7u) * 2u;
}

__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
	return (uint32_t)__cvta_generic_to_shared(p);
}

/* Shared-memory matrix descriptor: start address, leading and stride byte
 * offsets (all in 16-byte units), descriptor version 1, layout type (0: no
 * swizzle; 2: 128-byte swizzle, whose leading offset is unused). */
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout)
{
	uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
	d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
	d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
	d |= (uint64_t)1u << 46;
	d |= (uint64_t)layout << 61;
	return d;
}

/* Arm a TMA barrier with the bytes of one tile and start the tile's load:
 * rows [row0, row0 + 128) of the [n][64] input, all 64 columns (x = 0). */
__device__ __forceinline__ void tma_tile(const CUtensorMap *map, uint32_t dst, uint32_t bar, int row0)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(TC_X_BYTES) : "memory");
	asm volatile(
		"cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
		:: "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(row0), "r"(bar) : "memory");
}

/* Instruction descriptor of kind::f16: FP32 accumulator, A and B both BF16
 * (or both FP16), both K-major, N and M. */
__device__ __forceinline__ uint32_t instr_desc(bool bf16, uint32_t n, uint32_t m)
{
	uint32_t f = bf16 ? 1u : 0u;
	return (1u << 4) | (f << 7) | (f << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

/* Barrier of one chain's 128 threads (named barrier 1 + chain; 0 is the CTA's)
 * with an AND over a flag of every thread. */
__device__ __forceinline__ bool chain_and(int chain, bool v)
{
	uint32_t r;
	asm volatile(
		"{\n\t.reg .pred p, q;\n\t"
		"setp.ne.u32 q, %1, 0;\n\t"
		"bar.red.and.pred p, %2, 128, q;\n\t"
		"selp.u32 %0, 1, 0, p;\n\t"
		"}"
		: "=r"(r) : "r"((uint32_t)v), "r"(chain + 1) : "memory");
	return r != 0;
}

__device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
	asm volatile(
		"{\n\t.reg .pred p;\n\t"
		"setp.ne.b32 p, %4, 0;\n\t"
		"tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
		"}"
		:: "r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}

/* The same with the A operand in tensor memory. */
__device__ __forceinline__ void tc_mma_ts(uint32_t tmem, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
	asm volatile(
		"{\n\t.reg .pred p;\n\t"
		"setp.ne.b32 p, %4, 0;\n\t"
		"tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
		"}"
		:: "r"(tmem), "r"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t bar)
{
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar)
		: "memory");
}

/* Poll the mbarrier for the completion of `parity`, at most `limit` times.
 * Returns false when it gave up. */
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, uint32_t limit)
{
	for (uint32_t i = 0; i < limit; i++) {
		uint32_t done;
		asm volatile(
			"{\n\t.reg .pred p;\n\t"
			"mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
			"selp.u32 %0, 1, 0, p;\n\t"
			"}"
			: "=r"(done) : "r"(bar), "r"(parity) : "memory");
		if (done)
			return true;
	}
	return false;
}

#define TC_R8(i) "=r"(v[i]), "=r"(v[i + 1]), "=r"(v[i + 2]), "=r"(v[i + 3]), "=r"(v[i + 4]), "=r"(v[i + 5]), \
	"=r"(v[i + 6]), "=r"(v[i + 7])

/* 64 consecutive FP32 columns of this thread's TMEM lane. */
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, uint32_t (&v)[64])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x64.b32 "
		"{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
		"%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, "
		"%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
		"%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];"
		: TC_R8(0), TC_R8(8), TC_R8(16), TC_R8(24), TC_R8(32), TC_R8(40), TC_R8(48), TC_R8(56)
		: "r"(taddr) : "memory");
}

/* 16 consecutive FP32 columns of this thread's TMEM lane. */
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
		"{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
		: TC_R8(0), TC_R8(8) : "r"(taddr) : "memory");
}

#define TC_I8(i) "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3]), "r"(v[i + 4]), "r"(v[i + 5]), \
	"r"(v[i + 6]), "r"(v[i + 7])

/* 32 consecutive 32-bit columns of this thread's TMEM lane, written. */
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32])
{
	asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
		"{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
		"%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
		:: TC_I8(0), TC_I8(8), TC_I8(16), TC_I8(24), "r"(taddr) : "memory");
}

__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

/* Two values rounded to half precision with ReLU, in one instruction: a NaN
 * stays a NaN. */
template <class T>
__device__ __forceinline__ uint32_t pack_relu(uint32_t lo, uint32_t hi)
{
	uint32_t r;
	if (std::is_same<T, __nv_bfloat16>::value)
		asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
	else
		asm("cvt.rn.relu.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
	return r;
}

template <class T, int UNROLL>
__global__ void __launch_bounds__(TC_THREADS, 1) mlp_infer_tc_kernel(const T *__restrict__ wt_g,
		const __grid_constant__ CUtensorMap xmap, uint32_t n, float4 *__restrict__ out,
		const uint32_t *__restrict__ n_dev, uint32_t *__restrict__ err, uint32_t withhold_first)
{
	const uint32_t limit = withhold_first ? TC_WAIT_TEST_LIMIT : TC_WAIT_LIMIT;
	if (n_dev) {
		uint32_t c = *n_dev;
		n = c < n ? c : n;
	}
	extern __shared__ __align__(1024) unsigned char sm[];
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	/* chain = warpgroup; a warp reads the TMEM lanes 32 (warp mod 4) .. +31 */
	const int chain = warp >> 2, ctid = tid & 127, cwarp = warp & 3;
	/* the 128-byte swizzle repeats every 1024 bytes; the kernel has no static
	 * shared memory, so its dynamic block starts on such a boundary.  If it
	 * did not, report it (bit 1) and do nothing. */
	if (smem_addr(sm) & 1023u) {
		if (tid == 0)
			atomicOr(err, 2u);
		return;
	}
	const bool bf16 = std::is_same<T, __nv_bfloat16>::value;
	const uint32_t mbar = smem_addr(sm + TC_BAR_OFF + 16u * (uint32_t)chain), tbar = mbar + 8u;
	uint32_t *slot = reinterpret_cast<uint32_t *>(sm + TC_SLOT_OFF);
	const uint32_t tiles = (n + TC_ROWS - 1) / TC_ROWS;
	/* tile t goes to CTA t mod grid: few tiles spread over the SMs */
	const uint32_t stride = gridDim.x * TC_CHAINS;
	uint32_t t = blockIdx.x + gridDim.x * (uint32_t)chain;

	if (tid == 0) {
		for (int i = 0; i < 2 * TC_CHAINS; i++)
			asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(sm + TC_BAR_OFF) + 8u * i),
				"r"(1u) : "memory");
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
		/* the first chain's first tile comes in under the weights */
		if (t < tiles && !withhold_first)
			tma_tile(&xmap, smem_addr(sm + TC_X_OFF), tbar, (int)(t * TC_ROWS));
	}
	if (warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
			:: "r"(smem_addr(slot)), "r"(TC_TMEM_COLS) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	/* weights: global [l][rows][64] row-major -> canonical layout */
	for (int l = 0; l < TC_LAYERS; l++) {
		int rows = l == TC_LAYERS - 1 ? TC_OUT : TC_W;
		const uint4 *src = reinterpret_cast<const uint4 *>(wt_g + (size_t)l * TC_W * TC_W);
		unsigned char *dst = sm + l * TC_LAYER_BYTES;
		for (int c = tid; c < rows * 8; c += TC_THREADS) {
			uint32_t r = (uint32_t)c >> 3, kb = (uint32_t)c & 7u;
			*reinterpret_cast<uint4 *>(dst + core_off(r, kb * 8u)) = __ldg(src + c);
		}
	}
	fence_async_smem();
	tc_before();
	__syncthreads();
	tc_after();
	const uint32_t tmem_base = *slot;
	const uint32_t act = tmem_base + TC_CHAIN_COLS * (uint32_t)chain, acc = act + 32u;
	const uint32_t my_lane = (uint32_t)(cwarp * 32) << 16;
	const uint32_t xbase = smem_addr(sm + TC_X_OFF + (uint32_t)chain * TC_X_BYTES);
	const uint32_t id_hidden = instr_desc(bf16, TC_W, TC_ROWS), id_out = instr_desc(bf16, TC_OUT, TC_ROWS);
	/* the operands' descriptors; an offset within them adds to the address
	 * field (16-byte units, all below 2^14).  Layout type 2: 128-byte swizzle */
	const uint64_t x_desc = smem_desc(xbase, 16u, 1024u, 2u), w_desc = smem_desc(smem_addr(sm), TC_LBO, TC_SBO, 0u);
	uint32_t parity = 0;
	bool ok = true;    /* the same in the chain's threads */
	bool sound = true; /* this thread's waits */
	/* thread 0 of the chain: a TMA load issued and not yet waited for, and how
	 * many have been */
	bool pending = false;
	uint32_t loads = 0;
	auto load = [&](uint32_t tile) {
		tma_tile(&xmap, xbase, tbar, (int)(tile * TC_ROWS));
		pending = true;
	};
	auto loaded = [&]() -> bool {
		if (!bar_wait(tbar, loads & 1u, limit))
			return false;
		loads++;
		pending = false;
		return true;
	};

	if (ctid == 0 && t < tiles && !withhold_first) {
		if (chain == 0)
			pending = true; /* issued above */
		else
			load(t);
	}
	/* ReLU keeps a NaN here, and a NaN among a row's activations makes all of
	 * the next layer's NaN, so a row that met one ends as NaN.  Such a tile is
	 * done again with the ReLU that makes a NaN 0; every other row is the same
	 * with either. */
	bool nan_relu = false;
	while (ok && t < tiles) {
		bool again = false;
#pragma unroll UNROLL
		for (int l = 0; ok && l < TC_LAYERS; l++) {
			const bool last = l == TC_LAYERS - 1;
			if (ctid == 0) {
				if (l == 0) {
					if (sound && loaded()) {
#pragma unroll
						for (uint32_t kc = 0; kc < 4; kc++)
							tc_mma(acc, x_desc + ((kc * 32u) >> 4), w_desc + ((kc * 256u) >> 4), id_hidden,
								kc > 0 ? 1u : 0u);
					} else {
						sound = false;
					}
				} else {
					/* 16 halves of K are 8 columns */
					const uint64_t wl = w_desc + (((uint32_t)l * TC_LAYER_BYTES) >> 4);
#pragma unroll
					for (uint32_t kc = 0; kc < 4; kc++)
						tc_mma_ts(acc, act + kc * 8u, wl + ((kc * 256u) >> 4), last ? id_out : id_hidden,
							kc > 0 ? 1u : 0u);
				}
				/* without an MMA the commit arrives at once */
				tc_commit(mbar);
			}
			sound = bar_wait(mbar, parity, limit) && sound;
			parity ^= 1u;
			tc_after();
			/* the MMA has read the tile: the next one comes into the same
			 * buffer under the other layers */
			if (l == 0 && ctid == 0 && sound && t + stride < tiles)
				load(t + stride);
			bool good = sound;
			if (!last) {
				uint32_t v[64], a[32];
				tmem_ld64(acc + my_lane, v);
				tmem_wait_ld();
				if (nan_relu) {
#pragma unroll
					for (int k = 0; k < 64; k++)
						v[k] = __float_as_uint(fmaxf(__uint_as_float(v[k]), 0.0f));
				}
#pragma unroll
				for (int k = 0; k < 32; k++)
					a[k] = pack_relu<T>(v[2 * k], v[2 * k + 1]);
				tmem_st32(act + my_lane, a);
				tmem_wait_st();
			} else {
				uint32_t v[16];
				tmem_ld16(acc + my_lane, v);
				tmem_wait_ld();
				const float y[3] = {__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2])};
				size_t row = (size_t)t * TC_ROWS + (uint32_t)(cwarp * 32 + lane);
				if (row < n && good) {
					out[row] = make_float4(y[0], y[1], y[2], 0.0f);
					good = nan_relu || (y[0] == y[0] && y[1] == y[1] && y[2] == y[2]);
				}
			}
			tc_before();
			ok = chain_and(chain, good);
			if (last && !ok) {
				ok = chain_and(chain, sound);
				again = ok;
			}
			tc_after();
		}
		nan_relu = again;
		if (!again)
			t += stride;
		else if (ctid == 0) {
			/* the next tile is on its way into the buffer: let it arrive, then
			 * fetch this one again */
			sound = !pending || loaded();
			if (sound)
				load(t);
		}
	}
	if (ctid == 0) {
		if (!ok)
			atomicOr(err, 1u);
		/* a load may still be in flight: give it its (bounded) time before
		 * the block frees its memory */
		if (pending)
			bar_wait(tbar, loads & 1u, limit);
	}
	tc_before();
	__syncthreads();
	tc_after();
	if (warp == 0)
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TC_TMEM_COLS)
			: "memory");
}

/* ------------------------------------------------------------ training -- */

/* Training (forward, loss, backward) on the fifth-generation tensor cores.
 * One CTA an SM: two chains of 128 threads, each walking tiles of 128 rows
 * (thread = row = TMEM lane), a warp a chain that issues its forward and delta
 * MMAs, and one that issues both chains' weight gradients.  All operands
 * are in the canonical layout without swizzle (8 x 8 core matrices of 128
 * contiguous bytes, column neighbours 128 bytes apart, 8-row groups 1024), and
 * each is stored once and read both ways, K-major or, with the descriptor's
 * offsets exchanged and the instruction's transpose bit, MN-major:
 *   W    the six layers' weights [out][in] (42 KB): the forward's B operand
 *        as it is, the delta's transposed;
 *   A    a layer's input [128][64]: the forward's A operand as it is, dW's
 *        transposed;
 *   D    the delta of a layer's output: the A operand of the delta of its
 *        input as it is, dW's B operand transposed.
 * A chain has five tiles of 16 KB and one [128][16] for the output's delta.
 * With A(l) the input of layer l, tile b(i) holds X = A(0) and then A(1) for
 * i = 0, else A(i + 1).  Twelve stages a tile, every one MMAs and then the
 * chain's epilogue of their result:
 *   forward l = 0..5    A(l) x W(l); ReLU, rounded, is A(l + 1) in b(l); the
 *                       last epilogue is the loss and the output's delta D(5);
 *   backward l = 5..0   dW(l) += A(l)^T D(l) (M = 64 inputs, N = outputs, K =
 *                       the 128 rows) and, but for l = 0, D(l) x W(l)^T; masked
 *                       by A(l) > 0 and rounded it is D(l - 1), which takes
 *                       A(l)'s place in b(l - 1).
 * X, overwritten by A(1), comes back into b(4) when stage 4 has read it, and
 * the next tile's X into b(3) when stage 3 has: the next tile counts its tiles
 * from there.  Both come by asynchronous copies under the other stages.
 *
 * The chains need not meet at any barrier: a thread writes its own row only.  A
 * chain's `ready` mbarrier (one arrival a warp) releases the warp that issues
 * its forward and delta MMAs, whose commit releases the chain (`done`).  The dW
 * have a pair of barriers of their own and a third issuing warp, which takes
 * the chains in turn, stage by stage, so that a dW, which both chains add to in
 * tensor memory, is summed in the order of the block's tiles; they run under
 * the delta's epilogue, which waits for its dW only before it stores.  TMEM: 64
 * columns of accumulator a chain, 64 a dW (16 for the last; with M = 64 its
 * rows 16q..16q+15 are lanes 32q..32q+15).  At the end the block writes its dW
 * to its slice of `partial`, which the host sums in block order; the rounding
 * points are those of mlp_train_kernel.
 *
 * What bounds it is the latency of a stage (arrive, issue, MMA, commit, read,
 * convert, store: 0.7 us), of which the second chain hides half; the tensor
 * cores are busy for 17% of the time.  So what does not depend on the stage's
 * MMAs is done before the wait for them (descriptors, masks: 3%).  Operands
 * stored a second time, transposed two bytes at a time with bank conflicts, the
 * weights in both layouts, one chain of 128 threads and a barrier on either side
 * of every stage: 114 us for 65,536 rows of FP16; two chains with one issuing
 * warp 34, this kernel 31.  A training step: 125 us then, now 38; 27 with one
 * tile an SM.
 *
 * Every wait is bounded; a warp whose wait runs out leaves, so that every
 * later wait of its chain and of the issuers runs out too.  The block meets at
 * its barrier, each issuer waits (bounded) for the MMAs it has issued, the block
 * sets bit 0 of the error word, writes zeros for its gradient, frees its tensor
 * memory and returns.  kgr_mlp_test_train_wait_timeout exercises that path
 * (WITHHOLD: each block's first warp never reports its first tile's rows, so
 * chain, issuer and the issuer of dW run out). */
#define TT_ROWS 128
#define TT_CHAINS 2
#define TT_WARPS (5 * TT_CHAINS + 1)            /* four a chain, its issuer, the issuer of dW */
#define TT_THREADS (32 * TT_WARPS)
#define TT_TILE_BYTES (TT_ROWS * TC_W * 2u)       /* 16 KB */
#define TT_BUFS 5u
#define TT_CHAIN_OFF TC_W_BYTES                   /* 43,008 */
#define TT_CHAIN_BYTES (TT_BUFS * TT_TILE_BYTES + TT_ROWS * TC_OUT * 2u)
#define TT_BAR_OFF (TT_CHAIN_OFF + TT_CHAINS * TT_CHAIN_BYTES) /* per chain: ready, done, the same for dW */
#define TT_DRAIN_OFF (TT_BAR_OFF + TT_CHAINS * 32u)            /* per issuer: its MMAs after a give-up */
#define TT_SLOT_OFF (TT_DRAIN_OFF + (TT_CHAINS + 1u) * 8u)
#define TT_SMEM (TT_SLOT_OFF + 8u)              /* 215,136 bytes */
#define TT_TMEM_COLS 512u
/* mbarrier polls before a wait gives up.  A poll suspends the thread for a while:
 * a pass whose waits run out after 2^16 of them takes 0.24 s, one with this
 * limit about a second, a million times a stage */
#define TT_WAIT_LIMIT (1u << 18)
#define TT_DW_COL(l) (64u * TT_CHAINS + 64u * (uint32_t)(l))   /* dW of layer l (layer 5: 16 columns) */
#define TT_TRANSPOSE_A (1u << 15)                 /* instruction descriptor: MN-major operands */
#define TT_TRANSPOSE_B (1u << 16)

/* Tile i of a chain whose b(0) is tile `start`. */
__device__ __forceinline__ uint32_t tile_at(uint32_t start, uint32_t i)
{
	i += start;
	return i >= TT_BUFS ? i - TT_BUFS : i;
}

/* 16 bytes from global to shared memory without a register; zeros if !valid
 * (src must be readable memory all the same). */
__device__ __forceinline__ void copy16(uint32_t dst, const void *src, bool valid)
{
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(valid ? 16u : 0u)
		: "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

/* Rows 8g..8g+7 of a [rows][64] matrix by one warp: eight lanes write a core
 * matrix (no bank conflict), four read a row's half (whole sectors). */
template <class T>
__device__ __forceinline__ void copy_rows8(uint32_t dst, const T *src, uint32_t g, uint32_t lane, bool valid)
{
	const uint32_t r = lane & 7u, c = lane >> 3;
#pragma unroll
	for (uint32_t h = 0; h < 2; h++)
		copy16(dst + g * TC_SBO + (c + 4u * h) * TC_LBO + r * 16u,
			src + (valid ? (size_t)(8u * g + r) * TC_W + (c + 4u * h) * 8u : 0), valid);
}

/* Two values rounded to half precision. */
template <class T>
__device__ __forceinline__ uint32_t pack2(float lo, float hi)
{
	uint32_t r;
	if (std::is_same<T, __nv_bfloat16>::value)
		asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
	else
		asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
	return r;
}

/* ReLU of two halves: a NaN and a negative zero are +0. */
template <class T>
__device__ __forceinline__ uint32_t relu2(uint32_t v)
{
	uint32_t r;
	if (std::is_same<T, __nv_bfloat16>::value)
		asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(0u));
	else
		asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(0u));
	return r;
}

/* 0xFFFF in each half of two ReLU outputs (no sign, no NaN) that is not zero. */
__device__ __forceinline__ uint32_t positive2(uint32_t a)
{
	uint32_t r;
	asm("prmt.b32 %0, %1, %2, 0xBB99;" : "=r"(r) : "r"(a + 0x7FFF7FFFu), "r"(0u));
	return r;
}

/* Eight words to 32 aligned bytes of global memory (zeros if !valid). */
__device__ __forceinline__ void store32(float *dst, const uint32_t *v, bool valid)
{
	asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
		:: "l"(dst), "r"(valid ? v[0] : 0u), "r"(valid ? v[1] : 0u), "r"(valid ? v[2] : 0u), "r"(valid ? v[3] : 0u),
		"r"(valid ? v[4] : 0u), "r"(valid ? v[5] : 0u), "r"(valid ? v[6] : 0u), "r"(valid ? v[7] : 0u) : "memory");
}

template <class T, bool WITHHOLD>
__global__ void __launch_bounds__(TT_THREADS, 1) mlp_train_tc_kernel(const T *__restrict__ wt_g,
		const T *__restrict__ x, const float4 *__restrict__ target, uint32_t n, float *__restrict__ partial,
		const uint32_t *__restrict__ n_dev, uint32_t *__restrict__ err)
{
	if (n_dev) {
		uint32_t c = *n_dev;
		n = c < n ? c : n;
	}
	constexpr uint32_t limit = WITHHOLD ? TC_WAIT_TEST_LIMIT : TT_WAIT_LIMIT;
	extern __shared__ __align__(1024) unsigned char sm[];
	const int tid = threadIdx.x, warp = tid >> 5;
	const uint32_t lane = (uint32_t)tid & 31u;
	const int chain = warp >> 2; /* TT_CHAINS: the issuers */
	const uint32_t cwarp = (uint32_t)warp & 3u;
	const bool bf16 = std::is_same<T, __nv_bfloat16>::value;
	const uint32_t base = smem_addr(sm), bars = base + TT_BAR_OFF;
	uint32_t *slot = reinterpret_cast<uint32_t *>(sm + TT_SLOT_OFF);
	const uint32_t tiles = (n + TT_ROWS - 1) / TT_ROWS;
	const uint32_t tile0 = base + TT_CHAIN_OFF + (uint32_t)chain * TT_CHAIN_BYTES;

	/* this warp's 32 rows of X of a tile */
	auto copy_x = [&](uint32_t buf, uint32_t tile) {
#pragma unroll
		for (uint32_t g = 0; g < 4; g++) {
			const uint32_t row = 32u * cwarp + 8u * g + (lane & 7u);
			const bool valid = (size_t)tile * TT_ROWS + row < n;
			copy_rows8(tile0 + buf * TT_TILE_BYTES, valid ? x + (size_t)tile * TT_ROWS * TC_W : x, 4u * cwarp + g,
				lane, valid);
		}
	};
	uint32_t t = blockIdx.x + gridDim.x * (uint32_t)chain;
	const uint32_t stride = gridDim.x * TT_CHAINS;
	if (chain < TT_CHAINS && t < tiles)
		copy_x(0, t);
	for (uint32_t g = (uint32_t)warp; g < 42u; g += TT_WARPS) /* 5 x 8 groups of rows, 2 of the last layer */
		copy_rows8(base, wt_g, g, lane, true);
	if (tid == 0) {
		for (uint32_t i = 0; i < 4u * TT_CHAINS; i++)
			asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bars + 8u * i), "r"(i & 1u ? 1u : 4u)
				: "memory");
		for (uint32_t i = 0; i <= TT_CHAINS; i++)
			asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(base + TT_DRAIN_OFF + 8u * i), "r"(1u)
				: "memory");
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
			:: "r"(smem_addr(slot)), "r"(TT_TMEM_COLS) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	copy_wait();
	fence_async_smem();
	tc_before();
	__syncthreads();
	tc_after();
	const uint32_t tmem = *slot;
	bool ok = true;
	float lsum = 0.0f;

	/* a [][64] matrix as it is and transposed, a [][16] one the same; an
	 * address adds to the address field (16-byte units, all below 2^14) */
	const uint64_t k64 = smem_desc(0u, TC_LBO, TC_SBO, 0u), m64 = smem_desc(0u, TC_SBO, TC_LBO, 0u);
	const uint64_t k16 = smem_desc(0u, 128u, 256u, 0u), m16 = smem_desc(0u, 256u, 128u, 0u);
	const uint32_t id_hidden = instr_desc(bf16, TC_W, TT_ROWS);
	if (warp == 5 * TT_CHAINS) {
		/* ---- the issuer of dW: both chains', stage by stage ---- */
		if (lane == 0) {
			const uint32_t id_dw = instr_desc(bf16, TC_W, 64) | TT_TRANSPOSE_A | TT_TRANSPOSE_B;
			const uint32_t id_dw_out = instr_desc(bf16, TC_OUT, 64) | TT_TRANSPOSE_A | TT_TRANSPOSE_B;
			uint32_t phase = 0, start = 0;
			for (uint32_t b = blockIdx.x; ok && b < tiles; b += stride) {
				const uint32_t chains = b + gridDim.x < tiles ? 2u : 1u;
				for (int l = TC_LAYERS - 1; ok && l >= 0; l--) {
					/* the tiles of A(l) and of D(l) (l < 5) */
					const uint32_t ia = tile_at(start, l > 0 ? (uint32_t)l - 1u : 4u), id = tile_at(start, (uint32_t)l);
					for (uint32_t c = 0; ok && c < chains; c++) {
						const uint32_t bar = bars + 32u * c + 16u, buf0 = base + TT_CHAIN_OFF + c * TT_CHAIN_BYTES;
						const uint64_t a = m64 + ((buf0 + ia * TT_TILE_BYTES) >> 4);
						const uint32_t d = (buf0 + (l == TC_LAYERS - 1 ? TT_BUFS : id) * TT_TILE_BYTES) >> 4;
						const uint32_t sum = b != blockIdx.x || c > 0 ? 1u : 0u, dw = tmem + TT_DW_COL(l);
						ok = bar_wait(bar, phase, limit);
						if (!ok)
							break;
						tc_after();
						if (l == TC_LAYERS - 1) {
#pragma unroll
							for (uint32_t kc = 0; kc < 8; kc++)
								tc_mma(dw, a + kc * 128u, m16 + d + kc * 32u, id_dw_out, kc > 0 ? 1u : sum);
						} else {
#pragma unroll
							for (uint32_t kc = 0; kc < 8; kc++)
								tc_mma(dw, a + kc * 128u, m64 + d + kc * 128u, id_dw, kc > 0 ? 1u : sum);
						}
						tc_commit(bar + 8u);
					}
					phase ^= 1u;
				}
				start = tile_at(start, 3u);
			}
		}
		ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
	} else if (chain >= TT_CHAINS) {
		/* ---- the issuer of a chain's forward and delta ---- */
		if (lane == 0) {
			const uint32_t c = (uint32_t)warp - 4u * TT_CHAINS;
			const uint32_t id_out = instr_desc(bf16, TC_OUT, TT_ROWS), id_delta = id_hidden | TT_TRANSPOSE_B;
			const uint32_t bar = bars + 32u * c, buf0 = base + TT_CHAIN_OFF + c * TT_CHAIN_BYTES;
			const uint32_t acc = tmem + 64u * c;
			uint32_t phase = 1, start = 0;
			/* X of the first tile came before the CTA's barrier, of a later one
			 * with the last D(0) */
			bool first = true;
			auto next = [&]() -> bool {
				phase ^= 1u;
				ok = first || bar_wait(bar, phase, limit);
				if (first)
					phase ^= 1u;
				first = false;
				tc_after();
				return ok;
			};
			for (uint32_t b = blockIdx.x + gridDim.x * c; ok && b < tiles; b += stride) {
				for (uint32_t l = 0; l < TC_LAYERS; l++) {
					const uint64_t a = k64 + ((buf0 + tile_at(start, l > 0 ? l - 1u : 0u) * TT_TILE_BYTES) >> 4);
					const uint64_t w = k64 + ((base + l * TC_LAYER_BYTES) >> 4);
					const uint32_t id = l == TC_LAYERS - 1 ? id_out : id_hidden;
					if (!next())
						break;
#pragma unroll
					for (uint32_t kc = 0; kc < 4; kc++)
						tc_mma(acc, a + kc * 16u, w + kc * 16u, id, kc > 0 ? 1u : 0u);
					tc_commit(bar + 8u);
				}
				if (!ok || !next())
					break;
				tc_mma(acc, k16 + ((buf0 + TT_BUFS * TT_TILE_BYTES) >> 4),
					m64 + ((base + (TC_LAYERS - 1) * TC_LAYER_BYTES) >> 4), id_delta, 0u);
				tc_commit(bar + 8u);
				for (uint32_t l = TC_LAYERS - 2; l > 0; l--) {
					const uint64_t d = k64 + ((buf0 + tile_at(start, l) * TT_TILE_BYTES) >> 4);
					const uint64_t w = m64 + ((base + l * TC_LAYER_BYTES) >> 4);
					if (!next())
						break;
#pragma unroll
					for (uint32_t kc = 0; kc < 4; kc++)
						tc_mma(acc, d + kc * 16u, w + kc * 128u, id_delta, kc > 0 ? 1u : 0u);
					tc_commit(bar + 8u);
				}
				start = tile_at(start, 3u);
			}
		}
		ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
	} else {
		/* ---- a chain ---- */
		const uint32_t ready = bars + 32u * (uint32_t)chain, done = ready + 8u, dw_ready = ready + 16u, dw_done = ready + 24u;
		const uint32_t acc = tmem + 64u * (uint32_t)chain + ((32u * cwarp) << 16);
		const uint32_t row = 32u * cwarp + lane;
		unsigned char *mine = sm + TT_CHAIN_OFF + (uint32_t)chain * TT_CHAIN_BYTES + (row >> 3) * TC_SBO + (row & 7u) * 16u;
		uint32_t phase = 0, dw_phase = 0, start = 0;
		/* wait for the committed MMAs: the chain's, a dW's */
		auto wait_for = [&](uint32_t bar, uint32_t &parity) -> bool {
			bool got = bar_wait(bar, parity, limit);
			parity ^= 1u;
			got = __all_sync(0xffffffffu, got) != 0;
			tc_after();
			return got;
		};
		auto wait = [&]() -> bool { return wait_for(done, phase); };
		auto wait_dw = [&]() -> bool { return wait_for(dw_done, dw_phase); };
		/* this warp's rows are written and its lanes read */
		auto publish = [&](bool dw) {
			fence_async_smem();
			tc_before();
			__syncwarp();
			if (lane == 0 && !(WITHHOLD && warp == 0)) {
				asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(ready) : "memory");
				if (dw)
					asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(dw_ready) : "memory");
			}
		};
		bool dw0 = false; /* the last tile's dW(0) is not waited for */
		while (ok && t < tiles) {
			const size_t gr = (size_t)t * TT_ROWS + row;
			const float4 tg = gr < n ? __ldg(target + gr) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			/* ---- forward ---- */
			for (uint32_t l = 0; l < TC_LAYERS - 1; l++) {
				ok = wait();
				if (!ok)
					break;
				uint32_t v[64];
				tmem_ld64(acc, v);
				tmem_wait_ld();
				unsigned char *dst = mine + tile_at(start, l) * TT_TILE_BYTES;
				/* dW(0) reads the tiles that A(2) and A(3) will take */
				if (l == 1 && dw0 && !(ok = wait_dw()))
					break;
#pragma unroll
				for (int kb = 0; kb < 8; kb++) {
					uint32_t h[4];
#pragma unroll
					for (int e = 0; e < 4; e++)
						h[e] = relu2<T>(pack2<T>(__uint_as_float(v[8 * kb + 2 * e]), __uint_as_float(v[8 * kb + 2 * e + 1])));
					*reinterpret_cast<uint4 *>(dst + kb * TC_LBO) = make_uint4(h[0], h[1], h[2], h[3]);
				}
				publish(false);
			}
			if (!ok || !(ok = wait()))
				break;
			/* ---- the loss and the output's delta (columns 0..2 of 16) ---- */
			{
				uint32_t v[16];
				tmem_ld16(acc, v);
				tmem_wait_ld();
				const float tv[3] = {tg.x, tg.y, tg.z};
				float d[3] = {0.0f, 0.0f, 0.0f};
				if (gr < n) {
#pragma unroll
					for (int col = 0; col < 3; col++) {
						float y = __uint_as_float(v[col]);
						float diff = y - tv[col];
						float den = y * y + 0.01f;
						lsum += diff * diff / den;
						d[col] = 2.0f * diff / den / (float)n;
					}
				}
				unsigned char *dst = sm + TT_CHAIN_OFF + (uint32_t)chain * TT_CHAIN_BYTES + TT_BUFS * TT_TILE_BYTES
					+ (row >> 3) * 256u + (row & 7u) * 16u;
				*reinterpret_cast<uint4 *>(dst) = make_uint4(pack2<T>(d[0], d[1]), pack2<T>(d[2], 0.0f), 0u, 0u);
				*reinterpret_cast<uint4 *>(dst + 128u) = make_uint4(0u, 0u, 0u, 0u);
			}
			publish(true);
			/* ---- backward ---- */
			for (uint32_t l = TC_LAYERS - 1; l > 0; l--) {
				/* the mask is ready before the MMAs are */
				unsigned char *dst = mine + tile_at(start, l - 1) * TT_TILE_BYTES;
				uint32_t h[32];
#pragma unroll
				for (int kb = 0; kb < 8; kb++) {
					const uint4 a = *reinterpret_cast<const uint4 *>(dst + kb * TC_LBO);
					h[4 * kb] = positive2(a.x);
					h[4 * kb + 1] = positive2(a.y);
					h[4 * kb + 2] = positive2(a.z);
					h[4 * kb + 3] = positive2(a.w);
				}
				ok = wait();
				if (!ok)
					break;
				uint32_t v[64];
				tmem_ld64(acc, v);
				tmem_wait_ld();
#pragma unroll
				for (int e = 0; e < 32; e++)
					h[e] &= pack2<T>(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
				/* dW(l) reads A(l), whose place D(l - 1) takes */
				ok = wait_dw();
				if (!ok)
					break;
#pragma unroll
				for (int kb = 0; kb < 8; kb++)
					*reinterpret_cast<uint4 *>(dst + kb * TC_LBO) =
						make_uint4(h[4 * kb], h[4 * kb + 1], h[4 * kb + 2], h[4 * kb + 3]);
				if (l == 4)
					copy_x(tile_at(start, 4u), t);
				if (l == 3 && t + stride < tiles)
					copy_x(tile_at(start, 3u), t + stride);
				if (l == 1) /* X is back, and the next tile's is there: the issuer takes it up with D(0) */
					copy_wait();
				publish(true);
			}
			dw0 = true;
			start = tile_at(start, 3u);
			t += stride;
		}
		if (ok && dw0)
			ok = wait_dw();
		copy_wait();
	}
	tc_before();
	ok = __syncthreads_and(ok) != 0;
	if (!ok) {
		/* MMAs that nobody has waited for: this thread's own, or none */
		if (chain >= TT_CHAINS && lane == 0) {
			const uint32_t bar = base + TT_DRAIN_OFF + 8u * ((uint32_t)warp - 4u * TT_CHAINS);
			tc_commit(bar);
			bar_wait(bar, 0u, limit);
		}
		if (tid == 0)
			atomicOr(err, 1u);
		__syncthreads();
	}
	tc_after();
	/* this block's dW: lanes 32q..32q+15 hold rows 16q..16q+15 of 64 */
	float *slice = partial + (size_t)blockIdx.x * TC_LAYERS * TC_W * TC_W;
	float *warp_loss = reinterpret_cast<float *>(sm); /* the weights are done with */
	if (chain < TT_CHAINS) {
		float *dst = slice + (size_t)(16u * cwarp + (lane & 15u)) * TC_W;
		const bool valid = ok && blockIdx.x < tiles;
		for (int l = chain; l < TC_LAYERS - 1; l += TT_CHAINS) {
			uint32_t v[64];
			tmem_ld64(tmem + ((32u * cwarp) << 16) + TT_DW_COL(l), v);
			tmem_wait_ld();
			if (lane < 16) {
#pragma unroll
				for (int j = 0; j < 64; j += 8)
					store32(dst + (size_t)l * TC_W * TC_W + j, v + j, valid);
			}
		}
		if (chain == TT_CHAINS - 1) {
			uint32_t v[16];
			tmem_ld16(tmem + ((32u * cwarp) << 16) + TT_DW_COL(TC_LAYERS - 1), v);
			tmem_wait_ld();
			if (lane < 16) {
#pragma unroll
				for (int j = 0; j < 16; j += 8)
					store32(dst + (size_t)(TC_LAYERS - 1) * TC_W * TC_W + j, v + j, valid);
			}
		}
		for (int off = 16; off > 0; off >>= 1)
			lsum += __shfl_down_sync(0xffffffffu, lsum, off);
		if (lane == 0)
			warp_loss[warp] = lsum;
	}
	tc_before();
	__syncthreads();
	tc_after();
	if (tid == 0) {
		float sum = 0.0f;
		for (int w = 0; w < 4 * TT_CHAINS; w++)
			sum += warp_loss[w];
		slice[MLP_LOSS_SLOT] = sum;
	}
	__syncwarp();
	if (warp == 0)
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(TT_TMEM_COLS)
			: "memory");
}

template <class K>
void set_tc_smem(K kernel)
{
	KGR_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
}

/* cuTensorMapEncodeTiled, looked up once through the runtime (no link
 * against the driver library). */
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
		const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
		CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled()
{
	static EncodeTiledFn fn = nullptr;
	static std::once_flag once;
	std::call_once(once, [] {
		void *p = nullptr;
		cudaDriverEntryPointQueryResult q;
		if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
				cudaSuccess && q == cudaDriverEntryPointSuccess)
			fn = reinterpret_cast<EncodeTiledFn>(p);
		cudaGetLastError();
	});
	KGR_REQUIRE(fn, KGR_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
	return fn;
}

template <class K>
void set_train_smem(K kernel)
{
	KGR_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TT_SMEM));
}

} /* namespace */

namespace {

template <class T, bool WITHHOLD>
void launch_train(const MlpParams &mp, const void *x, const float4 *target, uint32_t n, int grid, const uint32_t *n_dev,
		cudaStream_t st)
{
	static bool once = (set_train_smem(mlp_train_tc_kernel<T, WITHHOLD>), true);
	(void)once;
	mlp_train_tc_kernel<T, WITHHOLD><<<grid, TT_THREADS, TT_SMEM, st>>>(static_cast<const T *>(mp.wt),
		static_cast<const T *>(x), target, n, mp.partial, n_dev, mp.tc_err);
}

} /* namespace */

void mlp_train_tc(const MlpParams &mp, const void *x, const float4 *target, uint32_t n, int grid, cudaStream_t st,
		const uint32_t *n_dev, bool withhold)
{
	KGR_REQUIRE(((uintptr_t)x & 15u) == 0, KGR_ERR_INVALID_ARGUMENT, "inputs must be 16-byte aligned");
	const bool bf16 = mp.dtype == KGR_MLP_BF16;
	if (withhold)
		(bf16 ? launch_train<__nv_bfloat16, true> : launch_train<__half, true>)(mp, x, target, n, grid, n_dev, st);
	else
		(bf16 ? launch_train<__nv_bfloat16, false> : launch_train<__half, false>)(mp, x, target, n, grid, n_dev, st);
	KGR_CUDA(cudaGetLastError());
}

namespace {

template <class T, int UNROLL>
void launch_infer_unrolled(const MlpParams &mp, const CUtensorMap &map, uint32_t n, int grid, float4 *out,
		const uint32_t *n_dev, uint32_t *err, bool withhold_first, cudaStream_t st)
{
	static bool once = (set_tc_smem(mlp_infer_tc_kernel<T, UNROLL>), true);
	(void)once;
	mlp_infer_tc_kernel<T, UNROLL><<<grid, TC_THREADS, TC_SMEM, st>>>(static_cast<const T *>(mp.wt), map, n, out, n_dev,
		err, withhold_first ? 1u : 0u);
}

template <class T>
void launch_infer(bool many, const MlpParams &mp, const CUtensorMap &map, uint32_t n, int grid, float4 *out,
		const uint32_t *n_dev, uint32_t *err, bool withhold_first, cudaStream_t st)
{
	if (many)
		launch_infer_unrolled<T, TC_LAYERS>(mp, map, n, grid, out, n_dev, err, withhold_first, st);
	else
		launch_infer_unrolled<T, 1>(mp, map, n, grid, out, n_dev, err, withhold_first, st);
}

} /* namespace */

void mlp_infer_tc(const MlpParams &mp, const void *x, uint32_t n, float4 *out, uint32_t *err, cudaStream_t st,
		const uint32_t *n_dev, bool withhold_first)
{
	if (n == 0)
		return;
	KGR_REQUIRE(((uintptr_t)x & 15u) == 0, KGR_ERR_INVALID_ARGUMENT, "inputs must be 16-byte aligned");
	/* the input as a 2-D tensor: 64 elements (128 bytes) per row, n rows;
	 * one box is a 128 x 64 tile, swizzled by 128 bytes on its way in */
	CUtensorMap map;
	cuuint64_t dims[2] = {TC_W, n};
	cuuint64_t strides[1] = {TC_W * 2};
	cuuint32_t box[2] = {TC_W, TC_ROWS};
	cuuint32_t estr[2] = {1, 1};
	CUresult r = encode_tiled()(&map,
		mp.dtype == KGR_MLP_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
		const_cast<void *>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
		CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	KGR_REQUIRE(r == CUDA_SUCCESS, KGR_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
	/* one CTA an SM; fewer when there are fewer tiles than SMs */
	long long tiles = ((long long)n + TC_ROWS - 1) / TC_ROWS;
	long long cap = device_sm_count();
	int grid = (int)(tiles < cap ? tiles : cap);
	/* the unrolled layers are six times the code, which a call of few tiles
	 * waits for: up to 20,000 rows about 13 us a call rolled and 14 unrolled,
	 * most of it the launch; 200,000 rows 18.6 and 16.1 us, 2.07M 102 and 81 */
	const bool many = tiles > 2 * cap;
	if (mp.dtype == KGR_MLP_BF16)
		launch_infer<__nv_bfloat16>(many, mp, map, n, grid, out, n_dev, err, withhold_first, st);
	else
		launch_infer<__half>(many, mp, map, n, grid, out, n_dev, err, withhold_first, st);
	KGR_CUDA(cudaGetLastError());
}

} /* namespace kgr */
