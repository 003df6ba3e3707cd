// Attention of a prompt portion on the 5th-generation tensor cores: many query rows over a head-major ring of fp16 or bf16 keys and
// values, one softmax per row (src/infer.cpp:216-248 per row; the layered models' windows, pooled blocks and sinks beside it).
//
// Rows.  The G query heads that share a kv head are stacked, row r = (position r / G, head r % G), so a tile of 128 rows covers
// 128 / G positions: a few positions already fill it, a causal edge wastes little, and every key tile is read once for all G heads.
// A CTA owns two such tiles (A, B) of one kv head, or (SPLIT) one tile, for which A and B are its even and its odd key tiles, joined from TMEM at the
// end; then a cluster of CTAs may share the keys too, and joins (sum, maximum, accumulator) through distributed shared memory in a fixed order.
//
// 12 warps, or 16.  Warp 0 streams key and value tiles of 128 positions with cp.async.bulk.tensor.3d into a ring of stages.  One thread of
// warp 1 issues the products: S = Q K^T into TMEM, O += P V with P out of TMEM (its fp16 / bf16 words take the place of the scores).
// Warps 4-7 and 8-11 are the softmax of A and B, a thread per row: scores from TMEM, online maximum and sum in fp32, P back to
// TMEM.  The two tiles alternate: while one's scores go through the softmax the tensor pipe works for the other.  O stays in TMEM and is
// rescaled whenever a row's maximum grows (by the softmax warps or, in long calls, by warps of their own), so that the weight of a row's largest
// score is 1 and takes no rounding.  (A reference that follows only growth beyond 2^8 saves 0.3 to 8 us of the calls below, but rounds the weight that
// counts most: a row that one key dominates is then off by up to 2^-9 over bf16; 512 rows, window 1024, against 64 bits: 2.30e-3 for 2.24e-3.)  Warps 2
// and 3 serve the layered models: they round pooled fp32 means into stages, and clear the value rows of a ring tile that hold no position (a weight of
// zero times whatever lies there must be zero).
//
// Bound by the chain softmax - products of a tile pair (some 3500 cycles per 128 keys: 1800 from scores to weights, of which the exponentials
// alone take 1024 at 16 a cycle and SM for each of the two tiles, 500 for the rescaling where the softmax warps do it, and 1100 for P V and the next scores: the late portion by
// itself takes 72.0 us at 1720 MHz, the tensor pipe active 58 % and the unit of the exponentials 58 % of the time; in a loop, at 1000 W, 74.6), for short
// contexts by launch, query staging and the store.  Back to back, against 64-row tiles on mma.sync: 507 rows at 7680 positions, 32 / 8 heads of 128:
// 667 -> 74 us (890 TFLOP/s; 66 in the first passes); 512 rows at 0: 32.8 -> 8.9 us; bf16 window 1024 and pooled blocks of 64, 512 rows, 16 / 4 heads: 57.3 -> 14.5 us.
// Of these SPLIT, with the queries of fp16 calls as boxes of a tensor map, made 80.5 to 78.4, 14.1 to 9.7 and 22.7 to 15.5: in pairs of tiles whose keys two CTAs
// share, staging took 2 us, and sending half of the accumulators (64 KB, some 20 bytes a cycle), both cluster barriers and the join 4 us.  (The even and the odd tiles'
// 16-bit weights are then rounded against a maximum each: results differ from those of one maximum by 3e-4, over bf16 1.3e-3, and are as far from 64 bits.)
//
// Weights are ex2.approx of score x c - maximum x c in one FMA, c = log2(e) scale rounded: an error that grows with the scores' size, 2^-24 of it, far below the 2^-9 or
// 2^-11 that the weights are rounded to behind it.  Registers: 168 a thread beside 128 scores; the forms for layered models spill 16 to 56
// bytes of them, the others 8 to 36 (with two tiles a CTA throughout it was 4 to 60), those that rescale in warps of their own none.
#include "common.cuh"
#include "launch.h"
#include "stack_rows.cuh"
#include "tcgen.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>

namespace yalm {
namespace prompt {

constexpr int kThreads = 384, kRescaleThreads = 512, kTile = 128, kMaxDevices = 64;

struct Args {
	void *out;          // fp16 rows (n, heads DV), or fp32 rows of stride ldo
	const void *q;      // fp16 rows (n, heads DK), or fp32 rows of stride ldq
	int ldo, ldq;
	const float *key_pool, *value_pool; // (kv head, block, channel) fp32 means
	const float *sink;                  // per query head, or null
	int n, G, n_kv, v_heads, ring, max_blocks, window, pool, pos0;
	const int *ctl;
	float q_sign, c; // score (in powers of two) = c (q q_sign) . k
	int parts;
	int wide;  // output rows are 16-byte aligned
	int q_map; // the queries come as boxes of the tensor map tq
};

// Key tiles of a CTA's rows: pooled blocks in tiles of 128 first, then the positions lo .. last in runs of slots that end at the ring's end.
struct Tiles {
	int ring, blocks, pooled, lo, last, s0, first_run, per_wrap, total;
	__device__ Tiles(const Args &a, int i_first, int i_last) : ring(a.ring), last(i_last) {
		lo = lo_of(a, i_first), blocks = blocks_of(a, i_last);
		pooled = (blocks + kTile - 1) / kTile;
		s0 = lo % ring, per_wrap = (ring + kTile - 1) / kTile;
		const int len = last - lo + 1, head = min(len, ring - s0), rest = len - head;
		first_run = (head + kTile - 1) / kTile;
		total = pooled + first_run + rest / ring * per_wrap + (rest % ring + kTile - 1) / kTile;
	}
	static __device__ __forceinline__ int lo_of(const Args &a, int i) { return a.window > 0 ? max(0, i - a.window + 1) : 0; }
	static __device__ __forceinline__ int blocks_of(const Args &a, int i) {
		return (a.window > 0 && a.pool > 0 && i - a.window + 1 >= a.pool) ? min((i - a.window + 1) / a.pool, a.max_blocks) : 0;
	}
	// tile k: first block, or first slot and its position; how many of its 128 rows are blocks / positions.  Returns whether it is a pooled one.
	__device__ __forceinline__ bool at(int k, int &slot, int &pos, int &valid) const {
		if (k < pooled) {
			slot = pos = k * kTile, valid = min(kTile, blocks - slot);
			return true;
		}
		k -= pooled;
		if (k < first_run) {
			slot = s0 + k * kTile, pos = lo + k * kTile;
		} else {
			k -= first_run;
			const int wrap = k / per_wrap;
			slot = (k - wrap * per_wrap) * kTile, pos = lo + (ring - s0) + wrap * ring + slot;
		}
		valid = min(min(kTile, ring - slot), last - pos + 1);
		return false;
	}
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, uint32_t bar) {
	asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(map),
	             "r"(c0), "r"(c1), "r"(c2), "r"(bar)
	             : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, uint32_t bar) {
	asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst), "l"(map),
	             "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
	             : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, int c0, int c1, int c2, int c3, uint32_t src) {
	asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(src)
	             : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]^T
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
	asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d), "r"(tmem_a),
	             "l"(bdesc), "r"(idesc), "r"(accumulate)
	             : "memory");
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
	float y;
	asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	return y;
}
template <int N>
__device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
// mbar_wait_warp() without a call: the compiler finds no registers for the roles' own numbers of them in a kernel that calls functions
__device__ __forceinline__ void wait_inline(uint32_t bar, uint32_t parity, bool &dead) {
	if (__all_sync(kFull, mbar_try(bar, parity)) || dead) return;
	const long long t0 = clock64();
	while (!__all_sync(kFull, mbar_try(bar, parity)))
		if (__any_sync(kFull, clock64() - t0 > 4000000000ll)) { // ~2 s
			dead = true;
			return;
		}
}
__device__ __forceinline__ float max3(float a, float b, float c) {
	float y;
	asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
	return y;
}
// two fp32 values in one 64-bit register: the packed FMA and add of sm_100 (same rounding, half the issue slots)
__device__ __forceinline__ uint64_t pack64(uint32_t lo, uint32_t hi) {
	uint64_t r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
	return r;
}
__device__ __forceinline__ void unpack64(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
	uint64_t r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
	return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
	uint64_t r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
	uint64_t r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
#define YALM_R32(r, o)                                                                                                                               \
	"=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7]), "=r"(r[o + 8]),      \
	    "=r"(r[o + 9]), "=r"(r[o + 10]), "=r"(r[o + 11]), "=r"(r[o + 12]), "=r"(r[o + 13]), "=r"(r[o + 14]), "=r"(r[o + 15]), "=r"(r[o + 16]),       \
	    "=r"(r[o + 17]), "=r"(r[o + 18]), "=r"(r[o + 19]), "=r"(r[o + 20]), "=r"(r[o + 21]), "=r"(r[o + 22]), "=r"(r[o + 23]), "=r"(r[o + 24]),     \
	    "=r"(r[o + 25]), "=r"(r[o + 26]), "=r"(r[o + 27]), "=r"(r[o + 28]), "=r"(r[o + 29]), "=r"(r[o + 30]), "=r"(r[o + 31])
#define YALM_V32(r, o)                                                                                                                               \
	"r"(r[o]), "r"(r[o + 1]), "r"(r[o + 2]), "r"(r[o + 3]), "r"(r[o + 4]), "r"(r[o + 5]), "r"(r[o + 6]), "r"(r[o + 7]), "r"(r[o + 8]), "r"(r[o + 9]), \
	    "r"(r[o + 10]), "r"(r[o + 11]), "r"(r[o + 12]), "r"(r[o + 13]), "r"(r[o + 14]), "r"(r[o + 15]), "r"(r[o + 16]), "r"(r[o + 17]),             \
	    "r"(r[o + 18]), "r"(r[o + 19]), "r"(r[o + 20]), "r"(r[o + 21]), "r"(r[o + 22]), "r"(r[o + 23]), "r"(r[o + 24]), "r"(r[o + 25]),             \
	    "r"(r[o + 26]), "r"(r[o + 27]), "r"(r[o + 28]), "r"(r[o + 29]), "r"(r[o + 30]), "r"(r[o + 31])
// 32 columns without waiting for them (tmem_wait_ld, then pin() the registers, before they are used)
template <int O, int N>
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t (&r)[N]) {
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
	             "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
	             "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
	             : YALM_R32(r, O)
	             : "r"(taddr)
	             : "memory");
}
template <int N>
__device__ __forceinline__ void pin(uint32_t (&r)[N]) {
#pragma unroll
	for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}
template <int O, int N>
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[N]) {
	asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
	             "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
	             "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};" ::YALM_V32(r, O),
	             "r"(taddr)
	             : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
	if constexpr (__is_same(T, __half)) {
		const __half2 h = __floats2half2_rn(a, b);
		return *reinterpret_cast<const uint32_t *>(&h);
	} else {
		const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
		return *reinterpret_cast<const uint32_t *>(&h);
	}
}
// Byte offset of 16-byte piece c of row r in an operand tile of 128 rows: sub-tiles of 64 elements a row, SWIZZLE_128B
__device__ __forceinline__ uint32_t tile_at(int r, int c) { return (uint32_t)((c >> 3) * (kTile * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4)); }
// Descriptor of a value tile as the B operand of P V: N (channels) is the contiguous direction.  Groups of 8 positions 1024 bytes
// apart, blocks of 64 channels one sub-tile apart.
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr) {
	return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)((kTile * 128) >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
constexpr uint32_t kBMajorMn = 1u << 16; // instruction descriptor: B is N-major

template <int N>
struct Width {
	static constexpr int value = N;
};

template <int DK, int DV>
struct Shape {
	static constexpr int DKP = DK < 64 ? 64 : DK, DVP = DV < 64 ? 64 : DV; // channels a row takes in shared memory
	static constexpr int Q_BYTES = kTile * DKP * 2, K_BYTES = Q_BYTES, V_BYTES = kTile * DVP * 2, STAGE = K_BYTES > V_BYTES ? K_BYTES : V_BYTES;
	static constexpr int STAGES = STAGE == 32768 ? 4 : 8;
	// the parts of shared keys exchange through space of their own (no CTA waits for the others' products before it sends): (parts - 1) shares of the
	// columns, (reference, sum) of every part
	static constexpr int smem(bool split, int parts) { // (behind the barriers also the factors of RESCALE, which has one part)
		return (parts == 1 ? 2 * kTile * 4 : 0) + (split ? 1 : 2) * Q_BYTES + STAGES * STAGE + 512 + 1024 + (parts > 1 ? (parts - 1) * (DV / parts) * kTile * 4 + parts * kTile * 8 : 0);
	}
	static constexpr int MERGE = 72 * 1024; // where the even and the odd key tiles' (reference, sum) meet: over stages that are done with, behind the patches
	static_assert(MERGE + 2 * kTile * 8 <= Q_BYTES + STAGES * STAGE, "");
};

__device__ __forceinline__ int first_position(const Args &a) {
	if (!a.ctl) return a.pos0;
	chain_wait();
	return a.ctl[CTL_POS];
}

// T: operand type.  LAYERED: fp32 rows in and out, pooled blocks, ring tiles with rows that hold no position, sinks.
// SPLIT: the CTA has one tile of rows, and A and B are its even and its odd key tiles.
// SHARED: a cluster shares the keys (a kernel of its own: with the join in it, calls without one took 0.3 us longer).  BOXES: the results leave as boxes of the
// tensor map to.  RESCALE (with BOXES): the accumulators are rescaled by four warps of their own, 12 - 15, while the softmax warps form the weights.
template <typename T, int DK, int DV, bool LAYERED, bool SPLIT, bool SHARED, bool BOXES, bool RESCALE>
__global__ void __launch_bounds__(RESCALE ? kRescaleThreads : kThreads, 1)
prompt_attn_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                   const __grid_constant__ CUtensorMap to, const __grid_constant__ Args a) {
	using SH = Shape<DK, DV>;
	constexpr int NST = SH::STAGES, ROWS = SPLIT ? kTile : 2 * kTile; // rows of the CTA
	// Of a tile's value rows only the groups of 16 that hold a position are cleared and multiplied (the weights of the others are 0): where values are wider than keys, a window
	// over few keys waited for both (heads of 64 / 128 channels, 16 / 4 of them, 16 rows at 0: 5.27 us, 5.07; 32 rows 6.02, 5.83).  Else that is done under the scores and
	// the softmax, and the conditions cost calls of many tiles 1 % (128 / 128 channels, 33 rows behind a window of 1500: 10.70 us against 10.88).
	constexpr bool FEWER = LAYERED && !SHARED && DK < DV;
	extern __shared__ uint8_t smem_raw[];
	const uint32_t base = (s32(smem_raw) + 1023u) & ~1023u, q0 = base, kv0 = q0 + (ROWS / kTile) * SH::Q_BYTES, bars = kv0 + NST * SH::STAGE;
	const uint32_t full0 = bars, empty0 = full0 + 8 * NST, s_full0 = empty0 + 8 * NST, p_full0 = s_full0 + 16, o_full = p_full0 + 32, v_clean0 = o_full + 8,
	               q_full = v_clean0 + 8 * NST, f_full0 = q_full + 8, tslot = f_full0 + 64;
	const uint32_t factors = bars + 512; // RESCALE: [A, B][row] by what a row's accumulator is rescaled
	const int warp = uniform_warp(), lane = threadIdx.x & 31;
	const int parts = SHARED ? a.parts : 1, part = parts > 1 ? (int)cluster_rank() : 0;
	const int rows = a.n * a.G, units = (rows + ROWS - 1) / ROWS;
	const int unit = units - 1 - (int)(blockIdx.x / parts); // the longest rows first
	const int g = blockIdx.y, r0 = unit * ROWS, nt = SPLIT || r0 + kTile < rows ? 2 : 1;
	if (threadIdx.x == 0) {
		// a value stage (odd) is free again once its products are done and, in a layered model, warps 2 and 3 have passed it
		for (int i = 0; i < NST; ++i) mbar_init(full0 + 8 * i, 1), mbar_init(empty0 + 8 * i, LAYERED && (i & 1) ? 3 : 1);
		for (int i = 0; i < 2; ++i) mbar_init(s_full0 + 8 * i, 1);
		for (int i = 0; i < 4; ++i) mbar_init(p_full0 + 8 * i, RESCALE && !(i & 1) ? 8 : 4); // [tile][half of the keys]: the softmax warps; for the first half those that rescale, too
		mbar_init(o_full, 1), mbar_init(q_full, 1);
		if (RESCALE)
			for (int i = 0; i < 8; ++i) mbar_init(f_full0 + 8 * i, 1); // [tile][quarter of the rows]
		if (LAYERED)
			for (int i = 0; i < NST; ++i) mbar_init(v_clean0 + 8 * i, 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (SHARED) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); // waited for before this CTA writes into the others
	if (warp == 0 && elect_one()) prefetch_map(&tk), prefetch_map(&tv), prefetch_map(&tq), prefetch_map(&to);
	if (warp == 1) tmem_alloc<1>(tslot, 512);
	tc_fence_before();
	__syncthreads(); // (tensor memory is this CTA's before the next kernel may take any)
	const int p0 = first_position(a); // (where no control block has it, the tiles' divisions run under the kernel before this one)
	const Tiles tiles(a, p0 + r0 / a.G, p0 + min((r0 + ROWS - 1) / a.G, a.n - 1));
	const int per = (tiles.total + parts - 1) / parts, k_begin = min(part * per, tiles.total), k_end = min(k_begin + per, tiles.total), nk = k_end - k_begin;
	const bool first_pooled = LAYERED && nk > 0 && k_begin < tiles.pooled;
	bool dead = false;
	auto wait = [&](uint32_t bar, uint32_t parity) {
		if constexpr (RESCALE) wait_inline(bar, parity, dead);
		else mbar_wait_warp(bar, parity, dead);
	};
	chain_wait();
	chain_next();
	tc_fence_after();

	// Key / value tile i of this part (0, 1, ..) takes ring entries 2 i (keys) and 2 i + 1 (values).  Every round of a stage is waited
	// for, also where the entry is not a copy: a parity tells neighbouring rounds apart and no more.
	auto load = [&](int i, int is_v) {
		const int e = 2 * i + is_v, s = e % NST;
		if (e >= NST) wait(empty0 + 8 * s, (uint32_t)(e / NST - 1) & 1u);
		int slot, pos, valid;
		if (tiles.at(k_begin + i, slot, pos, valid) || dead) return; // pooled tiles are filled by other warps
		const uint32_t dst = kv0 + s * SH::STAGE, bar = full0 + 8 * s;
		const int d = is_v ? SH::DVP : SH::DKP, head = is_v ? g % a.v_heads : g;
		if (elect_one()) {
			mbar_expect_tx(bar, is_v ? SH::V_BYTES : SH::K_BYTES);
			for (int c = 0; c < d; c += 64) tma_load_3d(dst + (c / 64) * (kTile * 128), is_v ? &tv : &tk, c, slot, head, bar);
		}
	};
	auto cleared_to = [](int valid) { return FEWER ? (valid + 15) / 16 * 16 : kTile; }; // the first value row of a tile that no product reads
	// a pooled tile's means into its two stages, rounded; value rows past the last block are zero (the scores of such keys are masked)
	auto fill_pooled = [&](int i, int tid, int nthreads) {
		int slot, pos, valid;
		tiles.at(k_begin + i, slot, pos, valid);
		constexpr int KP = SH::DKP / 8, VP = SH::DVP / 8; // 16-byte pieces of a row
		const int v_head = g % a.v_heads;
#pragma unroll 4
		for (int x = tid; x < valid * (KP + VP); x += nthreads) { // keys and values together: their loads travel at the same time
			const bool is_v = x >= valid * KP;
			const int y = is_v ? x - valid * KP : x, r = is_v ? y / VP : y / KP, c = is_v ? y % VP : y % KP, D = is_v ? DV : DK, head = is_v ? v_head : g;
			const float *src = (is_v ? a.value_pool : a.key_pool) + ((size_t)head * a.max_blocks + slot + r) * D + c * 8;
			float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
			if (c * 8 < D) lo = *reinterpret_cast<const float4 *>(src), hi = *reinterpret_cast<const float4 *>(src + 4);
			st_shared4(kv0 + ((2 * i + is_v) % NST) * SH::STAGE + tile_at(r, c),
			           make_float4(__uint_as_float(pack2<T>(lo.x, lo.y)), __uint_as_float(pack2<T>(lo.z, lo.w)), __uint_as_float(pack2<T>(hi.x, hi.y)),
			                       __uint_as_float(pack2<T>(hi.z, hi.w))));
		}
		for (int x = valid * VP + tid; x < cleared_to(valid) * VP; x += nthreads) st_shared4(kv0 + ((2 * i + 1) % NST) * SH::STAGE + tile_at(x / VP, x % VP), make_float4(0.f, 0.f, 0.f, 0.f));
		proxy_fence();
	};

	if (warp == 0) {
		__syncwarp();
		if (!LAYERED && a.q_map && nk > 0 && elect_one()) { // a box is the 128 / G positions of a tile, all G heads of each; positions past the last are zero
			mbar_expect_tx(q_full, (ROWS / kTile == 2 && nt == 2 ? 2 : 1) * SH::Q_BYTES);
			for (int t = 0; t < (SPLIT ? 1 : nt); ++t)
				for (int c = 0; c < SH::DKP; c += 64)
					tma_load_4d(q0 + t * SH::Q_BYTES + (c / 64) * (kTile * 128), &tq, c, 0, g, (r0 + t * kTile) / a.G, q_full);
		}
		__syncwarp();
		for (int e = 0; e < NST && e < 2 * nk; ++e) load(e >> 1, e & 1); // the stages are free: the first tiles travel while the queries are staged
	}
	if (!BOXES && warp > 0 && (LAYERED || !a.q_map)) { // the queries' rows (rows past the last: zero), and the first tile where it is a pooled one
		// a thread keeps its 16-byte column and steps down the rows (the position and head of a row follow without a division); all loads of
		// a batch are in flight together: one at a time this took as long as four key tiles
		constexpr int PIECES = DK / 8, DOWN = (kThreads - 32) / PIECES, STEPS = (ROWS + DOWN - 1) / DOWN, BATCH = LAYERED && !SPLIT ? (STEPS + 1) / 2 : STEPS;
		const int c = (threadIdx.x - 32) % PIECES, di = DOWN / a.G, dh = DOWN % a.G;
		int r = (threadIdx.x - 32) / PIECES, i = (r0 + r) / a.G, hh = (r0 + r) % a.G;
		for (int s0 = 0; s0 < STEPS; s0 += BATCH) {
			float4 lo[BATCH], hi[LAYERED ? BATCH : 1];
			const int first = r;
#pragma unroll
			for (int b = 0; b < BATCH; ++b) {
				lo[b] = make_float4(0.f, 0.f, 0.f, 0.f);
				if constexpr (LAYERED) hi[b] = lo[b];
				if (r < ROWS && r0 + r < rows) {
					if constexpr (LAYERED) {
						const float *src = static_cast<const float *>(a.q) + (size_t)i * a.ldq + (size_t)(g * a.G + hh) * DK + c * 8;
						lo[b] = *reinterpret_cast<const float4 *>(src), hi[b] = *reinterpret_cast<const float4 *>(src + 4);
					} else
						lo[b] = *reinterpret_cast<const float4 *>(static_cast<const T *>(a.q) + ((size_t)(i * a.n_kv + g) * a.G + hh) * DK + c * 8);
				}
				r += DOWN, i += di, hh += dh;
				if (hh >= a.G) hh -= a.G, ++i;
			}
#pragma unroll
			for (int b = 0; b < BATCH; ++b) {
				const int rr = first + b * DOWN;
				if (rr >= ROWS) break;
				float4 v = lo[b];
				if constexpr (LAYERED) {
					const float f = a.q_sign;
					v = make_float4(__uint_as_float(pack2<T>(lo[b].x * f, lo[b].y * f)), __uint_as_float(pack2<T>(lo[b].z * f, lo[b].w * f)),
					                __uint_as_float(pack2<T>(hi[b].x * f, hi[b].y * f)), __uint_as_float(pack2<T>(hi[b].z * f, hi[b].w * f)));
				}
				st_shared4(q0 + (rr / kTile) * SH::Q_BYTES + tile_at(rr % kTile, c), v);
			}
		}
		if constexpr (LAYERED)
			if (first_pooled) fill_pooled(0, threadIdx.x - 32, kThreads - 32);
		proxy_fence();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	uint32_t tmem;
	asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tslot));

	float mref = -INFINITY, l = 0.f; // of this thread's row: reference of the weights (in powers of two), their sum
	auto leave = [&] { // RESCALE: every role runs to its own end.  Behind a join of the branches the compiler would have to do with the fewest registers of them
		tc_fence_before();
		asm volatile("bar.sync 0;" ::: "memory");
	};

	if (warp < 4) {
		if constexpr (RESCALE) fewer_registers<56>(); // 512 threads x 128 registers, as launched, are 128 threads x (56 + 2 x 192 + 72)
		if (warp == 0) {
			if (first_pooled && elect_one()) mbar_arrive(full0), mbar_arrive(full0 + 8);
			for (int e = NST; e < 2 * nk; ++e) load(e >> 1, e & 1);
			__syncwarp();
		} else if (warp == 1) {
			if (nk > 0) { // ---- products ----
				constexpr uint32_t fmt = __is_same(T, __half) ? 0u : kInstrDescBf16;
				const uint32_t qk_desc = instr_desc_f16(128, kTile) | fmt, pv_desc = instr_desc_f16(128, SH::DVP) | fmt | kBMajorMn;
				auto wait_full = [&](int e) {
					wait(full0 + 8 * (e % NST), (uint32_t)(e / NST) & 1u);
					tc_fence_after();
				};
				auto scores = [&](int t, int e) {
					const uint64_t qa = smem_desc_sw128(q0 + (SPLIT ? 0 : t) * SH::Q_BYTES), ka = smem_desc_sw128(kv0 + (e % NST) * SH::STAGE);
					if (elect_one()) {
#pragma unroll
						for (int k = 0; k < DK / 16; ++k) {
							const uint32_t off = ((k >> 2) * (kTile * 128) + (k & 3) * 32) >> 4;
							umma_f16<1>(tmem + t * kTile, qa + off, ka + off, qk_desc, k);
						}
						umma_commit(s_full0 + 8 * t);
					}
				};
				uint32_t cleaned = 0; // a bit per stage: parity of its rounds of clearing
				auto wait_values = [&](int i) { // returns how many groups of 16 rows count
					const int ev = 2 * i + 1;
					wait_full(ev);
					if constexpr (LAYERED) {
						int slot, pos, valid;
						if (!tiles.at(k_begin + i, slot, pos, valid) && valid < cleared_to(valid)) {
							const int sv = ev % NST;
							wait(v_clean0 + 8 * sv, (cleaned >> sv) & 1u);
							cleaned ^= 1u << sv;
							tc_fence_after();
						}
						return cleared_to(valid) / 16;
					} else
						return kTile / 16;
				};
				auto products = [&](int t, int i, int round, bool last, int groups) { // weights of round `round` of t times the values of tile i
					const int ev = 2 * i + 1;
					const uint64_t vdesc = desc_mn(kv0 + (ev % NST) * SH::STAGE);
#pragma unroll
					for (int half = 0; half < 2; ++half) {
						wait(p_full0 + 16 * t + 8 * half, (uint32_t)round & 1u);
						tc_fence_after();
						if (elect_one()) {
#pragma unroll
							for (int k = 4 * half; k < 4 * half + 4; ++k) // 16 positions = 2048 bytes further in every sub-tile, 8 columns of P
								if (!FEWER || k < groups) umma_ts(tmem + 256 + t * SH::DVP, tmem + t * kTile + 8 * k, vdesc + (2048 >> 4) * k, pv_desc, (round | k) != 0);
							if (half && last) umma_commit(empty0 + 8 * (ev % NST));
						}
					}
				};
				if (!LAYERED && a.q_map) wait(q_full, 0);
				if constexpr (SPLIT) {
					auto next_scores = [&](int i) {
						wait_full(2 * i);
						scores(i & 1, 2 * i);
						if (elect_one()) umma_commit(empty0 + 8 * (2 * i % NST));
					};
					next_scores(0);
					if (nk > 1) next_scores(1);
					for (int i = 0; i < nk && !dead; ++i) {
						const int groups = wait_values(i);
						products(i & 1, i, i >> 1, true, groups);
						if (i + 2 < nk) next_scores(i + 2);
					}
				} else {
					wait_full(0);
					for (int t = 0; t < nt; ++t) scores(t, 0);
					if (elect_one()) umma_commit(empty0);
					for (int i = 0; i < nk && !dead; ++i) {
						const int ek = 2 * i + 2;
						const int groups = wait_values(i);
						for (int t = 0; t < nt; ++t) {
							products(t, i, i, t == nt - 1, groups);
							if (i + 1 < nk) {
								if (t == 0) wait_full(ek);
								scores(t, ek);
								if (t == nt - 1 && elect_one()) umma_commit(empty0 + 8 * (ek % NST));
							}
						}
					}
				}
				if (!dead && elect_one()) umma_commit(o_full);
			}
			__syncwarp();
		} else {
			if constexpr (LAYERED) {
				const int tid = threadIdx.x - 64;
				for (int i = 0; i < nk; ++i) {
					int slot, pos, valid;
					const bool pooled = tiles.at(k_begin + i, slot, pos, valid);
					const int ek = 2 * i, ev = 2 * i + 1;
					if (pooled && i > 0) {
						if (ek >= NST) wait(empty0 + 8 * (ek % NST), (uint32_t)(ek / NST - 1) & 1u);
						if (ev >= NST) wait(empty0 + 8 * (ev % NST), (uint32_t)(ev / NST - 1) & 1u);
						fill_pooled(i, tid, 64);
						asm volatile("bar.sync 1, 64;" ::: "memory");
						if (tid == 0) mbar_arrive(full0 + 8 * (ek % NST)), mbar_arrive(full0 + 8 * (ev % NST));
					}
					wait(full0 + 8 * (ev % NST), (uint32_t)(ev / NST) & 1u); // of every tile, to stay with the rounds
					if (!pooled && valid < cleared_to(valid)) {
						const uint32_t dst = kv0 + (ev % NST) * SH::STAGE;
						constexpr int PIECES = SH::DVP / 8;
						for (int x = valid * PIECES + tid; x < cleared_to(valid) * PIECES; x += 64) st_shared4(dst + tile_at(x / PIECES, x % PIECES), make_float4(0.f, 0.f, 0.f, 0.f));
						proxy_fence();
						asm volatile("bar.sync 1, 64;" ::: "memory");
						if (tid == 0) mbar_arrive(v_clean0 + 8 * (ev % NST));
					}
					__syncwarp();
					if (lane == 0) mbar_arrive(empty0 + 8 * (ev % NST));
				}
			}
			__syncwarp();
		}
		if constexpr (RESCALE) {
			leave();
			if (warp == 1) {
				tc_fence_after();
				tmem_dealloc<1>(tmem, 512);
			}
			return;
		}
	} else if (RESCALE && warp >= 12) { // ---- rescaling: rows 32 q .. of A and B in turn ----
		fewer_registers<72>();
		const int q = warp & 3;
		for (int k = 0; k < nk; ++k)
			for (int t = SPLIT ? k & 1 : 0; t < (SPLIT ? (k & 1) + 1 : nt); ++t) {
				const int round = SPLIT ? k >> 1 : k;
				wait(s_full0 + 8 * t, (uint32_t)round & 1u); // (of every round: a parity tells neighbouring ones apart and no more)
				if (round > 0) { // before it there is nothing to rescale; the products into O so far are complete: they were issued before these scores
					wait(f_full0 + 32 * t + 8 * q, (uint32_t)(round - 1) & 1u);
					__syncwarp();
					tc_fence_after();
					float f;
					asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(factors + (uint32_t)((t * kTile + q * 32 + lane) * 4)) : "memory");
					if (__any_sync(kFull, f != 1.0f)) {
						const uint32_t op = tmem + ((uint32_t)(q * 32) << 16) + 256 + t * SH::DVP;
						const uint64_t f2 = pack64(__float_as_uint(f), __float_as_uint(f));
#pragma unroll 1
						for (int x = 0; x < DV; x += 32) {
							uint32_t o[32];
							tmem_ld32_async<0>(op + x, o);
							tmem_wait_ld();
							pin(o);
#pragma unroll
							for (int y = 0; y < 32; y += 2) {
								float lo, hi;
								unpack64(mul2(pack64(o[y], o[y + 1]), f2), lo, hi);
								o[y] = __float_as_uint(lo), o[y + 1] = __float_as_uint(hi);
							}
							tmem_st32<0>(op + x, o);
						}
						tmem_wait_st();
					}
					tc_fence_before();
				}
				__syncwarp();
				if (!dead && lane == 0) mbar_arrive(p_full0 + 16 * t);
			}
		leave();
		return;
	} else {
		if constexpr (RESCALE) more_registers<192>();
		const int t = (warp - 4) >> 2, q = warp & 3, r = r0 + (SPLIT ? 0 : t * kTile) + q * 32 + lane;
		if (t < nt && nk > 0) { // ---- softmax: one row per thread ----
			const int i = p0 + min(r, rows - 1) / a.G; // rows past the last repeat it: finite values that are never stored
			const int lo = Tiles::lo_of(a, i), nb = LAYERED ? Tiles::blocks_of(a, i) : 0;
			const uint32_t lanes = (uint32_t)(q * 32) << 16, sp = tmem + lanes + t * kTile, op = tmem + lanes + 256 + t * SH::DVP;
			const float c = a.c;
			for (int k = SPLIT ? t : 0; k < nk; k += SPLIT ? 2 : 1) {
				const int round = SPLIT ? k >> 1 : k;
				int slot, pos, valid;
				const bool pooled = tiles.at(k_begin + k, slot, pos, valid);
				const int from = pooled ? 0 : lo - pos, to = pooled ? nb - slot - 1 : min(i - pos, valid - 1); // visible: from .. to of the tile
				wait(s_full0 + 8 * t, (uint32_t)round & 1u);
				__syncwarp();
				tc_fence_after();
				uint32_t s[kTile];
				tmem_ld32_async<0>(sp, s);
				tmem_ld32_async<32>(sp + 32, s);
				tmem_ld32_async<64>(sp + 64, s);
				tmem_ld32_async<96>(sp + 96, s);
				tmem_wait_ld();
				pin(s);
				if (__any_sync(kFull, from > 0 || to < kTile - 1)) {
#pragma unroll
					for (int x0 = 0; x0 < kTile; x0 += 32) {
						const int first = from - x0, end = to - x0;
						const uint32_t seen = (end < 0 ? 0u : end >= 31 ? ~0u : (2u << end) - 1u) & (first <= 0 ? ~0u : first > 31 ? 0u : ~0u << first);
#pragma unroll
						for (int x = 0; x < 32; ++x)
							if (!(seen & (1u << x))) s[x0 + x] = 0xff800000u; // -inf
					}
				}
				float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
				for (int x = 0; x < kTile; x += 8)
#pragma unroll
					for (int y = 0; y < 4; ++y) mx4[y] = max3(mx4[y], __uint_as_float(s[x + 2 * y]), __uint_as_float(s[x + 2 * y + 1]));
				const float top = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * c;
				const bool grow = top > mref; // (not later: the largest weight of a row is then 1 and takes no rounding)
				if constexpr (RESCALE) {
					const float f = grow ? ex2(mref - top) : 1.0f; // mref -inf: 0
					if (grow) mref = top;
					l *= f;
					if (round > 0) { // warp 12 + q rescales O while the weights are formed
						asm volatile("st.shared.f32 [%0], %1;" ::"r"(factors + (uint32_t)((t * kTile + q * 32 + lane) * 4)), "f"(f) : "memory");
						__syncwarp();
						if (lane == 0) mbar_arrive(f_full0 + 32 * t + 8 * q);
					}
				} else if (__any_sync(kFull, grow)) {
					const float f = grow ? ex2(mref - top) : 1.0f; // mref -inf: 0
					if (grow) mref = top;
					l *= f;
					if (round > 0) { // the products into O so far are complete: they were issued before these scores
#pragma unroll 1
						for (int x = 0; x < DV; x += 32) {
							uint32_t o[32];
							tmem_ld32_async<0>(op + x, o);
							tmem_wait_ld();
							pin(o);
#pragma unroll
							for (int y = 0; y < 32; ++y) o[y] = __float_as_uint(__uint_as_float(o[y]) * f);
							tmem_st32<0>(op + x, o);
						}
					}
				}
				const float ref = mref == -INFINITY ? 0.f : mref; // a row may see nothing yet: all its weights are then 0
				const uint64_t c2 = pack64(__float_as_uint(c), __float_as_uint(c)), ref2 = pack64(__float_as_uint(-ref), __float_as_uint(-ref));
				uint64_t l2[4] = {0, 0, 0, 0};
#pragma unroll
				for (int half = 0; half < 2; ++half) { // the first half's products start while the second half's weights are formed
					uint32_t p[32];
#pragma unroll
					for (int x = 0; x < 32; ++x) {
						float e0, e1;
						unpack64(fma2(pack64(s[64 * half + 2 * x], s[64 * half + 2 * x + 1]), c2, ref2), e0, e1);
						e0 = ex2(e0), e1 = ex2(e1);
						l2[x & 3] = add2(l2[x & 3], pack64(__float_as_uint(e0), __float_as_uint(e1)));
						p[x] = pack2<T>(e0, e1);
					}
					tmem_st32<0>(sp + 32 * half, p);
					tmem_wait_st();
					tc_fence_before();
					__syncwarp();
					if (lane == 0) mbar_arrive(p_full0 + 16 * t + 8 * half);
				}
				float la, lb;
				unpack64(add2(add2(l2[0], l2[1]), add2(l2[2], l2[3])), la, lb);
				l += la + lb;
			}
			wait(o_full, 0);
			__syncwarp();
			tc_fence_after();
		}
	}

	// ---- the rows' results: this part finishes columns part DV / parts .. of its rows; in SPLIT each group of softmax warps half of these ----
	const bool softmax_warp = warp >= 4;
	const int t = (warp - 4) >> 2, q = warp & 3, tr = q * 32 + lane, row = r0 + (SPLIT ? 0 : t * kTile) + tr, share = DV / parts;
	const int mine = SPLIT ? max(share / 2, 8) : share, first_col = SPLIT ? t * mine : 0; // columns that a thread handles of a share, from where
	const bool has_columns = !SHARED || first_col < share; // (a share of 8 is the even group's)
	const uint32_t op = tmem + ((uint32_t)(q * 32) << 16) + 256 + (SPLIT ? 0 : t * SH::DVP);
	// [other part][4 columns][row][4], then (reference, sum) [part][row]
	const uint32_t exch = bars + 512, ml0 = exch + (uint32_t)((parts - 1) * share * kTile * 4);
	if (dead) l = __int_as_float(0x7fc00000);
	__syncwarp();
	float w0 = 1.f, w1 = 1.f; // SPLIT: factors of the sums over the even and the odd key tiles
	bool any0 = true, any1 = true; // whether this row sees any of them (where not, the accumulator may hold anything)
	if constexpr (SPLIT) {
		if (softmax_warp) {
			const uint32_t merge = base + SH::MERGE; // (reference, sum) [even, odd][row]
			asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(merge + (uint32_t)((t * kTile + tr) * 8)), "f"(mref), "f"(l) : "memory");
			asm volatile("bar.sync 2, 256;" ::: "memory");
			float m0, l0, m1, l1;
			asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(m0), "=f"(l0) : "r"(merge + (uint32_t)(tr * 8)) : "memory");
			asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(m1), "=f"(l1) : "r"(merge + (uint32_t)((kTile + tr) * 8)) : "memory");
			mref = fmaxf(m0, m1);
			any0 = l0 != 0.f, any1 = l1 != 0.f, w0 = ex2(m0 - mref), w1 = ex2(m1 - mref);
			l = (any0 ? w0 * l0 : 0.f) + (any1 ? w1 * l1 : 0.f);
		}
	}
	// W columns from x on of this thread's row, of this part's keys
	auto own_columns = [&](auto &v, int x) {
		constexpr int W = sizeof(v) / 4;
		if constexpr (SPLIT) {
			float odd[W];
			if constexpr (W == 32) tmem_ld32(op + x, v);
			else tmem_ld8(op + x, v);
			if (!FEWER || nk > 1) { // (one key tile: no odd ones)
				if constexpr (W == 32) tmem_ld32(op + SH::DVP + x, odd);
				else tmem_ld8(op + SH::DVP + x, odd);
			}
#pragma unroll
			for (int y = 0; y < W; ++y) {
				v[y] = any0 ? w0 * v[y] : 0.f;
				if (any1) v[y] = fmaf(w1, odd[y], v[y]);
			}
		} else {
			if constexpr (W == 32) tmem_ld32(op + x, v);
			else tmem_ld8(op + x, v);
		}
	};
	if (parts > 1) {
		asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); // the other CTAs run
		if (softmax_warp) {
			for (int p = 0; p < parts; ++p) {
				const uint32_t there = map_rank(exch, (uint32_t)p);
				if (t == 0)
					asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(there + (ml0 - exch) + (uint32_t)((part * kTile + tr) * 8)), "f"(mref), "f"(l) : "memory");
				if (p == part || nk == 0 || !has_columns) continue;
				const uint32_t dst = there + (uint32_t)((part < p ? part : part - 1) * share * kTile * 4);
				auto send = [&](auto width, int x) {
					constexpr int W = decltype(width)::value;
					float v[W];
					own_columns(v, p * share + x);
#pragma unroll
					for (int y = 0; y < W; y += 4) st_cluster4(dst + (uint32_t)((((x + y) >> 2) * kTile + tr) * 16), make_float4(v[y], v[y + 1], v[y + 2], v[y + 3]));
				};
				if (mine % 32 == 0)
					for (int x = first_col; x < first_col + mine; x += 32) send(Width<32>(), x);
				else
					for (int x = first_col; x < first_col + mine; x += 8) send(Width<8>(), x);
			}
		}
		__syncwarp();
		cluster_sync(); // the other parts' share of these columns is here
	}
	if (softmax_warp && t < nt && has_columns) {
		float M = mref, Lsum = l;
		auto of_part = [&](int p, float &pm, float &pl) {
			asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(pm), "=f"(pl) : "r"(ml0 + (uint32_t)((p * kTile + tr) * 8)) : "memory");
		};
		if (parts > 1) {
			M = -INFINITY, Lsum = 0.f;
			for (int p = 0; p < parts; ++p) {
				float pm, pl;
				of_part(p, pm, pl);
				M = fmaxf(M, pm);
			}
			for (int p = 0; p < parts; ++p) {
				float pm, pl;
				of_part(p, pm, pl);
				if (pl != 0.f) Lsum += pl * ex2(pm - M); // (a part whose rows see nothing has 0; a NaN counts)
			}
		}
		const int h = g * a.G + min(row, rows - 1) % a.G;
		float f = LAYERED ? stack::softmax_finish(M * 0.69314718055994531f, Lsum, a.sink, h) : 1.0f / Lsum;
		// through a patch of shared memory per warp (over queries and stages, which are done with), so that neighbouring lanes store neighbouring
		// bytes: a row per lane, every 16-byte piece went to a line of its own (5 us for 256 rows of 128)
		const uint32_t ld = (uint32_t)mine * 4 + 16, patch = base + (warp - 4) * 32 * ld;
		// or all rows of a tile as fp16 in the layout of an operand tile, which the copy engine stores: no reads back, no addresses, rows past the last left out
		const uint32_t tile = base + (SPLIT ? 0 : t * SH::Q_BYTES);
		auto put = [&](int x, float4 v, float4 w) { // 8 columns
			v = make_float4(v.x * f, v.y * f, v.z * f, v.w * f), w = make_float4(w.x * f, w.y * f, w.z * f, w.w * f);
			if constexpr (BOXES) {
				st_shared4(tile + tile_at(tr, (first_col + x) / 8), make_float4(__uint_as_float(pack2<T>(v.x, v.y)), __uint_as_float(pack2<T>(v.z, v.w)),
				                                                                __uint_as_float(pack2<T>(w.x, w.y)), __uint_as_float(pack2<T>(w.z, w.w))));
			} else
				st_shared4(patch + lane * ld + x * 4, v), st_shared4(patch + lane * ld + x * 4 + 16, w);
		};
		auto join = [&](auto width, int x) { // columns x .. x + width - 1 of this thread's, the parts of the keys in order
			constexpr int W = decltype(width)::value;
			float own[W];
			__syncwarp();
			own_columns(own, part * share + first_col + x);
			if (parts == 1) {
#pragma unroll
				for (int y = 0; y < W; y += 8)
					put(x + y, make_float4(own[y], own[y + 1], own[y + 2], own[y + 3]), make_float4(own[y + 4], own[y + 5], own[y + 6], own[y + 7]));
				return;
			}
			if constexpr (SHARED) {
				float v[W];
#pragma unroll
				for (int y = 0; y < W; ++y) v[y] = 0.f;
				for (int p = 0; p < parts; ++p) {
					float pm, pl;
					of_part(p, pm, pl);
					if (pl == 0.f) continue;
					const float w = ex2(pm - M);
					if (p == part) {
#pragma unroll
						for (int y = 0; y < W; ++y) v[y] += w * own[y];
					} else {
						const uint32_t src = exch + (uint32_t)((p < part ? p : p - 1) * share * kTile * 4);
#pragma unroll
						for (int y = 0; y < W; y += 4) {
							const float4 o = ld_shared4(src + (uint32_t)((((first_col + x + y) >> 2) * kTile + tr) * 16));
							v[y] += w * o.x, v[y + 1] += w * o.y, v[y + 2] += w * o.z, v[y + 3] += w * o.w;
						}
					}
				}
#pragma unroll
				for (int y = 0; y < W; y += 8) put(x + y, make_float4(v[y], v[y + 1], v[y + 2], v[y + 3]), make_float4(v[y + 4], v[y + 5], v[y + 6], v[y + 7]));
			}
		};
		if (mine % 32 == 0)
			for (int x = 0; x < mine; x += 32) join(Width<32>(), x);
		else
			for (int x = 0; x < mine; x += 8) join(Width<8>(), x);
		__syncwarp();
		if constexpr (BOXES) { // a sub-tile of 64 channels is one group's or (SPLIT, 64 channels in all) half by each
			constexpr bool shared = SPLIT && DV == 64;
			proxy_fence();
			if (shared) asm volatile("bar.sync 2, 256;" ::: "memory");
			else asm volatile("bar.sync %0, 128;" ::"r"(3 + t) : "memory");
			if (q == 0 && (!shared || t == 0) && elect_one()) {
				for (int c = first_col; c < (shared ? 64 : first_col + mine); c += 64) tma_store_4d(&to, c, 0, g, (row - tr) / a.G, tile + (c / 64) * (kTile * 128));
				asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group.read 0;" ::: "memory");
			}
			__syncwarp();
		} else {
			const int pieces = LAYERED ? mine / 4 : mine / 8, lg = 31 - __clz(pieces); // 16-byte pieces of a row: a power of two up to 32
			const int down = 32 >> lg, cc = lane & (pieces - 1), di = down / a.G, dh = down % a.G;
			const int row0 = row - lane;
			int rr = lane >> lg, to = row0 + rr, hh = to % a.G;
			// where this lane's piece of row `to` goes, `ahead` further every `down` rows, and by `wrap` more past the group's last head: one warp's arithmetic for its 32
			// rows, which with the address formed anew for each took 0.2 us more of a window over few keys (16 / 4 heads of 64, 16 rows at 0: 4.65 us, 4.47)
			const size_t ldo = LAYERED ? (size_t)a.ldo : (size_t)a.n_kv * a.G * DV, ahead = di * ldo + dh * DV, wrap = ldo - (size_t)a.G * DV;
			size_t at_out = (to / a.G) * ldo + (size_t)((g * a.G + hh) * DV + part * share + first_col + cc * (LAYERED ? 4 : 8));
			for (; rr < 32 && row0 + rr - (lane >> lg) < rows;) { // (ends after the warp's last valid row)
				constexpr int BATCH = 8; // reads first, then stores
				float4 lo[BATCH], hi[LAYERED ? 1 : BATCH];
#pragma unroll
				for (int x = 0; x < BATCH; ++x) {
					const int at = min(rr + x * down, 31);
					lo[x] = ld_shared4(patch + at * ld + cc * (LAYERED ? 16 : 32));
					if constexpr (!LAYERED) hi[x] = ld_shared4(patch + at * ld + cc * 32 + 16);
				}
#pragma unroll
				for (int x = 0; x < BATCH; ++x) {
					if (rr < 32 && to < rows) {
						if constexpr (LAYERED) {
							float *dst = static_cast<float *>(a.out) + at_out;
							if (a.wide) *reinterpret_cast<float4 *>(dst) = lo[x];
							else *reinterpret_cast<float2 *>(dst) = make_float2(lo[x].x, lo[x].y), *reinterpret_cast<float2 *>(dst + 2) = make_float2(lo[x].z, lo[x].w);
						} else {
							const uint4 pk = make_uint4(pack2<T>(lo[x].x, lo[x].y), pack2<T>(lo[x].z, lo[x].w), pack2<T>(hi[x].x, hi[x].y), pack2<T>(hi[x].z, hi[x].w));
							T *dst = static_cast<T *>(a.out) + at_out;
							if (a.wide) {
								*reinterpret_cast<uint4 *>(dst) = pk;
							} else {
								uint32_t *d32 = reinterpret_cast<uint32_t *>(dst);
								d32[0] = pk.x, d32[1] = pk.y, d32[2] = pk.z, d32[3] = pk.w;
							}
						}
					}
					rr += down, to += down, hh += dh, at_out += ahead;
					if (hh >= a.G) hh -= a.G, at_out += wrap;
				}
			}
		}
	}
	if constexpr (RESCALE) leave();
	else {
		tc_fence_before();
		__syncthreads();
		if (warp == 1) {
			tc_fence_after();
			tmem_dealloc<1>(tmem, 512);
		}
	}
}

// ---- host side ------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
	static EncodeTiledFn fn = nullptr;
	static std::once_flag once;
	std::call_once(once, [] {
		void *p = nullptr;
		cudaDriverEntryPointQueryResult q;
		if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
			fn = reinterpret_cast<EncodeTiledFn>(p);
	});
	return fn;
}
// (heads, ring, d) ring of which `rows` slots count -> boxes of 64 channels x 128 slots of one head; channels and slots past the end are zero
static int make_map(CUtensorMap *map, const void *ptr, int d, int rows, int ring, int heads, bool bf16) {
	EncodeTiledFn fn = encode_fn();
	if (!fn) return YALM_EINVAL;
	const cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)rows, (cuuint64_t)heads};
	const cuuint64_t strides[2] = {(cuuint64_t)d * 2, (cuuint64_t)ring * d * 2};
	const cuuint32_t box[3] = {64, kTile, 1}, estr[3] = {1, 1, 1};
	const CUresult r = fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(ptr), dims, strides, box, estr,
	                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
	                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	return r == CUDA_SUCCESS ? 0 : YALM_EINVAL;
}

// (n, kv heads, G, d) queries or results -> boxes of 64 channels x the G heads of one kv head x 128 / G positions: the rows of a tile, in their order
static int make_query_map(CUtensorMap *map, const void *ptr, int d, int G, int n_kv, int n) {
	EncodeTiledFn fn = encode_fn();
	if (!fn) return YALM_EINVAL;
	const cuuint64_t dims[4] = {(cuuint64_t)d, (cuuint64_t)G, (cuuint64_t)n_kv, (cuuint64_t)n};
	const cuuint64_t strides[3] = {(cuuint64_t)d * 2, (cuuint64_t)G * d * 2, (cuuint64_t)n_kv * G * d * 2};
	const cuuint32_t box[4] = {64, (cuuint32_t)G, 1, (cuuint32_t)(kTile / G)}, estr[4] = {1, 1, 1, 1};
	const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
	                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	return r == CUDA_SUCCESS ? 0 : YALM_EINVAL;
}

template <typename T, int DK, int DV, bool LAYERED, bool SPLIT, bool SHARED, bool BOXES, bool RESCALE>
static int launch_of(Args &a, const void *keys, const void *values, int map_rows, cudaStream_t st) {
	using SH = Shape<DK, DV>;
	auto kernel = prompt_attn_kernel<T, DK, DV, LAYERED, SPLIT, SHARED, BOXES, RESCALE>;
	const int smem = SH::smem(SPLIT, a.parts);
	YALM_TRY(allow_smem((const void *)kernel, smem));
	CUtensorMap tq, tk, tv, to;
	int rc = make_map(&tk, keys, DK, map_rows, a.ring, a.n_kv, LAYERED);
	if (!rc) rc = make_map(&tv, values, DV, map_rows, a.ring, a.v_heads, LAYERED);
	if (rc) return rc;
	a.q_map = !LAYERED && kTile % a.G == 0;
	tq = to = tk;
	if (a.q_map) rc = make_query_map(&tq, a.q, DK, a.G, a.n_kv, a.n);
	if (!rc && BOXES) rc = make_query_map(&to, a.out, DV, a.G, a.n_kv, a.n);
	if (rc) return rc;
	constexpr int ROWS = SPLIT ? kTile : 2 * kTile;
	return launch_chained(kernel, dim3((a.n * a.G + ROWS - 1) / ROWS * a.parts, a.n_kv), dim3(RESCALE ? kRescaleThreads : kThreads), smem, st, a.parts, tq, tk, tv, to, a);
}
// Clusters of 2, 4, 8 CTAs that share keys and run at once, of the current device
template <typename T, int DK, int DV, bool LAYERED>
static int clusters_at_once(int (&room)[4]) {
	using SH = Shape<DK, DV>;
	static int at_once[kMaxDevices][4]; // 0: not asked yet
	static std::mutex mu;
	auto kernel = prompt_attn_kernel<T, DK, DV, LAYERED, true, true, false, false>;
	const DeviceInfo &dev = device_info();
	if (dev.device < 0 || dev.device >= kMaxDevices) return YALM_EINVAL;
	std::lock_guard<std::mutex> lock(mu);
	if (!at_once[dev.device][1]) {
		for (int i = 3; i >= 1; --i) {
			const int smem = SH::smem(true, 1 << i);
			YALM_TRY(allow_smem((const void *)kernel, smem));
			cudaLaunchConfig_t cfg = {};
			cudaLaunchAttribute at[1];
			at[0].id = cudaLaunchAttributeClusterDimension;
			at[0].val.clusterDim.x = 1 << i, at[0].val.clusterDim.y = 1, at[0].val.clusterDim.z = 1;
			cfg.gridDim = dim3(1 << i), cfg.blockDim = dim3(kThreads), cfg.dynamicSmemBytes = smem, cfg.attrs = at, cfg.numAttrs = 1;
			YALM_TRY(cudaOccupancyMaxActiveClusters(&at_once[dev.device][i], kernel, &cfg));
		}
	}
	for (int i = 1; i < 4; ++i) room[i] = at_once[dev.device][i];
	return 0;
}
// One tile of rows a CTA while these run all at once, one per SM, and two beyond, which read a key tile once for both (64 / 8 heads of 128, 512 rows: at 0
// 17.3 us in single tiles, 14.5 in pairs, at 7680 132 and 128).  Where tiles of rows leave SMs idle, a cluster shares the keys: as many parts as still run all at
// once, at least four key tiles in all and more tiles than parts (17 rows, 32 / 8 heads of 128: three key tiles in one part 7.8 us, in two 8.4; five in two 9.7, in
// four 9.2; nine, 128 rows of 8 / 2 heads, in four 10.9, in eight 9.9).  Every part finishes 8 columns at least: 33 rows at 7680, 16 / 8 heads of 32: 29.2 us in two parts, 17.5 in four;
// 12 / 4 of 64: 19.5 in four, 13.5 in eight.  est_tiles: key tiles of the longest rows.
// fp16 results of more tiles than leave two parts a place leave through the copy engine (512 rows at 0, 32 / 8 heads of 128: 9.7 -> 8.9 us; 64 / 8, in pairs: 14.2 -> 13.4);
// a store of few CTAs is there as soon from their threads.
// Those calls leave the rescaling to warps of their own: pairs of tiles always (64 / 8 heads of 128, 512 rows at 0 13.4 -> 12.7 us, at 1536 37.7 -> 34.4, 507 at 7680 143 -> 130; of 64
// 11.2 -> 10.8, 33.5 -> 30.9, 120 -> 107), single ones from kManyTiles key tiles on (32 / 8 heads at 7680: 79.7 -> 74.0 us, of 64 63.8 -> 54.6; at 2048, 20 key tiles, 26.1 on
// both; at 0 9.0 against 9.6 at 16 / 4 heads: what a round hands over costs more than it hides in few of them).
constexpr int kManyTiles = 32;
template <typename T, int DK, int DV, bool LAYERED>
static int launch(Args &a, const void *keys, const void *values, int map_rows, int est_tiles, cudaStream_t st) {
	const long tiles = (long)((a.n * (long)a.G + kTile - 1) / kTile) * a.n_kv;
	const int sms = device_info().sms;
	a.parts = 1;
	if (tiles > sms / 2 + 1) {
		const bool split = tiles <= sms;
		if constexpr (!LAYERED && DV % 64 == 0)
			if (kTile % a.G == 0 && a.wide) {
				if (!split) return launch_of<T, DK, DV, LAYERED, false, false, true, true>(a, keys, values, map_rows, st);
				return est_tiles >= kManyTiles ? launch_of<T, DK, DV, LAYERED, true, false, true, true>(a, keys, values, map_rows, st)
				                               : launch_of<T, DK, DV, LAYERED, true, false, true, false>(a, keys, values, map_rows, st);
			}
		if (!split) return launch_of<T, DK, DV, LAYERED, false, false, false, false>(a, keys, values, map_rows, st);
	} else if (est_tiles >= 4) {
		int room[4];
		if (int rc = clusters_at_once<T, DK, DV, LAYERED>(room)) return rc;
		for (int i = 1; i < 4 && (1 << i) <= DV / 8 && tiles <= room[i] && est_tiles > (1 << i); ++i) a.parts = 1 << i;
		if (a.parts > 1) return launch_of<T, DK, DV, LAYERED, true, true, false, false>(a, keys, values, map_rows, st);
	}
	return launch_of<T, DK, DV, LAYERED, true, false, false, false>(a, keys, values, map_rows, st);
}

constexpr float kLog2e = 1.4426950408889634f;

// Causal attention over an fp16 ring without wrap (slot = position): rows past the portion's last position are zero-filled by the copies.
int causal_f16(void *out, const void *q, const void *keys, const void *values, int n, int pos0, int n_heads, int n_kv, int head_dim, int max_seq_len,
               cudaStream_t st) {
	Args a{};
	a.out = out, a.q = q, a.n = n, a.G = n_heads / n_kv, a.n_kv = n_kv, a.v_heads = n_kv, a.ring = max_seq_len, a.pos0 = pos0;
	a.q_sign = 1.f, a.c = kLog2e / sqrtf((float)head_dim), a.wide = ((uintptr_t)out & 15) == 0;
	const int rows = pos0 + n, est = (rows + kTile - 1) / kTile;
	switch (head_dim) {
	case 128: return launch<__half, 128, 128, false>(a, keys, values, rows, est, st);
	case 64: return launch<__half, 64, 64, false>(a, keys, values, rows, est, st);
	case 32: return launch<__half, 32, 32, false>(a, keys, values, rows, est, st);
	}
	return YALM_EINVAL;
}

int window_bf16(float *out, int ldo, const float *q, int ldq, const void *keys, const void *values, const float *key_pool, const float *value_pool, int n,
                int n_heads, int n_kv, int dk, int dv, int ring, int max_blocks, int window, int pool, float scale, int pos0, const int *ctl, const float *sink,
                int v_heads, cudaStream_t st) {
	Args a{};
	a.out = out, a.ldo = ldo, a.q = q, a.ldq = ldq, a.key_pool = key_pool, a.value_pool = value_pool, a.sink = sink;
	a.n = n, a.G = n_heads / n_kv, a.n_kv = n_kv, a.v_heads = v_heads, a.ring = ring, a.max_blocks = max_blocks, a.window = window;
	a.pool = key_pool ? pool : 0, a.pos0 = pos0, a.ctl = ctl, a.wide = ldo % 4 == 0 && ((uintptr_t)out & 15) == 0;
	a.q_sign = scale > 0.f ? 1.f : scale < 0.f ? -1.f : 0.f, a.c = scale == 0.f ? 1.f : fabsf(scale) * kLog2e; // the maximum is taken before the scale
	int seen = ctl ? ring : pos0 + n; // positions that the longest row can see (the position of a control block is known on the device only)
	if (window > 0) seen = std::min(seen, window + 2 * kTile / a.G);
	const int est = (std::min(seen, ring) + kTile - 1) / kTile;
#define YALM_WINDOW_CASE(K_, V_) \
	if (dk == K_ && dv == V_) return launch<__nv_bfloat16, K_, V_, true>(a, keys, values, ring, est, st)
	YALM_WINDOW_CASE(64, 32);
	YALM_WINDOW_CASE(64, 64);
	YALM_WINDOW_CASE(64, 128);
	YALM_WINDOW_CASE(128, 32);
	YALM_WINDOW_CASE(128, 64);
	YALM_WINDOW_CASE(128, 128);
#undef YALM_WINDOW_CASE
	return YALM_EINVAL;
}

} // namespace prompt
} // namespace yalm
