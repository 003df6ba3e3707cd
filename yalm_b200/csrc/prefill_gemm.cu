// Dense fp16 / bf16 GEMM on the 5th-generation tensor cores for the batched prefill / perplexity path.
//
// The reference has no batched pass at all: it hydrates the KV cache and scores a text one token at a time, every token a
// full sweep over the weights (src/main.cpp:91-97, 174-184).  With many positions in flight the projections ARE
// GEMMs, C[M, N] = A[M, K] * W[N, K]^T - W exactly as the .yalm file stores it ((out, in) row-major = K-major "B") - and
// this is the one place in the project where tensor cores are the right tool.
//
// Two kernels, 192 threads a CTA and the same roles: warp 0 brings 64-column (128-byte, SWIZZLE_128B) boxes of both operands
// with cp.async.bulk.tensor.2d into a ring of pipeline stages (mbarrier complete_tx; rows / columns past the edge are
// zero-filled), one thread of warp 1 issues tcgen05.mma.kind::f16 out of shared memory into a fp32 accumulator in TMEM,
// warps 2-5 read it back (tcgen05.ld) and run the fused tail: plain fp32 store (q | k | v and logits of few rows), fp32 residual add in place
// (wo, w2: x += ...), act(w1 x) * (w3 x) -> fp16 (the A operand of the w2 GEMM); of many rows also q, k and v rotated and appended, and what the
// softmax of a row of logits needs of a tile.
//
//  * gemm_pair_kernel (many rows): a pair of CTAs (cta_group::2) owns a tile of 256 rows x n columns, each CTA staging 128 rows of A
//    and half of the columns of W: twice the products per staged byte of one CTA per 128 x 128 tile.  Persistent over tiles, the
//    accumulator double-buffered so that a tile's tail runs under the next tile's products.  n and the number of K parts are
//    picked per shape (plan_pair).  Bound by the tensor pipe (gate and up of 512 rows: active 85 % of the time, at 1510 MHz in a launch by itself and less
//    in a loop) or by SMs that have no tile (512 x 4096 x 14336: 128 of 148 work, the pipe is active 79 % of their time).
//    512 rows, cold L2, against one CTA per 128 x 128 tile: 4096 x 14336 88 -> 65 us (919 TFLOP/s), w1 | w3 14336 x 4096 158 -> 109 us
//    (1108), 32000 x 4096 242 -> 117 us (1150), q | k | v 74 -> 41 us, 4096 x 4096 41 -> 35 us.
//  * gemm_few_kernel (few rows): bound by the bytes of W.  W is the 128-row operand, the positions are the N of the
//    instruction (16 .. 128), so a stage is W bytes and little else; K is split over a cluster of CTAs until the GPU is full.
//    17 rows, cold L2, against the 128 x 128 tiles: 4096 x 4096 35 -> 18 us, 4096 x 14336 80 -> 36 us, w1 | w3 82 -> 59 us, 32000 x 4096 84 -> 63 us.
//
// K parts of a tile are summed through distributed shared memory in a fixed order: each CTA of the cluster finishes its share
// of the columns, so results do not depend on timing and no workspace is needed.
// Activations enter as fp16 (rmsnorm / attention / GLU outputs are rounded once, like the KV cache); sums are fp32.
#include "common.cuh"

#include <cuda.h> // CUtensorMap + enums only: cuTensorMapEncodeTiled is resolved at run time (cudaGetDriverEntryPoint)

#include <algorithm>
#include <cfloat>
#include <mutex>

#include "gemv.cuh"
#include "launch.h"
#include "prefill.h"
#include "tcgen.cuh"

namespace yalm {
namespace prefill {

constexpr int BK = 64;            // 64 16-bit elements = 128 bytes = one SWIZZLE_128B row
constexpr int kRowBytes = 2 * BK; // of an operand row in a stage
constexpr int kGemmThreads = 192;
constexpr int kSegments = 8;

enum Tail { kStoreF32 = 0, kAddF32 = 1, kGluF16 = 2 };
enum Kind { kPlain = 0, kGlu = 1, kRotate = 2, kScore = 3, kResidual = 4 }; // of the pair kernel

// kRotate: q | k | v columns are clipped, the pairs of q and k turned, and all stored as fp16, q as rows, k and v into the head-major ring.
struct RotateArgs {
	__half *q, *k, *v;
	const float2 *turns; // (row, pair of a head): cosine, sine
	int head_dim, ring, pos0;
	float clip;
};
// kScore: of every row and column tile (maximum, sum of exponentials), and the row's value at its target column
struct ScoreArgs {
	float2 *parts; // (tile, row of kPortionRows)
	float *at_target;
	const int *targets;
};

struct GemmArgs {
	int M, N, K; // valid rows of A, rows of W (per matrix), inner dimension
	int tail, act;
	float *c;    // kStoreF32 / kAddF32: (M, ldc) fp32
	__half *h;   // kGluF16: (M, ldc) fp16
	int ldc;
	float alpha; // kStoreF32 / kAddF32: the product is scaled before it is stored / added
	int bf16;    // operands are bf16 instead of fp16 (same instruction kind, other format bits and tensor-map type)
	int nseg;    // output columns [seg_end[s - 1], seg_end[s]) are segment s; tiles never straddle two segments
	int seg_end[kSegments];
	int a_step;  // segment s multiplies rows s a_step .. s a_step + M - 1 of the A operand (0: the same rows for all)
	int n_tile;  // columns of a tile (per matrix)
	int m_tiles, items, splits, kb_per; // 256-row tiles, tiles in all, K parts of a tile and their length in 64-wide blocks
	int stages;
	RotateArgs rotate;
	ScoreArgs score;
};

// One tensor map per weight matrix: the segments' own matrices (wq, wk, wv), or w1 and w3, or one W.
struct WeightMaps {
	CUtensorMap m[3];
};

// ---- tails ------------------------------------------------------------------------------------------------------------
constexpr int kPatch = 32 * 36 * 4; // bytes of one warp's staging patch: 32 rows of 32 fp32, padded to 36

// What store_patch_f32 adds to a warp's 32 rows x 32 columns, read a step ahead of it (behind the products every step waited for its own: 512 x 4096 x 4096
// 19.8 -> 18.7 us, 6144 x 4096 28.7 -> 26.6, 4096 x 14336 53.6 -> 52.6, in a loop, under the power limit, within its noise)
__device__ __forceinline__ void load_residual(const GemmArgs &g, float4 (&x)[8], int row0, int col, int col_end) {
	const int lane = threadIdx.x & 31, r0 = lane >> 3, c0 = col + (lane & 7) * 4;
	const float *base = g.c + (size_t)(row0 + r0) * g.ldc + c0;
#pragma unroll
	for (int t = 0; t < 8; ++t)
		x[t] = c0 + 4 <= col_end && row0 + r0 + 4 * t < g.M ? *reinterpret_cast<const float4 *>(base + (size_t)(4 * t) * g.ldc) : make_float4(0.f, 0.f, 0.f, 0.f);
}
// A warp's 32 rows x 32 columns: lane = row holds v.  Through the warp's patch of shared memory, so that 8 lanes store (and for the
// residual read) 128 consecutive bytes of a row: straight from the lanes every 16-byte piece would be half a sector of its own.
template <bool ADD>
__device__ __forceinline__ void store_patch_f32(const GemmArgs &g, uint32_t patch, const float (&v)[32], const float4 (&x)[ADD ? 8 : 1], int row0, int col, int col_end) {
	const int lane = threadIdx.x & 31, r0 = lane >> 3, cc = (lane & 7) * 4;
	__syncwarp();
#pragma unroll
	for (int i = 0; i < 32; i += 4) st_shared4(patch + (lane * 36 + i) * 4, make_float4(g.alpha * v[i], g.alpha * v[i + 1], g.alpha * v[i + 2], g.alpha * v[i + 3]));
	__syncwarp();
	const int c0 = col + cc;
	float *base = g.c + (size_t)(row0 + r0) * g.ldc + c0;
	if (c0 + 4 <= col_end) {
#pragma unroll
		for (int t = 0; t < 8; ++t) {
			if (row0 + r0 + 4 * t >= g.M) continue;
			float4 o = ld_shared4(patch + ((r0 + 4 * t) * 36 + cc) * 4);
			if constexpr (ADD) // x += W v (src/infer.cpp:335-337), residual stream stays fp32
				o.x += x[t].x, o.y += x[t].y, o.z += x[t].z, o.w += x[t].w;
			*reinterpret_cast<float4 *>(base + (size_t)(4 * t) * g.ldc) = o;
		}
	} else if (c0 < col_end) {
		for (int t = 0; t < 8; ++t) {
			if (row0 + r0 + 4 * t >= g.M) continue;
			const float4 o = ld_shared4(patch + ((r0 + 4 * t) * 36 + cc) * 4);
			const float oo[4] = {o.x, o.y, o.z, o.w};
			float *dst = base + (size_t)(4 * t) * g.ldc;
			for (int j = 0; j < 4 && c0 + j < col_end; ++j) dst[j] = ADD ? dst[j] + oo[j] : oo[j];
		}
	}
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
	const __half2 h = __floats2half2_rn(a, b);
	return *reinterpret_cast<const uint32_t *>(&h);
}
// The same for fp16 results: 4 lanes store the 64 bytes of a row; base: row 0, column 0.
__device__ __forceinline__ void store_patch_f16(const GemmArgs &g, __half *base, size_t ld, uint32_t patch, const float (&v)[32], int row0, int col, int col_end) {
	const int lane = threadIdx.x & 31, r0 = lane >> 2, cc = (lane & 3) * 8;
	__syncwarp();
#pragma unroll
	for (int i = 0; i < 32; i += 8)
		st_shared4(patch + (lane * 20 + i / 2) * 4, make_float4(__uint_as_float(pack_half2(v[i], v[i + 1])), __uint_as_float(pack_half2(v[i + 2], v[i + 3])),
		                                                        __uint_as_float(pack_half2(v[i + 4], v[i + 5])), __uint_as_float(pack_half2(v[i + 6], v[i + 7]))));
	__syncwarp();
	const int c0 = col + cc;
	for (int t = 0; t < 4; ++t) {
		const int row = row0 + r0 + 8 * t;
		if (row >= g.M || c0 >= col_end) continue;
		const float4 o = ld_shared4(patch + ((r0 + 8 * t) * 20 + cc / 2) * 4);
		__half *dst = base + row * ld + c0;
		if (c0 + 8 <= col_end) {
			*reinterpret_cast<float4 *>(dst) = o;
		} else {
			const uint32_t w[4] = {__float_as_uint(o.x), __float_as_uint(o.y), __float_as_uint(o.z), __float_as_uint(o.w)};
			for (int j = 0; j < 8 && c0 + j < col_end; ++j) {
				const __half2 p = *reinterpret_cast<const __half2 *>(&w[j >> 1]);
				dst[j] = (j & 1) ? __high2half(p) : __low2half(p);
			}
		}
	}
}
// act(a) u, rounded to fp16 by the caller.  Both activations as a / (1 + exp(-b)) (0.5 (1 + tanh(y)) = 1 / (1 + exp(-2 y))), the
// quotient by __fdividef: its 2 ulp vanish in the fp16 rounding, and the branch-free form lets a thread's values overlap, where
// the IEEE quotient's and tanhf's branches ran one after another (13 us for a 128 x 128 tile's tail, as long as 8 K blocks).
__device__ __forceinline__ float glu(const GemmArgs &g, float a, float u) {
	const float b = g.act == YALM_ACT_GELU ? 2.0f * 0.797885f * (a + 0.044715f * (a * a * a)) : a;
	return __fdividef(a, 1.0f + expf(-b)) * u;
}
constexpr float kNaN = __builtin_nanf("");

// 32 columns of a segment (col: from its start), all of one head: row i at position pos0 + i (src/infer.cpp:200-213, 282-301)
__device__ __forceinline__ void rotate_store(const GemmArgs &g, int seg, uint32_t patch, float (&v)[32], int row0, int col, int col_end) {
	const RotateArgs &r = g.rotate;
	const int head = col / r.head_dim, c0 = col - head * r.head_dim;
#pragma unroll
	for (int i = 0; i < 32; ++i) v[i] = clipf(v[i], r.clip);
	if (seg < 2) {
		const int row = min(row0 + (int)(threadIdx.x & 31), g.M - 1);
		const float4 *t = reinterpret_cast<const float4 *>(r.turns + ((size_t)row * r.head_dim + c0) / 2);
#pragma unroll
		for (int i = 0; i < 32; i += 4) {
			const float4 cs = t[i / 4];
			rope_turn(v[i], v[i + 1], cs.x, cs.y);
			rope_turn(v[i + 2], v[i + 3], cs.z, cs.w);
		}
	}
	if (seg == 0) store_patch_f16(g, r.q, (size_t)g.seg_end[0], patch, v, row0, col, col_end);
	else store_patch_f16(g, (seg == 1 ? r.k : r.v) + ((size_t)head * r.ring + r.pos0) * r.head_dim, (size_t)r.head_dim, patch, v, row0, c0, c0 + (col_end - col));
}

// Column tile t of the output: its segment, first column and the segment's end.
__device__ __forceinline__ void tile_columns(const GemmArgs &g, int t, int &seg, int &seg0, int &n0, int &n_end) {
	seg = 0, seg0 = 0;
	for (; seg < g.nseg - 1; ++seg) {
		const int tiles = (g.seg_end[seg] - seg0 + g.n_tile - 1) / g.n_tile;
		if (t < tiles) break;
		t -= tiles, seg0 = g.seg_end[seg];
	}
	n0 = seg0 + t * g.n_tile, n_end = min(g.seg_end[seg], n0 + g.n_tile);
}

// Shared memory, from a 1024-byte boundary (the swizzle pattern repeats every 1024 bytes): the stages, the tail warps' patches
// (pair kernel), the barriers.
constexpr int kTailBytes = 4 * kPatch + 512;

// kGlu: w1 | w3 tiles side by side, the pair's first CTA staging w1's rows and the second w3's; accumulator columns n .. 2 n - 1 are w3's.
// kRotate: every segment has a weight matrix of its own.
template <int KIND>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ WeightMaps tb, const __grid_constant__ GemmArgs g) {
	constexpr bool GLU = KIND == kGlu, B_SEG = KIND == kRotate, ADD = KIND == kResidual;
	extern __shared__ uint8_t smem_raw[];
	const int nacc = GLU ? 2 * g.n_tile : g.n_tile; // accumulator columns = N of the instruction; each CTA stages half of them
	const uint32_t a_bytes = 128 * kRowBytes, b_bytes = (uint32_t)(nacc / 2) * kRowBytes, stage_bytes = a_bytes + b_bytes;
	const uint32_t base = (s32(smem_raw) + 1023u) & ~1023u, patch0 = base + g.stages * stage_bytes, bars = patch0 + 4 * kPatch;
	const uint32_t full0 = bars, empty0 = bars + 8 * g.stages, acc_full0 = empty0 + 8 * g.stages, acc_empty0 = acc_full0 + 16, tslot = acc_empty0 + 16;
	const int warp = uniform_warp(), lane = threadIdx.x & 31;
	const int rank = (int)cluster_rank(), half = rank & 1, part = rank >> 1; // CTA of its pair; the pair's part of K
	const int csize = 2 * g.splits, cluster = blockIdx.x / csize, nclusters = gridDim.x / csize;
	const int nkb = (g.K + BK - 1) / BK, kb0 = part * g.kb_per, kb1 = min(nkb, kb0 + g.kb_per);
	bool dead = false;

	if (threadIdx.x == 0) {
		for (int i = 0; i < g.stages; ++i) mbar_init(full0 + 8 * i, 1), mbar_init(empty0 + 8 * i, 1);
		for (int i = 0; i < 2; ++i) mbar_init(acc_full0 + 8 * i, 1), mbar_init(acc_empty0 + 8 * i, 8);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 1) tmem_alloc<2>(tslot, 512);
	tc_fence_before();
	cluster_sync();
	chain_wait();
	chain_next();
	tc_fence_after();
	uint32_t tmem;
	asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tslot));

	if (warp == 0) {
		{ // ---- TMA producer: this CTA's rows of both operands, counted on the first CTA's barrier ----
			const uint32_t lead_full0 = map_rank(full0, rank & ~1);
			Ring ring;
			ring.phase = 1; // the first round of every stage is free
			for (int item = cluster; item < g.items; item += nclusters) {
				int seg, seg0, n0, n_end;
				tile_columns(g, item / g.m_tiles, seg, seg0, n0, n_end);
				const int a0 = seg * g.a_step + (item % g.m_tiles) * 256 + half * 128;
				const CUtensorMap *w = B_SEG ? &tb.m[seg] : GLU ? &tb.m[half] : &tb.m[0];
				const int b0 = GLU ? n0 : (B_SEG ? n0 - seg0 : n0) + half * (nacc / 2);
				for (int kb = kb0; kb < kb1; ++kb, ring.next(g.stages)) {
					mbar_wait_warp(empty0 + 8 * ring.s, ring.phase, dead);
					if (dead) break;
					const uint32_t dst = base + ring.s * stage_bytes, bar = lead_full0 + 8 * ring.s;
					if (elect_one()) {
						if (half == 0) mbar_expect_tx(full0 + 8 * ring.s, 2 * stage_bytes);
						tma_load_2d<2>(dst, &ta, kb * BK, a0, bar);
						tma_load_2d<2>(dst + a_bytes, w, kb * BK, b0, bar);
					}
				}
			}
		}
		__syncwarp();
	} else if (warp == 1) {
		if (half == 0) { // ---- MMA issuer, for both CTAs ----
			const uint32_t idesc = instr_desc_f16(256, nacc) | (g.bf16 ? kInstrDescBf16 : 0u);
			const uint16_t pair_mask = (uint16_t)(3u << (rank & ~1));
			const uint64_t adesc0 = smem_desc_sw128(base), bdesc0 = smem_desc_sw128(base + a_bytes);
			Ring ring;
			int done = 0;
			for (int item = cluster; item < g.items; item += nclusters, ++done) {
				const int b = done & 1;
				if (done >= 2) mbar_wait_warp(acc_empty0 + 8 * b, (uint32_t)(done / 2 - 1) & 1u, dead);
				tc_fence_after();
				uint32_t more = 0;
				for (int kb = kb0; kb < kb1; ++kb, ring.next(g.stages)) {
					mbar_wait_warp(full0 + 8 * ring.s, ring.phase, dead);
					if (dead) break;
					tc_fence_after();
					const uint64_t at = (uint64_t)((ring.s * stage_bytes) >> 4);
					if (elect_one()) {
#pragma unroll
						for (int k = 0; k < BK / 16; ++k) // 16 elements = 32 bytes further along K, inside the 128-byte swizzle row
							umma_f16<2>(tmem + 256 * b, adesc0 + at + 2 * k, bdesc0 + at + 2 * k, idesc, more | k);
						umma_commit_pair(empty0 + 8 * ring.s, pair_mask); // the stage is free in both CTAs once these MMAs have read it
					}
					more = 1;
				}
				if (!dead && elect_one()) umma_commit_pair(acc_full0 + 8 * b, pair_mask); // the accumulator is complete
			}
		}
		__syncwarp();
	} else if (g.splits == 1) { // ---- tail: warp w reads TMEM lanes 32 (w % 4) .. + 31 (the hardware's lane quarter of a warp) ----
		const int q = warp & 3;
		const uint32_t patch = patch0 + q * kPatch, lead_empty0 = map_rank(acc_empty0, rank & ~1);
		int done = 0;
		for (int item = cluster; item < g.items; item += nclusters, ++done) {
			int seg, seg0, n0, n_end;
			tile_columns(g, item / g.m_tiles, seg, seg0, n0, n_end);
			const int b = done & 1, row0 = (item % g.m_tiles) * 256 + half * 128 + q * 32;
			float4 next[ADD ? 8 : 1];
			if constexpr (ADD) load_residual(g, next, row0, n0, n_end);
			mbar_wait_warp(acc_full0 + 8 * b, (uint32_t)(done / 2) & 1u, dead);
			__syncwarp();
			tc_fence_after();
			const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + 256 * b;
			if (row0 < g.M) {
				float top = -FLT_MAX, sum = 0.f; // kScore: of this thread's row (a finite start: columns of -infinity then count as 0)
				int target = -1;
				if constexpr (KIND == kScore)
					if (row0 + lane < g.M) target = g.score.targets[row0 + lane] - n0;
#pragma unroll 1
				for (int c0 = 0; n0 + c0 < n_end; c0 += 32) {
					float4 x[ADD ? 8 : 1];
					if constexpr (ADD) {
#pragma unroll
						for (int i = 0; i < 8; ++i) x[i] = next[i];
						load_residual(g, next, row0, n0 + c0 + 32, n_end);
					}
					float v[32];
					tmem_ld32(trow + c0, v);
					if (GLU) {
						float u[32];
						tmem_ld32(trow + g.n_tile + c0, u);
#pragma unroll
						for (int i = 0; i < 32; ++i) v[i] = glu(g, v[i], u[i]);
					}
					if (dead)
						for (int i = 0; i < 32; ++i) v[i] = kNaN;
					if constexpr (KIND == kScore) {
						float t4[4] = {top, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
						for (int i = 0; i < 32; ++i) {
							if (n0 + c0 + i >= n_end) v[i] = -INFINITY;
							t4[i & 3] = fmaxf(t4[i & 3], v[i]);
							if (target == c0 + i) g.score.at_target[row0 + lane] = v[i];
						}
						const float m = fmaxf(fmaxf(t4[0], t4[1]), fmaxf(t4[2], t4[3]));
						sum *= expf(top - m);
						top = m;
						float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
						for (int i = 0; i < 32; ++i) s4[i & 3] += expf(v[i] - m);
						sum += (s4[0] + s4[1]) + (s4[2] + s4[3]);
					} else if constexpr (KIND == kRotate) {
						rotate_store(g, seg, patch, v, row0, n0 - seg0 + c0, n_end - seg0);
					} else if constexpr (GLU)
						store_patch_f16(g, g.h, (size_t)g.ldc, patch, v, row0, n0 + c0, n_end);
					else
						store_patch_f32<ADD>(g, patch, v, x, row0, n0 + c0, n_end);
				}
				if constexpr (KIND == kScore)
					if (row0 + lane < g.M) g.score.parts[(size_t)(item / g.m_tiles) * kPortionRows + row0 + lane] = make_float2(top, sum);
			}
			tc_fence_before();
			__syncwarp();
			if (lane == 0) mbar_arrive_cluster(lead_empty0 + 8 * b);
		}
	}

	if (KIND != kScore && g.splits > 1) { // one tile per cluster: the pairs' sums meet in shared memory, pair p finishes columns p n / splits ..
		int seg, seg0, n0, n_end;
		tile_columns(g, cluster / g.m_tiles, seg, seg0, n0, n_end);
		const int q = warp & 3, row = q * 32 + lane, row0 = (cluster % g.m_tiles) * 256 + half * 128 + q * 32;
		const int share = g.n_tile / g.splits;                    // columns (per matrix) that a pair finishes: a multiple of 32
		const int mats = GLU ? 2 : 1, words = share * mats * 128; // floats that one pair sends another (per CTA)
		const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
		float4 next[ADD ? 8 : 1];
		if (warp >= 2) {
			if constexpr (ADD) load_residual(g, next, row0, n0 + part * share, n_end);
			mbar_wait_warp(acc_full0, 0, dead);
			__syncwarp();
			tc_fence_after();
		}
		__syncwarp();
		cluster_sync(); // every pair's products are complete: the stages may be overwritten
		if (warp >= 2) {
			for (int p = 0; p < g.splits; ++p) {
				if (p == part) continue;
				// slot of this pair in p's buffer: pairs in order, p itself left out; a float4 of columns per thread, rows side by side
				const uint32_t dst = map_rank(base, (uint32_t)(2 * p + half)) + (uint32_t)((part < p ? part : part - 1) * words) * 4;
				for (int m = 0; m < mats; ++m)
#pragma unroll 1
					for (int c0 = 0; c0 < share; c0 += 32) {
						float v[32];
						tmem_ld32(trow + m * g.n_tile + p * share + c0, v);
						if (dead)
							for (int i = 0; i < 32; ++i) v[i] = kNaN;
#pragma unroll
						for (int i = 0; i < 32; i += 4)
							st_cluster4(dst + (uint32_t)((((m * share + c0 + i) >> 2) * 128 + row) * 16), make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
					}
			}
		}
		__syncwarp();
		cluster_sync(); // the other pairs' sums of this pair's columns are here
		if (warp >= 2 && row0 < g.M) {
			const uint32_t patch = patch0 + q * kPatch;
#pragma unroll 1
			for (int c0 = part * share; c0 < (part + 1) * share; c0 += 32) {
				float4 x[ADD ? 8 : 1];
				if constexpr (ADD) {
#pragma unroll
					for (int i = 0; i < 8; ++i) x[i] = next[i];
					if (c0 + 32 < (part + 1) * share) load_residual(g, next, row0, n0 + c0 + 32, n_end);
				}
				float v[32], u[GLU ? 32 : 1];
				auto total = [&](float (&out)[32], int m) { // the parts of K in order
					float own[32];
					tmem_ld32(trow + m * g.n_tile + c0, own);
#pragma unroll
					for (int i = 0; i < 32; ++i) out[i] = 0.f;
#pragma unroll 1
					for (int p = 0; p < g.splits; ++p) {
						if (p == part) {
#pragma unroll
							for (int i = 0; i < 32; ++i) out[i] += own[i];
							continue;
						}
						const uint32_t src = base + (uint32_t)((p < part ? p : p - 1) * words) * 4;
#pragma unroll
						for (int i = 0; i < 32; i += 4) {
							const float4 o = ld_shared4(src + (uint32_t)((((m * share + c0 - part * share + i) >> 2) * 128 + row) * 16));
							out[i] += o.x, out[i + 1] += o.y, out[i + 2] += o.z, out[i + 3] += o.w;
						}
					}
				};
				total(v, 0);
				if constexpr (GLU) {
					total(u, 1);
#pragma unroll
					for (int i = 0; i < 32; ++i) v[i] = glu(g, v[i], u[i]);
				}
				if (dead)
					for (int i = 0; i < 32; ++i) v[i] = kNaN;
				if (n0 + c0 < n_end) {
					if constexpr (KIND == kRotate) rotate_store(g, seg, patch, v, row0, n0 - seg0 + c0, n_end - seg0);
					else if constexpr (GLU) store_patch_f16(g, g.h, (size_t)g.ldc, patch, v, row0, n0 + c0, n_end);
					else store_patch_f32<ADD>(g, patch, v, x, row0, n0 + c0, n_end);
				}
			}
		}
	}
	tc_fence_before();
	__syncwarp();
	cluster_sync(); // no CTA leaves while another may still signal its barriers or work on its TMEM
	if (warp == 1) {
		tc_fence_after();
		tmem_dealloc<2>(tmem, 512);
	}
}

// Few rows: 128 rows of W (of w1 and w3 each for GLU) against all M <= 128 positions.  A cluster of `splits` CTAs shares a tile's K;
// CTA r finishes the groups of 8 positions g with g % splits == r.  TMEM lane = row of W, column = position.
// ADD: the results are added to what lies in c, a kernel of its own: with the choice made at run time plain stores paid for the residuals' registers and steps
// (100 x 6144 x 4096 16.6 us, 15.4 without; 128 x 512 x 512 9.5 and 8.1).
template <bool GLU, bool B_SEG, bool ADD>
__global__ void __launch_bounds__(kGemmThreads)
gemm_few_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ WeightMaps tb, const __grid_constant__ GemmArgs g) {
	extern __shared__ uint8_t smem_raw[];
	constexpr int MATS = GLU ? 2 : 1;
	const int np = (g.M + 15) / 16 * 16; // positions, padded to the instruction's N
	const uint32_t w_bytes = 128 * kRowBytes, a_bytes = (uint32_t)np * kRowBytes, stage_bytes = MATS * w_bytes + a_bytes;
	const uint32_t base = (s32(smem_raw) + 1023u) & ~1023u, bars = base + g.stages * stage_bytes, exch = bars + 512;
	const uint32_t full0 = bars, empty0 = bars + 8 * g.stages, acc_bar = empty0 + 8 * g.stages, tslot = acc_bar + 8;
	const int warp = uniform_warp(), lane = threadIdx.x & 31;
	const int part = g.splits > 1 ? (int)cluster_rank() : 0, tile = blockIdx.x / g.splits;
	const int nkb = (g.K + BK - 1) / BK, kb0 = part * g.kb_per, kb1 = min(nkb, kb0 + g.kb_per);
	const uint32_t cols = MATS * np <= 32 ? 32 : MATS * np <= 64 ? 64 : MATS * np <= 128 ? 128 : 256; // TMEM columns
	int seg, seg0, n0, n_end;
	tile_columns(g, tile, seg, seg0, n0, n_end);
	bool dead = false;

	if (threadIdx.x == 0) {
		for (int i = 0; i < g.stages; ++i) mbar_init(full0 + 8 * i, 1), mbar_init(empty0 + 8 * i, 1);
		mbar_init(acc_bar, 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (g.splits > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); // waited for before this CTA writes into the others
	if (warp == 0 && elect_one()) prefetch_map(&ta), prefetch_map(&tb.m[B_SEG ? seg : 0]);
	if (warp == 1) tmem_alloc<1>(tslot, cols);
	tc_fence_before();
	__syncthreads();
	chain_wait();
	chain_next();
	tc_fence_after();
	uint32_t tmem;
	asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tslot));

	if (warp == 0) {
		{ // ---- TMA producer ----
			const CUtensorMap *w = &tb.m[B_SEG ? seg : 0];
			const int w0 = B_SEG ? n0 - seg0 : n0;
			Ring ring;
			ring.phase = 1; // the first round of every stage is free
			for (int kb = kb0; kb < kb1; ++kb, ring.next(g.stages)) {
				mbar_wait_warp(empty0 + 8 * ring.s, ring.phase, dead);
				if (dead) break;
				const uint32_t dst = base + ring.s * stage_bytes, bar = full0 + 8 * ring.s;
				if (elect_one()) {
					mbar_expect_tx(bar, stage_bytes);
					tma_load_2d<1>(dst, w, kb * BK, w0, bar);
					if (GLU) tma_load_2d<1>(dst + w_bytes, &tb.m[1], kb * BK, w0, bar);
					tma_load_2d<1>(dst + MATS * w_bytes, &ta, kb * BK, seg * g.a_step, bar);
				}
			}
		}
		__syncwarp();
	} else if (warp == 1) {
		{ // ---- MMA issuer ----
			const uint32_t idesc = instr_desc_f16(128, np) | (g.bf16 ? kInstrDescBf16 : 0u);
			const uint64_t wdesc0 = smem_desc_sw128(base), vdesc0 = smem_desc_sw128(base + w_bytes), adesc0 = smem_desc_sw128(base + MATS * w_bytes);
			Ring ring;
			uint32_t more = 0;
			for (int kb = kb0; kb < kb1; ++kb, ring.next(g.stages)) {
				mbar_wait_warp(full0 + 8 * ring.s, ring.phase, dead);
				if (dead) break;
				tc_fence_after();
				const uint64_t at = (uint64_t)((ring.s * stage_bytes) >> 4);
				if (elect_one()) {
#pragma unroll
					for (int k = 0; k < BK / 16; ++k) {
						umma_f16<1>(tmem, wdesc0 + at + 2 * k, adesc0 + at + 2 * k, idesc, more | k);
						if (GLU) umma_f16<1>(tmem + np, vdesc0 + at + 2 * k, adesc0 + at + 2 * k, idesc, more | k);
					}
					umma_commit(empty0 + 8 * ring.s);
				}
				more = 1;
			}
			if (!dead && elect_one()) umma_commit(acc_bar);
		}
		__syncwarp();
	}
	// ---- tail ----
	const int q = warp & 3, row = q * 32 + lane, groups = (g.M + 7) / 8, mine = (groups + g.splits - 1) / g.splits;
	const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
	// words of a group of 8 positions: [matrix][4-position half][row][4]
	auto slot = [&](uint32_t buf, int src, int group, int m, int j) { return buf + (uint32_t)((((src * mine + group / g.splits) * MATS + m) * 2 + j) * 128 + row) * 16; };
	// residuals of this CTA's groups, kBatch groups at a time, the first while the products run: behind them every group waited for its own (1.1 of 9.4 us at
	// 17 x 4096 x 4096).  With the exchange's own space: 9.4 -> 8.8 us, 128 rows 15.8 -> 13.2, 100 x 6144 x 4096 20.8 -> 17.9, 17 x 1024 x 1024 4.5 -> 4.1
	constexpr int kBatch = ADD ? 4 : 1;
	const int col = n0 + row; // lanes are neighbouring output columns
	// (ADD says as much; without the tail asked again the compiler's order of this costs 0.3 to 2 %, 1 x 1024 x 1024 3.46 -> 3.53 us)
	const bool add = ADD && g.tail == kAddF32 && col < n_end;
	float x[kBatch][ADD ? 8 : 1];
	auto fetch = [&](int first) {
		if constexpr (ADD) {
#pragma unroll
			for (int b = 0; b < kBatch; ++b)
#pragma unroll
				for (int i = 0; i < 8; ++i) {
					const int r = (first + b * g.splits) * 8 + i;
					x[b][i] = add && r < g.M ? g.c[(size_t)r * g.ldc + col] : 0.f;
				}
		}
	};
	if (warp >= 2) {
		fetch(part);
		mbar_wait_warp(acc_bar, 0, dead);
		__syncwarp();
		tc_fence_after();
	}
	__syncwarp();
	if (g.splits > 1) {
		asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); // the other CTAs run
		if (warp >= 2)
			for (int gr = 0; gr < groups; ++gr) {
				const int p = gr % g.splits;
				if (p == part) continue;
				const uint32_t buf = map_rank(exch, (uint32_t)p);
#pragma unroll
				for (int m = 0; m < MATS; ++m) {
					float v[8];
					tmem_ld8(trow + m * np + gr * 8, v);
					if (dead)
						for (int i = 0; i < 8; ++i) v[i] = kNaN;
					st_cluster4(slot(buf, part < p ? part : part - 1, gr, m, 0), make_float4(v[0], v[1], v[2], v[3]));
					st_cluster4(slot(buf, part < p ? part : part - 1, gr, m, 1), make_float4(v[4], v[5], v[6], v[7]));
				}
			}
		__syncwarp();
		cluster_sync(); // the other CTAs' sums of this CTA's positions are here
	}
	if (warp >= 2) {
		for (int g0 = part; g0 < groups; g0 += kBatch * g.splits) {
			if (g0 != part) fetch(g0);
#pragma unroll
			for (int b = 0; b < kBatch; ++b) {
				const int gr = g0 + b * g.splits;
				if (gr >= groups) break;
				__syncwarp();
				float v[MATS][8];
#pragma unroll
				for (int m = 0; m < MATS; ++m) {
					float own[8];
					tmem_ld8(trow + m * np + gr * 8, own);
#pragma unroll
					for (int i = 0; i < 8; ++i) v[m][i] = 0.f;
					for (int p = 0; p < g.splits; ++p) { // the parts of K in order
						if (p == part) {
#pragma unroll
							for (int i = 0; i < 8; ++i) v[m][i] += own[i];
							continue;
						}
						const float4 lo = ld_shared4(slot(exch, p < part ? p : p - 1, gr, m, 0)), hi = ld_shared4(slot(exch, p < part ? p : p - 1, gr, m, 1));
						v[m][0] += lo.x, v[m][1] += lo.y, v[m][2] += lo.z, v[m][3] += lo.w, v[m][4] += hi.x, v[m][5] += hi.y, v[m][6] += hi.z, v[m][7] += hi.w;
					}
				}
				if (col < n_end) {
					const int rows = min(8, g.M - gr * 8);
					if (GLU) {
						__half *dst = g.h + (size_t)(gr * 8) * g.ldc + col;
#pragma unroll
						for (int i = 0; i < 8; ++i) v[0][i] = dead ? kNaN : glu(g, v[0][i], v[MATS - 1][i]);
#pragma unroll
						for (int i = 0; i < 8; ++i)
							if (i < rows) dst[(size_t)i * g.ldc] = __float2half_rn(v[0][i]);
					} else {
						float *dst = g.c + (size_t)(gr * 8) * g.ldc + col;
#pragma unroll
						for (int i = 0; i < 8; ++i)
							if (i < rows) dst[(size_t)i * g.ldc] = dead ? kNaN : (ADD ? x[b][ADD ? i : 0] : 0.f) + g.alpha * v[0][i];
					}
				}
			}
		}
		tc_fence_before();
	}
	__syncthreads();
	if (warp == 1) {
		tc_fence_after();
		tmem_dealloc<1>(tmem, cols);
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

// (rows, cols) row-major 16-bit matrix -> tensor map with a box_rows x 64-column box, 128-byte swizzle, zero fill past the edges
static int make_map(CUtensorMap *map, const void *ptr, int rows, int cols, int box_rows, bool bf16) {
	EncodeTiledFn fn = encode_fn();
	if (!fn) return YALM_EINVAL;
	const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
	const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
	const cuuint32_t box[2] = {BK, (cuuint32_t)box_rows}, estr[2] = {1, 1};
	const CUresult r = fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
	                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
	                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	return r == CUDA_SUCCESS ? 0 : YALM_EINVAL;
}

constexpr int kMaxDevices = 64;

static int column_tiles(const GemmArgs &g, int n) {
	int tiles = 0;
	for (int i = 0, at = 0; i < g.nseg; ++i) tiles += (g.seg_end[i] - at + n - 1) / n, at = g.seg_end[i];
	return tiles;
}

static size_t pair_stage_bytes(bool glu, int n) { return (size_t)(128 + (glu ? n : n / 2)) * kRowBytes; }
static int pair_stages(bool glu, int n) { return (int)std::min<size_t>(10, 196608 / pair_stage_bytes(glu, n)); }
static size_t pair_smem(bool glu, int n) { return pair_stages(glu, n) * pair_stage_bytes(glu, n) + kTailBytes + 1024; }

// Tile width and K parts of the pair kernel, by estimated cycles: waves of tiles x K blocks x (190 + 2.05 per accumulator column and block, the
// MMA and what a block costs beside it), the last tail, and with K parts the exchange.  The constants are fitted to sweeps over both at 256 .. 512
// rows: 4096 x 4096 in one part 32.1 us at 256 columns, 21.3 at 128, in two 23.0; 2048 x 8192 44.2 (128 columns, one part) against 30.8 (two); 1024 x 4096
// 23.4 (64, one) against 16.7 (two) and 25.7 (256, four: a cluster of 8 costs some 8 us).  slots: clusters of 2, 4, 8 CTAs that run at once.
// Parts of K only where all tiles run at once.
static void plan_pair(GemmArgs &g, bool glu, const int (&slots)[3]) {
	const int nkb = (g.K + BK - 1) / BK;
	double best = 1e30;
	g.m_tiles = (g.M + 255) / 256;
	const int widest = glu ? 128 : 256, step = glu ? 16 : 32;
	for (int si = 0; si < 3; ++si) {
		const int S = 1 << si, per = (nkb + S - 1) / S;
		if (S > 1 && (nkb < 8 * S || (nkb + per - 1) / per != S)) break; // (the last part must not be empty)
		for (int n = widest; n >= 2 * step; n -= step) {
			if (S > 1 && n % (32 * S)) continue;
			const int items = g.m_tiles * column_tiles(g, n);
			if (slots[si] < 1 || (S > 1 && items > slots[si])) continue;
			const int waves = (items + slots[si] - 1) / slots[si], nacc = glu ? 2 * n : n;
			const double cost = waves * per * (190 + 2.05 * nacc) + 16.0 * nacc / S + (S > 1 ? (S == 2 ? 1000 : 15000) + 36.0 * nacc : 0);
			if (cost < best * 0.999) best = cost, g.n_tile = n, g.splits = S, g.items = items, g.kb_per = per;
		}
	}
	g.stages = pair_stages(glu, g.n_tile);
}

template <int KIND>
static int launch_pair(GemmArgs &g, const void *a, int a_rows, const void *const (&w)[3], const int (&w_rows)[3], int nw, cudaStream_t st) {
	constexpr bool GLU = KIND == kGlu;
	static int slots[kMaxDevices][3]; // 0: not asked yet
	static std::mutex mu;
	auto kernel = gemm_pair_kernel<KIND>;
	const int dev = device_info().device;
	if (dev < 0 || dev >= kMaxDevices) return YALM_EINVAL;
	int here[3];
	{
		std::lock_guard<std::mutex> lock(mu);
		if (!slots[dev][0]) {
			const size_t most = pair_smem(GLU, GLU ? 128 : 256);
			YALM_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(most + 4096)));
			for (int i = 2; i >= 0; --i) {
				cudaLaunchConfig_t cfg = {};
				cfg.gridDim = dim3(2 << i), cfg.blockDim = dim3(kGemmThreads), cfg.dynamicSmemBytes = most;
				cudaLaunchAttribute at[1];
				at[0].id = cudaLaunchAttributeClusterDimension;
				at[0].val.clusterDim.x = 2 << i, at[0].val.clusterDim.y = 1, at[0].val.clusterDim.z = 1;
				cfg.attrs = at, cfg.numAttrs = 1;
				YALM_TRY(cudaOccupancyMaxActiveClusters(&slots[dev][i], kernel, &cfg));
			}
		}
		for (int i = 0; i < 3; ++i) here[i] = slots[dev][i];
	}
	if (here[0] < 1) return (int)cudaErrorLaunchOutOfResources;
	if (KIND == kScore) here[1] = here[2] = 0; // a row's sum over a tile needs the whole products
	plan_pair(g, GLU, here);
	CUtensorMap ta;
	WeightMaps tb;
	int rc = make_map(&ta, a, a_rows, g.K, 128, g.bf16);
	for (int i = 0; i < 3 && !rc; ++i) {
		if (i < nw) rc = make_map(&tb.m[i], w[i], w_rows[i], g.K, GLU ? g.n_tile : g.n_tile / 2, g.bf16);
		else tb.m[i] = tb.m[0];
	}
	if (rc) return rc;
	const int clusters = g.splits > 1 ? g.items : std::min(g.items, here[0]);
	return launch_chained(kernel, dim3(clusters * 2 * g.splits), dim3(kGemmThreads), pair_smem(GLU, g.n_tile), st, 2 * g.splits, ta, tb, g);
}

// Few rows: an SM's shared memory for stages, or half of it (two CTAs at once) where there are more tiles than SMs.  K parts
// while every CTA still has an SM to itself: more CTAs than SMs would halve the stages of each.
template <bool GLU, bool B_SEG, bool ADD>
static int launch_few(GemmArgs &g, const void *a, int a_rows, const void *const (&w)[3], const int (&w_rows)[3], int nw, cudaStream_t st) {
	static bool configured[kMaxDevices];
	static std::mutex mu;
	auto kernel = gemm_few_kernel<GLU, B_SEG, ADD>;
	const DeviceInfo &d = device_info();
	if (d.device < 0 || d.device >= kMaxDevices) return YALM_EINVAL;
	const int np = (g.M + 15) / 16 * 16, mats = GLU ? 2 : 1, nkb = (g.K + BK - 1) / BK;
	const size_t stage = (size_t)(mats * 128 + np) * kRowBytes;
	g.n_tile = 128, g.m_tiles = 1, g.items = column_tiles(g, 128);
	g.splits = 1, g.kb_per = nkb;
	for (int S = 2; S <= 8 && nkb >= 4 * S && g.items * S <= d.sms; S *= 2) {
		const int per = (nkb + S - 1) / S;
		if ((nkb + per - 1) / per == S) g.splits = S, g.kb_per = per; // (the last part must not be empty)
	}
	// the exchange has space of its own, so that no CTA waits for the others' products before it sends: (parts - 1) x groups of 8 positions per CTA x 4 KB x matrices
	const size_t groups = ((g.M + 7) / 8 + g.splits - 1) / g.splits, exchange = (size_t)(g.splits - 1) * groups * mats * 4096;
	const size_t room = g.items * g.splits <= d.sms ? std::min<size_t>(212992, d.max_smem_optin - 1536 - exchange) : 106496;
	g.stages = std::max(2, std::min(std::min(16, g.kb_per), (int)(room / stage)));
	const size_t smem = g.stages * stage + exchange + 512 + 1024;
	if ((int)smem > d.max_smem_optin) return YALM_EINVAL;
	{
		std::lock_guard<std::mutex> lock(mu);
		if (!configured[d.device]) {
			YALM_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, d.max_smem_optin));
			configured[d.device] = true;
		}
	}
	CUtensorMap ta;
	WeightMaps tb;
	int rc = make_map(&ta, a, a_rows, g.K, np, g.bf16);
	for (int i = 0; i < 3 && !rc; ++i) {
		if (i < nw) rc = make_map(&tb.m[i], w[i], w_rows[i], g.K, 128, g.bf16);
		else tb.m[i] = tb.m[0];
	}
	if (rc) return rc;
	return launch_chained(kernel, dim3(g.items * g.splits), dim3(kGemmThreads), smem, st, g.splits, ta, tb, g);
}

// Where the few-rows kernel ends: 128 positions are one operand of it, and up to there it is ahead of the pairs (4096 x 14336: 43 us
// against 53 at 128 rows, 35 against 53 at 1 row).  With two matrices its two 128-row products read as much shared memory a cycle as
// there is from about 80 positions on (14336 x 4096: 65.6 us against 67.6 at 64 rows, 73.8 against 68.3 at 128).
template <bool GLU>
static int launch(GemmArgs &g, const void *a, int a_rows, const void *const (&w)[3], const int (&w_rows)[3], int nw, cudaStream_t st) {
	const bool few = g.M <= kFewRows / (GLU ? 2 : 1);
	if constexpr (!GLU)
		if (g.tail == kAddF32) return few ? launch_few<false, false, true>(g, a, a_rows, w, w_rows, nw, st) : launch_pair<kResidual>(g, a, a_rows, w, w_rows, nw, st);
	if (few) return launch_few<GLU, false, false>(g, a, a_rows, w, w_rows, nw, st);
	return launch_pair<GLU ? kGlu : kPlain>(g, a, a_rows, w, w_rows, nw, st);
}

// c (M, ldc) fp32 = a (M, K) fp16 times the rows of wq, wk and wv, side by side: the three projections of a layer as one launch, of up to 128 rows.
int gemm_qkv_f16(float *c, int ldc, const void *a, const void *wq, const void *wk, const void *wv, int M, int q_dim, int kv_dim, int K, cudaStream_t st) {
	if (M > kFewRows) return YALM_EINVAL;
	GemmArgs g{M, q_dim + 2 * kv_dim, K, kStoreF32, 0, c, nullptr, ldc, 1.0f, 0, 3, {q_dim, q_dim + kv_dim, q_dim + 2 * kv_dim}, 0};
	return launch_few<false, true, false>(g, a, M, {wq, wk, wv}, {q_dim, kv_dim, kv_dim}, 3, st);
}

// The same for more rows than the few-rows kernel takes, finished: q (M, q_dim) fp16 rotated, k and v rotated and appended at positions pos0 .. of their
// head-major rings.  turns: (M, head_dim / 2) cosines and sines.  Saves the fp32 rows on their way to a kernel of their own and back (512 rows of 32 + 2 x 8
// heads of 128: four layers and a head 1268 -> 1221 us).
int gemm_qkv_rotate(void *q, void *k, void *v, const void *turns, const void *a, const void *wq, const void *wk, const void *wv, int M, int q_dim, int kv_dim, int K,
                    int head_dim, int ring, int pos0, float clip, cudaStream_t st) {
	if (M <= kFewRows || head_dim % 32) return YALM_EINVAL;
	GemmArgs g{M, q_dim + 2 * kv_dim, K, kStoreF32, 0, nullptr, nullptr, 0, 1.0f, 0, 3, {q_dim, q_dim + kv_dim, q_dim + 2 * kv_dim}, 0};
	g.rotate = {static_cast<__half *>(q), static_cast<__half *>(k), static_cast<__half *>(v), static_cast<const float2 *>(turns), head_dim, ring, pos0, clip};
	return launch_pair<kRotate>(g, a, M, {wq, wk, wv}, {q_dim, kv_dim, kv_dim}, 3, st);
}

// Probability of every row's target column under the softmax of its row of a w^T (src/sampler.cpp:11-25), the products themselves not stored: (maximum, sum)
// of every column tile, joined tile by tile (512 rows of 32000 columns were 65 MB to store and to read: four layers and a head 1221 -> 1180 us).
// kFewRows < M <= kPortionRows.  scratch: a float for every row, then (tile, row) float2.
__global__ void __launch_bounds__(256) join_scores_kernel(const float2 *parts, const float *at_target, const int *targets, float *probs, int tiles, int M, int N) {
	chain_wait();
	chain_next();
	const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
	if (row >= M) return;
	float m = -FLT_MAX, l = 0.f; // (finite, as of a tile whose columns are all -infinity)
	for (int i = lane; i < tiles; i += 32) {
		const float2 p = parts[(size_t)i * kPortionRows + row];
		const float top = fmaxf(m, p.x);
		l = l * expf(m - top) + p.y * expf(p.x - top);
		m = top;
	}
	const float top = warp_max(m);
	l = warp_sum(l * expf(m - top));
	const int t = targets[row];
	if (lane == 0) probs[row] = (t >= 0 && t < N) ? expf(at_target[row] - top) / l : 0.f;
}
size_t score_bytes(int N) { return ((size_t)((N + 63) / 64) * 2 + 1) * kPortionRows * sizeof(float); } // (tiles of 64 columns at least)
int gemm_score(float *probs, void *scratch, const int *targets, const void *a, const void *w, int M, int N, int K, cudaStream_t st) {
	if (M <= kFewRows || M > kPortionRows || N % 4) return YALM_EINVAL; // (N as for stored rows)
	GemmArgs g{M, N, K, kStoreF32, 0, nullptr, nullptr, 0, 1.0f, 0, 1, {N}, 0};
	float *at_target = static_cast<float *>(scratch);
	g.score = {reinterpret_cast<float2 *>(at_target + kPortionRows), at_target, targets};
	if (int rc = launch_pair<kScore>(g, a, M, {w, nullptr, nullptr}, {N, 0, 0}, 1, st)) return rc;
	return launch_chained(join_scores_kernel, dim3((M + 7) / 8), dim3(256), 0, st, 1, (const float2 *)g.score.parts, (const float *)at_target, targets, probs,
	                      g.items / g.m_tiles, M, N);
}

} // namespace prefill
} // namespace yalm

using namespace yalm;
using namespace yalm::prefill;

// c (M, ldc) fp32 (=|+=) a (M, K) fp16 * w (N, K)^T fp16.  a, w, c: device pointers, 16-byte aligned rows (K % 8 == 0).
extern "C" int yalm_gemm_16(float *c, int ldc, const void *a, const void *w, int M, int N, int K, int accumulate, int bf16, float alpha, yalm_stream_t s) {
	if (!c || !a || !w || M < 1 || N < 1 || K < 8 || K % 8 || ldc < N || ldc % 4 || ((uintptr_t)a & 15) || ((uintptr_t)w & 15) || ((uintptr_t)c & 15))
		return YALM_EINVAL;
	GemmArgs g{M, N, K, accumulate ? kAddF32 : kStoreF32, 0, c, nullptr, ldc, alpha, bf16 != 0, 1, {N}, 0};
	return launch<false>(g, a, M, {w, nullptr, nullptr}, {N, 0, 0}, 1, (cudaStream_t)s);
}
// The same with one input per segment of output columns: columns [segment_end[i - 1], segment_end[i]) of c = a_i w^T, a_i = rows
// i M .. i M + M - 1 of a (n_segments M, K).  Segment bounds are multiples of 4 (the last one is N).
extern "C" int yalm_gemm_16_segments(float *c, int ldc, const void *a, const void *w, int M, int N, int K, int n_segments, const int *segment_end, int bf16,
                                     yalm_stream_t s) {
	if (!c || !a || !w || M < 1 || N < 1 || K < 8 || K % 8 || ldc < N || ldc % 4 || ((uintptr_t)a & 15) || ((uintptr_t)w & 15) || ((uintptr_t)c & 15) || n_segments < 1 ||
	    n_segments > kSegments || !segment_end || segment_end[n_segments - 1] != N)
		return YALM_EINVAL;
	GemmArgs g{M, N, K, kStoreF32, 0, c, nullptr, ldc, 1.0f, bf16 != 0, n_segments, {}, M};
	for (int i = 0, at = 0; i < n_segments; ++i) {
		if (segment_end[i] <= at || (i + 1 < n_segments && segment_end[i] % 4)) return YALM_EINVAL;
		g.seg_end[i] = at = segment_end[i];
	}
	return launch<false>(g, a, n_segments * M, {w, nullptr, nullptr}, {N, 0, 0}, 1, (cudaStream_t)s);
}
extern "C" int yalm_gemm_f16(float *c, int ldc, const void *a, const void *w, int M, int N, int K, int accumulate, yalm_stream_t s) {
	return yalm_gemm_16(c, ldc, a, w, M, N, K, accumulate, 0, 1.0f, s);
}

// h (M, ldh) fp16 = act(a w1^T) * (a w3^T): the fused w1 / w3 projection + GLU of the FFN (src/infer.cpp:360-375).
extern "C" int yalm_gemm_glu_f16(void *h, int ldh, const void *a, const void *w1, const void *w3, int M, int N, int K, int act,
                                 yalm_stream_t s) {
	if (!h || !a || !w1 || !w3 || M < 1 || N < 1 || K < 8 || K % 8 || ldh < N || ldh % 8) return YALM_EINVAL;
	GemmArgs g{M, N, K, kGluF16, act, nullptr, static_cast<__half *>(h), ldh, 1.0f, 0, 1, {N}, 0};
	return launch<true>(g, a, M, {w1, w3, nullptr}, {N, N, 0}, 2, (cudaStream_t)s);
}

// Host-pointer test entry: c (M, N) fp32 = a (M, K) fp16 * w (N, K)^T fp16 [+ c]; w3 != NULL: h (M, N) fp16 = GLU.
extern "C" int yalm_gemm_host(float *c, void *h, const void *a, const void *w, const void *w3, int M, int N, int K, int accumulate,
                              int act) {
	int n = 0;
	if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) return YALM_ENOGPU;
	if ((!c && !h) || !a || !w || M < 1 || N < 1 || K < 8) return YALM_EINVAL;
	void *da = nullptr, *dw = nullptr, *dw3 = nullptr, *dc = nullptr;
	const size_t ab = (size_t)M * K * 2, wb = (size_t)N * K * 2, cb = (size_t)M * N * (w3 ? 2 : 4);
	YALM_TRY(cudaMalloc(&da, ab));
	YALM_TRY(cudaMalloc(&dw, wb));
	YALM_TRY(cudaMalloc(&dc, cb));
	YALM_TRY(cudaMemcpy(da, a, ab, cudaMemcpyHostToDevice));
	YALM_TRY(cudaMemcpy(dw, w, wb, cudaMemcpyHostToDevice));
	int rc;
	if (w3) {
		YALM_TRY(cudaMalloc(&dw3, wb));
		YALM_TRY(cudaMemcpy(dw3, w3, wb, cudaMemcpyHostToDevice));
		rc = yalm_gemm_glu_f16(dc, N, da, dw, dw3, M, N, K, act, nullptr);
	} else {
		YALM_TRY(cudaMemcpy(dc, c, cb, cudaMemcpyHostToDevice));
		rc = yalm_gemm_f16(static_cast<float *>(dc), N, da, dw, M, N, K, accumulate, nullptr);
	}
	if (!rc) rc = (int)cudaDeviceSynchronize();
	if (!rc) rc = (int)cudaMemcpy(w3 ? h : (void *)c, dc, cb, cudaMemcpyDeviceToHost);
	cudaFree(da), cudaFree(dw), cudaFree(dw3), cudaFree(dc);
	return rc;
}
