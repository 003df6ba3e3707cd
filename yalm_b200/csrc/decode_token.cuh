// Whole-token persistent decode kernel for dense models on one GPU: the phases, hand-over words and arithmetic of decode_mega.cuh (which serves mixtures
// of experts, several GPUs and what it is faster at: token_geometry(), decode_mega.cu) with another division of the work inside a CTA.
//
// 12 warps, one CTA per SM, cooperative launch.  Two warps stream the CTA's rows of every matrix, the norms' weights and its pieces of the KV ring, phase after
// phase, through a ring of 24 stages of 8 KB (cp.async.bulk, mbarriers): they wait for free stages and for nothing else.  The other eight:
//   * The rows of a product.  A stage is a row (a piece of a long one, several short ones) and all eight warps share it: a warp always holds the same
//     columns, so its part of the input vector stays in registers and is polled for by this warp alone, with no staging in shared memory and no CTA barrier
//     in front of the first product.  The last bytes of a phase are done with a few hundred cycles after they land (a warp per row group takes 2.4 us over
//     its last tiles).  The warps' sums of up to 64 rows meet in shared memory, then a thread per row (or pair) runs the epilogue: norm scale (the
//     norm's weights are applied to the vector, its scale to the sums), clip, RoPE and append; residual, kept in shared memory by the CTA that owns the
//     row; act x up; logits.
//   * Attention.  A task is up to four query heads of one KV head over half a stage (8 positions of 128 channels).  q and the appended key and value
//     travel as flagged words too, so no grid barrier stands before it (but for a ring that has wrapped, whose sink keys are rotated in place).  The CTAs'
//     partial sums are flagged words; every CTA of the head joins its slice of the outputs.
// The hand-over buffers are used again a layer later.  That is safe because every CTA owns a row of wo and of w2 (token_geometry() sees to it) and
// stores it when all its warps have read that phase's input, and those of the phases before; the next phase's input needs every such row.  So whoever stores into a buffer a second
// time has waited for every CTA's row of a product that comes after its reading of the first.
//
// Bound by HBM inside the phases (w1 / w3 235 MB in 35 us) and by the hand-overs between them.  A layer of 4096 / 14336 at 4096 positions, us, here and with
// decode_mega.cuh: q k v 9.7 / 11, attention 8.7 / 13, wo 6.4 / 9, w1 w3 37.9 / 37, w2 21.7 / 24: 85 / 94; four layers and the head, a call on the host 461 -> 437;
// three layers at 600 positions on the device, 2048 / 7168 149 -> 123, 1024 / 3584 112 -> 77.  Without any copies a layer takes 75, with no arithmetic on rows and keys 75.  What shaped it:
//   * Registers.  Any spill in the row loops is a round trip to an L2 that is busy with the weights: 100 bytes of them cost 10 us a layer.  Hence eight warps
//     with 224 registers (setmaxnreg) instead of 16 with 112, q in shared memory, vectors polled for 32 words at a time.
//   * One instruction for the barriers of four stages (lane l asks for stage l % 8) and no branches around the loads: with a wait, a release and two
//     branches for each stage in turn, w1 / w3 took 60 us.
//   * Stages freed four at a time: eight at a time is 20 % less work and still slower under load, the ring being that much shorter.
//
// A wait that runs out (a bug) turns what the warp computes into NaN, its later waits return at once, and the kernel leaves a record, which the host reads behind
// the launch and fails on (mega.h: fault_record, check_fault).  Such a warp gives no stage back, so the stream gives up in turn and waits for its own copies, again with a
// limit, before it leaves.
#pragma once

#include "decode_mega.cuh"
#include "stream_rows.cuh"

#include <type_traits>

namespace yalm {
namespace mega {
namespace token {

constexpr int kW = kTokenWarps, kTokenThreads = 32 * (kW + 4), kCT2 = 32 * kW, kCap = 64, kChunk = 512;
constexpr int kFloats = 64; // of an input vector in a lane's registers
constexpr int kOffRope2 = 0, kOffRed2 = 512, kOffMisc2 = 640, kOffLayer = 720, kOffZero = 1136, kOffFull2 = 1152, kOffEmpty2 = kOffFull2 + 8 * kTokenStages, kOffPart = 2048;
constexpr int kIssuers = 2;
static_assert(kTokenStages % kIssuers == 0, "a stage is one warp's");
static_assert(kOffLayer + 2 * sizeof(Layer) <= kOffZero && kOffZero + 16 <= kOffFull2 && kOffEmpty2 + 8 * kTokenStages <= kOffPart, "header");
constexpr int kOffRes = kOffPart + 2 * kW * kCap * 4, kOffRec = kOffRes + 4 * kTokenMaxRows;
__host__ __device__ constexpr int task_heads(int g) { return g < 4 ? g : 4; } // query heads of an attention task
// the warps' records of an attention (also, after them, the partial joins), its weights, the KV head's queries, the ring
__host__ __device__ constexpr int off_ps(int hd, int g) { return (kOffRec + kW * task_heads(g) * (hd + 2) * 4 + 127) / 128 * 128; }
__host__ __device__ constexpr int off_q(int hd, int g) { return off_ps(hd, g) + kW * (kStageBytes / (8 * hd)) * task_heads(g) * 4; }
__host__ __device__ constexpr int off_ring(int hd, int g) { return off_q(hd, g) + g * hd * 4; }
constexpr size_t smem_bytes(int hd, int g) { return off_ring(hd, g) + (size_t)kTokenStages * kStageBytes; }

constexpr int kMiscTok = 16, kMiscPos = 17, kMiscGen = 18; // words of the scratch behind the warps' own
// Registers a thread: 12 warps get 168 at launch (plan_token() checks it); the stream's group gives most of its share to the others.
constexpr int kStreamRegs = 56, kRowRegs = 224;
constexpr bool regs_suffice(int at_launch) { return (at_launch + 7) / 8 * 8 * kTokenThreads >= kCT2 * kRowRegs + (kTokenThreads - kCT2) * kStreamRegs; }

__device__ __forceinline__ void tbar() { asm volatile("bar.sync 1, %0;" ::"n"(kCT2) : "memory"); }

// Bounded waits.  Nobody traps: whoever gave up goes on with NaN.  (No calls in them: what lives across a call is spilled.)
constexpr long long kPatience = 8000000000ll; // cycles, some 4 s, unless YALM_MEGA_TIMEOUT_S says otherwise (g_timeout_cycles, looked up when a wait is long)
__device__ __forceinline__ bool out_of_patience(long long t0) {
	const long long waited = clock64() - t0;
	return waited > 1000000 && waited > *(volatile long long *)&g_timeout_cycles;
}
__device__ __forceinline__ void wait_stage(uint32_t bar, uint32_t parity, bool &dead) { // whole warp
	if (__all_sync(kFull, mbar_try_wait(bar, parity))) return;
	dead = __any_sync(kFull, dead);
	const long long t0 = clock64();
	while (!dead && !__all_sync(kFull, mbar_try_wait(bar, parity))) dead = __any_sync(kFull, out_of_patience(t0));
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) { // does not wait
	uint32_t ok;
	asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
	return ok != 0;
}

// Rows of one phase: np pieces of a row, `piece` chunks of 512 bytes each, RS rows in a stage.  Up to 8 chunks a row: a warp holds one chunk of two rows of a
// stage (RS / 2 rows side by side, then as many more); longer rows: two chunks of every stage.
struct Geo {
	int np, piece, RS;
};

// Four consecutive 64-bit words, one request in flight per pair; good: all carry the flag.
struct Words4 {
	ulonglong2 a, b;
	__device__ __forceinline__ void load(const unsigned long long *p) { a = ll_load2(p), b = ll_load2(p + 2); }
	__device__ __forceinline__ bool good(unsigned flag) const { return ll_ok(a.x, flag) && ll_ok(a.y, flag) && ll_ok(b.x, flag) && ll_ok(b.y, flag); }
	__device__ __forceinline__ float4 value() const { return make_float4(ll_val(a.x), ll_val(a.y), ll_val(b.x), ll_val(b.y)); }
};
struct Backoff {
	int round = 0;
	long long t0 = 0;
	__device__ __forceinline__ bool over() { // sleeps; true once patience is at its end
		if (round == 0) t0 = clock64();
		__nanosleep((unsigned)YALM_MEGA_LL_NS << min(round, 4));
		++round;
		return out_of_patience(t0);
	}
};
// DT: weight type, HD: head size, G: query heads per KV head
template <int DT, int HD, int G>
__global__ void __launch_bounds__(kTokenThreads, 1) decode_token_kernel(const __grid_constant__ Args a) {
	using T = WTraits<DT>;
	constexpr int B = T::BYTES, EP = T::EP, CH = 32 * EP, Q = EP / 4;
	constexpr float NaN = __builtin_nanf("");
	extern __shared__ __align__(1024) unsigned char smem_raw[];
	unsigned char *sm = smem_raw;
	const uint32_t sm0 = smem_u32(sm), full0 = sm0 + kOffFull2, empty0 = sm0 + kOffEmpty2, ring0 = sm0 + off_ring(HD, G);
	float2 *rope = reinterpret_cast<float2 *>(sm + kOffRope2);
	float *red = reinterpret_cast<float *>(sm + kOffRed2), *part = reinterpret_cast<float *>(sm + kOffPart), *xres = reinterpret_cast<float *>(sm + kOffRes);
	int *misc = reinterpret_cast<int *>(sm + kOffMisc2);
	const int cta = blockIdx.x, ncta = gridDim.x, tid = threadIdx.x, lane = tid & 31;
	const int warp = __shfl_sync(kFull, tid >> 5, 0);
	const int n_phases = a.n_layers * 5 + (a.mode != kHydrate ? 1 : 0);
	bool dead = false;

	int kv_sink, kv_pos, kv_len;
	{
		const int tok = a.token < 0 ? a.ctl[CTL_TOKEN] : a.token, pos = a.token < 0 ? a.ctl[CTL_POS] : a.pos;
		mega::derive_ring(pos, a.max_seq_len, &kv_sink, &kv_pos, &kv_len);
		if (tid < 4) reinterpret_cast<int *>(sm + kOffZero)[tid] = 0;
		if (tid == 0) misc[kMiscTok] = tok, misc[kMiscPos] = pos, misc[kMiscGen] = 0;
	}
	if (tid == 0) {
		for (int i = 0; i < kTokenStages; ++i) mbar_init(full0 + 8 * i, 1), mbar_init(empty0 + 8 * i, kW);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	__syncthreads();

	// rows (or pairs, or positions' chunks) of phase kind k that this CTA owns
	auto share = [&](int items, int &lo, int &n) {
		lo = (int)((unsigned)cta * (unsigned)items / (unsigned)ncta), n = (int)((unsigned)(cta + 1) * (unsigned)items / (unsigned)ncta) - lo;
	};
	auto geo_of = [&](int k) { return Geo{a.token_geo[k][0], a.token_geo[k][1], a.token_geo[k][2]}; }; // 0: dim, 1: q_dim, 2: hidden

	if (warp >= kW) { // ================================ the stream ================================
		asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kStreamRegs));
		// two warps take the stages in turn (one thread issues a copy in some 130 cycles, and a stage is due every 330); the other two only complete the
		// group whose registers change hands
		if (warp >= kW + kIssuers) return;
		const uint64_t policy = policy_evict_first();
		const uint32_t mine = (uint32_t)(warp - kW);
		uint32_t s = mine, phase = 1, turn = 0; // the first round of every stage is free; turn: index % kIssuers of the next stage in the whole sequence
		auto acquire = [&](uint32_t &dst, uint32_t &bar) { // false: another warp's stage
			const bool yes = turn == mine;
			turn = turn + 1 == kIssuers ? 0 : turn + 1;
			if (!yes) return false;
			wait_stage(empty0 + 8 * s, phase, dead);
			dst = ring0 + s * kStageBytes, bar = full0 + 8 * s;
			s += kIssuers;
			if (s >= kTokenStages) s -= kTokenStages, phase ^= 1;
			return !dead; // (left earlier, where it gave up, it took 12 us a layer: place and address were no longer the same for the whole warp)
		};
		for (int ph = 0; ph < n_phases && !dead; ++ph) {
			const int l = min(ph / 5, a.n_layers - 1), k = ph < a.n_layers * 5 ? ph % 5 : 5;
			const Layer &L = a.layers[l];
			uint32_t dst, bar;
			if (k == 1) {
				constexpr int C = kStageBytes / (4 * HD);
				const AttnSplit sp = attn_split(cta, ncta, a.n_kv_heads, (kv_len + C - 1) / C);
				const char *kc = reinterpret_cast<const char *>(L.kc), *vc = reinterpret_cast<const char *>(L.vc);
				for (int i = 0; i < sp.nu && !dead; ++i) {
					const int r0 = (sp.k0 + i) * C;
					const uint32_t bytes = (uint32_t)min(C, kv_len - r0) * HD * 2;
					const size_t off = ((size_t)sp.kvh * a.max_seq_len + r0) * HD * 2;
					if (acquire(dst, bar) && elect_one()) {
						mbar_expect_tx(bar, 2 * bytes);
						bulk_g2s(dst, kc + off, bytes, bar, policy);
						bulk_g2s(dst + kStageBytes / 2, vc + off, bytes, bar, policy);
					}
					__syncwarp();
				}
				continue;
			}
			const Geo ge = geo_of(k == 2 ? 1 : k == 4 ? 2 : 0);
			const size_t row_bytes = (size_t)(k == 2 ? a.q_dim : k == 4 ? a.hidden : a.dim) * B;
			int lo, n;
			if (k == 0) share((a.q_dim + 2 * a.kv_dim) / 2, lo, n), lo *= 2, n *= 2;
			else share(k == 3 ? a.hidden : k == 5 ? a.vocab : a.dim, lo, n);
			const char *m = k == 0 ? L.wq : k == 2 ? L.wo : k == 3 ? L.w1 : k == 4 ? L.w2 : a.wcls;
			const uint32_t piece_bytes = (uint32_t)ge.piece * kChunk;
			const float *norm = k == 0 ? L.rms_att : k == 3 ? L.rms_ffn : k == 5 ? a.rms_final : nullptr;
			for (uint32_t off = 0; norm && off < (uint32_t)a.dim * 4u; off += kStageBytes) // the norm's weights
				if (acquire(dst, bar) && elect_one()) {
					const uint32_t bytes = min((uint32_t)kStageBytes, (uint32_t)a.dim * 4u - off);
					mbar_expect_tx(bar, bytes);
					bulk_g2s_plain(dst, reinterpret_cast<const char *>(norm) + off, bytes, bar);
				}
			const int groups = (n + ge.RS - 1) / ge.RS * (k == 3 ? 2 : 1);
			for (int g = 0; g < groups && !dead; ++g) {
				const int first = (k == 3 ? g >> 1 : g) * ge.RS, rows = min(ge.RS, n - first);
				int row = lo + first;
				for (int p = 0; p < ge.np; ++p) {
					const uint32_t off = p * piece_bytes;
					if (acquire(dst, bar) && elect_one()) {
						if (ge.RS == 1) {
							const char *src = m;
							int r = row;
							if (k == 0 && row >= a.q_dim) { // q rows, then k, then v
								r -= a.q_dim, src = L.wk;
								if (r >= a.kv_dim) r -= a.kv_dim, src = L.wv;
							} else if (k == 3 && (g & 1)) src = L.w3;
							const uint32_t bytes = min(piece_bytes, (uint32_t)row_bytes - off);
							mbar_expect_tx(bar, bytes);
							bulk_g2s(dst, src + (size_t)r * row_bytes + off, bytes, bar, policy);
						} else {
							mbar_expect_tx(bar, (uint32_t)(rows * row_bytes));
							for (int done = 0; done < rows;) { // a run of rows of one matrix
								const char *src = k == 3 && (g & 1) ? L.w3 : m;
								int r = row + done, run = rows - done;
								if (k == 0) {
									int end = a.q_dim;
									if (r >= a.q_dim + a.kv_dim) src = L.wv, r -= a.q_dim + a.kv_dim, end = a.kv_dim;
									else if (r >= a.q_dim) src = L.wk, r -= a.q_dim, end = a.kv_dim;
									run = min(run, end - r);
								}
								bulk_g2s(dst + (uint32_t)(done * row_bytes), src + (size_t)r * row_bytes, (uint32_t)(run * row_bytes), bar, policy);
								done += run;
							}
						}
					}
					__syncwarp();
				}
			}
		}
		// its own copies have landed before it leaves (the parity that a stage's last one completes is that of the round in which it would be free; the stage that
		// it gave up on, if it did, was not filled and runs out)
		bool late = false;
		for (int i = 0; i < kTokenStages / kIssuers; ++i) {
			wait_stage(full0 + 8 * s, phase, late);
			s += kIssuers;
			if (s >= kTokenStages) s -= kTokenStages, phase ^= 1;
		}
		return;
	}

	// ================================ the other warps ================================
	asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRowRegs));
	// RoPE table of this token: cos/sin(pos * theta^(-j/rotary_dim)) with the reference's fp32 formula (src/infer.cpp:200-213)
	if (tid < HD / 2) {
		const int j = 2 * tid;
		const float freq = j >= a.rotary_dim ? 0.f : 1.0f / powf(a.theta, (float)j / (float)a.rotary_dim);
		const float val = misc[kMiscPos] * freq;
		rope[tid] = make_float2(cosf(val), sinf(val));
	}
	// the layer's pointers, from shared memory (a global load here is a round trip to L2), fetched a layer ahead
	Layer *layer = reinterpret_cast<Layer *>(sm + kOffLayer);
	auto fetch_layer = [&](int l) {
		if (l < a.n_layers && lane < (int)(sizeof(Layer) / 8)) reinterpret_cast<unsigned long long *>(layer + (l & 1))[lane] = reinterpret_cast<const unsigned long long *>(a.layers + l)[lane];
	};
	if (warp == 0) fetch_layer(0);
	auto embed4 = [&](int e) {
		const int tok = misc[kMiscTok];
		const size_t base = (size_t)tok * a.dim + e;
		const float sc = (DT == YALM_F8E4M3 && a.embed_scale) ? a.embed_scale[tok] : 1.0f;
		return make_float4(T::to_float(a.embed, base) * sc, T::to_float(a.embed, base + 1) * sc, T::to_float(a.embed, base + 2) * sc, T::to_float(a.embed, base + 3) * sc);
	};
	int row0, nrows; // this CTA's rows of x
	share(a.dim, row0, nrows);
	for (int i = tid; i < nrows; i += kCT2) {
		const int tok = misc[kMiscTok];
		const float sc = (DT == YALM_F8E4M3 && a.embed_scale) ? a.embed_scale[tok] : 1.0f;
		xres[i] = T::to_float(a.embed, (size_t)tok * a.dim + row0 + i) * sc;
	}
	tbar();

	uint32_t s = 0, sphase = 0; // this warp's place in the ring
	// Up to eight stages at once: lane l looks after stage l % 8, so that waits and releases cost a warp one instruction and not four in a row.
	auto stage_of_lane = [&](uint32_t &st, uint32_t &par) {
		st = s + (lane & 7), par = sphase;
		if (st >= kTokenStages) st -= kTokenStages, par ^= 1;
	};
	auto landed = [&](int m) { // the next m <= 8 stages
		uint32_t st, par;
		stage_of_lane(st, par);
		bool ok = (lane & 7) >= m || mbar_try_wait(full0 + 8 * st, par);
		if (!__all_sync(kFull, ok)) {
			dead = __any_sync(kFull, dead);
			const long long t0 = clock64();
			while (!dead) {
				ok = (lane & 7) >= m || mbar_try_wait(full0 + 8 * st, par);
				if (__all_sync(kFull, ok)) break;
				dead = __any_sync(kFull, out_of_patience(t0));
			}
		}
		__syncwarp();
	};
	auto peek = [&](int m) { // this lane's one of the next m stages has landed: asked before work that does not need them, whose time hides the answer's
		uint32_t st, par;
		stage_of_lane(st, par);
		return (lane & 7) >= m || mbar_test(full0 + 8 * st, par);
	};
	auto leave = [&](int m) { // this warp has read them
		uint32_t st, par;
		stage_of_lane(st, par);
		__syncwarp();
		if (lane < m && !dead) mbar_arrive(empty0 + 8 * st); // (who gave up gives nothing back: it could be filled again under a copy on its way)
		s += m;
		if (s >= kTokenStages) s -= kTokenStages, sphase ^= 1;
	};
	auto stage_at = [&](int u) { // address of the stage u < 8 ahead
		const uint32_t t = s + u;
		return ring0 + (t >= kTokenStages ? t - kTokenStages : t) * kStageBytes;
	};
	int flip = 0;
	const int c_kv_len = kv_len;
	auto grid_wait = [&]() { // all CTAs; the release / acquire of the memory before it
		tbar();
		if (tid == 0) {
			const unsigned target = (unsigned)++misc[kMiscGen] * (unsigned)ncta;
			asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.sync) : "memory");
			unsigned v;
			const long long t0 = clock64();
			do {
				asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.sync) : "memory");
				if (v < target && out_of_patience(t0)) dead = true;
			} while (v < target && !dead);
			asm volatile("fence.acq_rel.gpu;" ::: "memory");
		}
		tbar();
	};
	const int cta_of_launch = cta;
	for (int ph = 0; ph < n_phases; ++ph) {
		// (opaque: what follows from them is the same in every phase, and kept in registers all the time it had the row loops spill)
		int cta = cta_of_launch, lane = tid & 31, kv_len = c_kv_len;
		asm volatile("" : "+r"(cta), "+r"(lane), "+r"(kv_len));
		const int l = min(ph / 5, a.n_layers - 1), k = ph < a.n_layers * 5 ? ph % 5 : 5;
		const Layer &L = layer[l & 1];
		const unsigned wflag = ll_flag(a.seq, ph + 1), rflag = ll_flag(a.seq, ph);
		auto mark = [&](int slot) {
			if (a.prof && tid == 0) a.prof[(((size_t)cta * a.n_layers + l) * kProfPhases + k) * kProfSlots + slot] = clock64();
		};
		mark(0);
		if (k == 1) {
			// ---- attention: fp32 dots over fp16 keys, / sqrt(head size) on q, exp(s - max) / sum, fp32 mix over fp16 values (src/infer.cpp:216-248) ----
			constexpr int kHeads = task_heads(G), LPR = HD / 8, RPS = 32 / LPR, C = kStageBytes / (4 * HD), ST = C / RPS / 2, V = ST * kHeads, NF = V / LPR, SB = ST / NF, HG = G / kHeads, UL = kW / HG, UB = UL / 2;
			static_assert(ST == 4 && V % LPR == 0 && SB * kHeads == LPR && G % kHeads == 0 && kW % HG == 0, "head size / group");
			if (kv_sink > 0) grid_wait(); // the sink keys are rotated in place
			if (warp == kW - 1) fetch_layer(l + 1); // (that record's readers are a layer behind)
			mark(1);
			const int sub = lane % LPR, rgrp = lane / LPR, hg = warp % HG, ul = warp / HG;
			const int my_h = sub / SB, my_st0 = (sub % SB) * NF; // this lane owns scores of head my_h of the task, steps my_st0 .. + NF
			const int nch = (kv_len + C - 1) / C;
			const AttnSplit sp = attn_split(cta, ncta, a.n_kv_heads, nch);
			float *rec = reinterpret_cast<float *>(sm + kOffRec);
			float *ps = reinterpret_cast<float *>(sm + off_ps(HD, G)) + warp * (C / 2) * kHeads; // weights of the task: [row group][head][step]
			if (sp.nu > 0) {
				float2 acc[kHeads][4];
				float *qs = reinterpret_cast<float *>(sm + off_q(HD, G));
				for (int e = tid * 2; e < G * HD; e += kCT2 * 2) { // the KV head's queries, / sqrt(head size)
					const unsigned long long *src = a.ll_q + (size_t)(cta % kLLRep) * a.q_dim + (size_t)sp.kvh * G * HD + e;
					Backoff wait;
					ulonglong2 w = ll_load2(src);
					while (!(ll_ok(w.x, rflag) && ll_ok(w.y, rflag)) && !dead) dead = wait.over(), w = ll_load2(src);
					const float div = sqrtf((float)HD);
					*reinterpret_cast<float2 *>(qs + e) = make_float2(ll_val(w.x) / div, ll_val(w.y) / div);
				}
				tbar();
				const uint32_t q0 = sm0 + off_q(HD, G) + (uint32_t)(hg * kHeads * HD + sub * 8) * 4;
#pragma unroll
				for (int h = 0; h < kHeads; ++h)
#pragma unroll
					for (int j = 0; j < 4; ++j) acc[h][j] = make_float2(0.f, 0.f);
				mark(2);
				float m = -INFINITY, lsum = 0.f; // of head my_h: maximum (the same in all its lanes), this lane's part of the sum
#pragma unroll 1
				for (int i0 = 0; i0 < sp.nu; i0 += UB) { // UB stages at a time: this warp takes half of one
					const int here = min(UB, sp.nu - i0), i = i0 + ul / 2;
					landed(here);
					const int t0 = (sp.k0 + i) * C + (ul & 1) * (C / 2), n = min(C / 2, kv_len - t0); // first position, how many
					if (i < i0 + here && n > 0) {
						const uint32_t at = stage_at(ul / 2) + (ul & 1) * (kStageBytes / 4), ks = at + lane * 16, vs = ks + kStageBytes / 2; // step st at + 512 st
						// the row appended by this token and the rotated sink keys were written after the copy: into the stage, from their words and from L2
						const int fresh = kv_pos - t0;
						if (fresh >= 0 && fresh < n) {
							const uint32_t row = at + fresh * HD * 2;
							constexpr int PER = HD / 32; // words of this lane: of the key, then of the value
							unsigned long long w[PER];
							const unsigned long long *src = a.ll_kv + (size_t)sp.kvh * (HD / 2);
							Backoff wait;
							for (;;) {
								bool good = true;
#pragma unroll
								for (int x = 0; x < PER; ++x) {
									const int j = lane + 32 * x;
									w[x] = ll_load1(src + (j < HD / 2 ? j : a.kv_dim / 2 + j - HD / 2));
								}
#pragma unroll
								for (int x = 0; x < PER; ++x) good = good && ll_ok(w[x], rflag);
								if (good || dead) break;
								dead = wait.over();
							}
#pragma unroll
							for (int x = 0; x < PER; ++x) {
								const int j = lane + 32 * x;
								asm volatile("st.shared.u32 [%0], %1;" ::"r"(row + (j < HD / 2 ? j * 4 : kStageBytes / 2 + (j - HD / 2) * 4)), "r"((unsigned)w[x]) : "memory");
							}
						}
						if (t0 < kv_sink)
							for (int j = lane; j < min(n, kv_sink - t0) * (HD / 2); j += 32) {
								const unsigned v = __ldcg(reinterpret_cast<const unsigned *>(L.kc) + ((size_t)sp.kvh * a.max_seq_len + t0) * (HD / 2) + j);
								asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + j * 4), "r"(v) : "memory");
							}
						if ((fresh >= 0 && fresh < n) || t0 < kv_sink) {
							asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // (before the next copy into the stage)
							__syncwarp();
						}
						float d[V];
						float2 kf[ST][4];
#pragma unroll
						for (int st = 0; st < ST; ++st) {
							const uint4 kv = lds128(ks + st * 512);
							kf[st][0] = WTraits<YALM_F16>::h2(kv.x), kf[st][1] = WTraits<YALM_F16>::h2(kv.y), kf[st][2] = WTraits<YALM_F16>::h2(kv.z), kf[st][3] = WTraits<YALM_F16>::h2(kv.w);
						}
#pragma unroll
						for (int h = 0; h < kHeads; ++h) {
							const float4 lo = lds128f(q0 + h * HD * 4), hi = lds128f(q0 + h * HD * 4 + 16);
#pragma unroll
							for (int st = 0; st < ST; ++st) {
								float2 s2 = ffma2(make_float2(lo.x, lo.y), kf[st][0], make_float2(0.f, 0.f));
								s2 = ffma2(make_float2(lo.z, lo.w), kf[st][1], s2), s2 = ffma2(make_float2(hi.x, hi.y), kf[st][2], s2), s2 = ffma2(make_float2(hi.z, hi.w), kf[st][3], s2);
								d[h * ST + st] = s2.x + s2.y;
							}
						}
						int nv = V; // each exchange halves the values a lane carries: value h ST + st ends in lane sub = (h ST + st) / NF
#pragma unroll
						for (int o = LPR / 2; o > 0; o >>= 1) {
							const bool up = (sub & o) != 0;
							nv /= 2;
#pragma unroll
							for (int x = 0; x < V / 2; ++x)
								if (x < nv) d[x] = (up ? d[x + nv] : d[x]) + __shfl_xor_sync(kFull, up ? d[x] : d[x + nv], o);
						}
						float mt = -INFINITY;
#pragma unroll
						for (int x = 0; x < NF; ++x) {
							if ((my_st0 + x) * RPS + rgrp >= n) d[x] = -INFINITY;
							mt = fmaxf(mt, d[x]);
						}
#pragma unroll
						for (int o = 1; o < SB; o <<= 1) mt = fmaxf(mt, __shfl_xor_sync(kFull, mt, o));
#pragma unroll
						for (int o = LPR; o < 32; o <<= 1) mt = fmaxf(mt, __shfl_xor_sync(kFull, mt, o));
						const float m_new = fmaxf(m, mt); // finite: every stage has a row
						const float corr = m == -INFINITY ? 0.f : __expf(m - m_new);
						m = m_new, lsum *= corr;
						__syncwarp(); // the task before has read its weights
#pragma unroll
						for (int x = 0; x < NF; ++x) {
							const float p = d[x] == -INFINITY ? 0.f : __expf(d[x] - m_new);
							lsum += p;
							ps[(rgrp * kHeads + my_h) * ST + my_st0 + x] = p;
						}
						__syncwarp();
						float c2[kHeads]; // every head's correction
						float4 pw[kHeads];
#pragma unroll
						for (int h = 0; h < kHeads; ++h) c2[h] = __shfl_sync(kFull, corr, h * SB), pw[h] = *reinterpret_cast<const float4 *>(ps + (rgrp * kHeads + h) * ST);
#pragma unroll
						for (int h = 0; h < kHeads; ++h)
#pragma unroll
							for (int j = 0; j < 4; ++j) acc[h][j].x *= c2[h], acc[h][j].y *= c2[h];
#pragma unroll
						for (int st = 0; st < ST; ++st) {
							if (st * RPS + rgrp >= n) continue; // (what lies there is no value: zero times it need not be zero)
							const uint4 vv = lds128(vs + st * 512);
							const float2 v0 = WTraits<YALM_F16>::h2(vv.x), v1 = WTraits<YALM_F16>::h2(vv.y), v2 = WTraits<YALM_F16>::h2(vv.z), v3 = WTraits<YALM_F16>::h2(vv.w);
#pragma unroll
							for (int h = 0; h < kHeads; ++h) {
								const float p = st == 0 ? pw[h].x : st == 1 ? pw[h].y : st == 2 ? pw[h].z : pw[h].w;
								const float2 pp = make_float2(p, p);
								acc[h][0] = ffma2(pp, v0, acc[h][0]), acc[h][1] = ffma2(pp, v1, acc[h][1]);
								acc[h][2] = ffma2(pp, v2, acc[h][2]), acc[h][3] = ffma2(pp, v3, acc[h][3]);
							}
						}
					}
					leave(here);
				}
				dead = __any_sync(kFull, dead);
				// this warp's record: its row groups joined
#pragma unroll
				for (int o = LPR; o < 32; o <<= 1) {
					lsum += __shfl_xor_sync(kFull, lsum, o);
#pragma unroll
					for (int h = 0; h < kHeads; ++h)
#pragma unroll
						for (int j = 0; j < 4; ++j) acc[h][j].x += __shfl_xor_sync(kFull, acc[h][j].x, o), acc[h][j].y += __shfl_xor_sync(kFull, acc[h][j].y, o);
				}
#pragma unroll
				for (int o = 1; o < SB; o <<= 1) lsum += __shfl_xor_sync(kFull, lsum, o);
				if (dead) lsum = NaN;
				if (rgrp == 0) {
#pragma unroll
					for (int h = 0; h < kHeads; ++h)
#pragma unroll
						for (int j = 0; j < 4; ++j) *reinterpret_cast<float2 *>(rec + (warp * kHeads + h) * (HD + 2) + sub * 8 + 2 * j) = acc[h][j];
					if (sub % SB == 0) rec[(warp * kHeads + my_h) * (HD + 2) + HD] = m, rec[(warp * kHeads + my_h) * (HD + 2) + HD + 1] = lsum;
				}
				mark(5);
				tbar();
				for (int o = tid; o < G * HD; o += kCT2) { // the warps' records in order -> this CTA's partial
					const int h = o / HD, d = o % HD;
					const float *r = rec + ((h / kHeads) * kHeads + h % kHeads) * (HD + 2); // warp u HG + h / 2 of unit lane u
					float mm[UL], M = -INFINITY, ls = 0.f, v = 0.f;
#pragma unroll
					for (int u = 0; u < UL; ++u) mm[u] = r[u * HG * kHeads * (HD + 2) + HD], M = fmaxf(M, mm[u]);
#pragma unroll
					for (int u = 0; u < UL; ++u) {
						const float w = mm[u] == -INFINITY ? 0.f : expf(mm[u] - M);
						v = fmaf(w, r[u * HG * kHeads * (HD + 2) + d], v), ls = fmaf(w, r[u * HG * kHeads * (HD + 2) + HD + 1], ls); // (an empty record is zero)
					}
					ll_store(a.ll_acc + (((size_t)sp.kvh * ncta + cta) * G + h) * HD + d, v, wflag);
					if (d == 0) ll_store2(a.ll_ml + (((size_t)sp.kvh * ncta + cta) * G + h) * 2, M, ls, wflag);
				}
				mark(7);
			}
			// ---- this CTA's slice of the head's outputs: a lane per output, a warp per CTAs w, w + 8, .. that hold positions, then the warps' joins in order ----
			const int r = cta - sp.c0, o_lo = r * (G * HD) / sp.nc, o_hi = (r + 1) * (G * HD) / sp.nc;
			float *join = reinterpret_cast<float *>(sm + kOffRec); // [maximum, sum, value][warp][lane]
			for (int ob = o_lo; ob < o_hi; ob += 32) {
				const int o = min(ob + lane, o_hi - 1), h = o / HD;
				constexpr int AT = 3; // partners in flight
				ulonglong2 w[AT];
				unsigned long long x[AT];
				bool there[AT];
				auto partners = [&](int p0) {
					const unsigned long long *ml[AT], *ac[AT];
#pragma unroll
					for (int i = 0; i < AT; ++i) {
						const int p = p0 + i * kW;
						there[i] = p < sp.nc && attn_has_unit(p, sp.nc, nch);
						ml[i] = a.ll_ml + (((size_t)sp.kvh * ncta + sp.c0 + p) * G + h) * 2, ac[i] = a.ll_acc + ((size_t)sp.kvh * ncta + sp.c0 + p) * G * HD + o;
					}
					Backoff wait;
					for (;;) {
						bool good = true;
#pragma unroll
						for (int i = 0; i < AT; ++i)
							if (there[i]) w[i] = ll_load2(ml[i]), x[i] = ll_load1(ac[i]);
#pragma unroll
						for (int i = 0; i < AT; ++i)
							if (there[i]) good = good && ll_ok(w[i].x, wflag) && ll_ok(w[i].y, wflag) && ll_ok(x[i], wflag);
						if (good || dead) break;
						dead = wait.over();
					}
				};
				float M = -INFINITY, ls = 0.f, v = 0.f;
				for (int p0 = warp; p0 < sp.nc; p0 += kW * AT) {
					partners(p0);
#pragma unroll
					for (int i = 0; i < AT; ++i)
						if (there[i]) M = fmaxf(M, ll_val(w[i].x));
				}
				tbar(); // (the records, and the join before, have been read)
				join[warp * 32 + lane] = M;
				tbar();
#pragma unroll
				for (int u = 0; u < kW; ++u) M = fmaxf(M, join[u * 32 + lane]); // of the head, before any weight
				for (int p0 = warp; p0 < sp.nc; p0 += kW * AT) {
					if (sp.nc > kW * AT) partners(p0); // (else they are still here)
#pragma unroll
					for (int i = 0; i < AT; ++i)
						if (there[i]) {
							const float pm = ll_val(w[i].x), f = pm == -INFINITY ? 0.f : expf(pm - M);
							ls = fmaf(f, ll_val(w[i].y), ls), v = fmaf(f, ll_val(x[i]), v);
						}
				}
				join[(kW + warp) * 32 + lane] = dead ? NaN : ls, join[(2 * kW + warp) * 32 + lane] = v;
				tbar();
				if (warp == (l & (kW - 1)) && ob + lane < o_hi) {
					float l2 = 0.f, v2 = 0.f;
#pragma unroll
					for (int u = 0; u < kW; ++u) l2 += join[(kW + u) * 32 + lane], v2 += join[(2 * kW + u) * 32 + lane];
					const float out = v2 / l2;
#pragma unroll
					for (int rp = 0; rp < kLLRep; ++rp) ll_store(a.ll_att + (size_t)rp * a.q_dim + (size_t)sp.kvh * G * HD + o, out, wflag);
					a.att_out[(size_t)sp.kvh * G * HD + o] = out;
				}
			}
			mark(3);
			continue;
		}

		// ---- a product: the warp's part of the input vector ----
		const Geo ge = geo_of(k == 2 ? 1 : k == 4 ? 2 : 0);
		const int n_in = k == 2 ? a.q_dim : k == 4 ? a.hidden : a.dim;
		int lo, n; // this CTA's rows (pairs of rows of w1 and w3)
		if (k == 0) share((a.q_dim + 2 * a.kv_dim) / 2, lo, n), lo *= 2, n *= 2;
		else share(k == 3 ? a.hidden : k == 5 ? a.vocab : a.dim, lo, n);
		// SIDES: two rows a stage and warp, one chunk of the vector; else one row, SL chunks: two of each piece
		auto product = [&](auto sides, auto slots) {
		constexpr bool SIDES = decltype(sides)::value;
		constexpr int SL = decltype(slots)::value;
		const bool norm = SL <= 2 && (k == 0 || k == 3 || k == 5); // (normed rows are one piece: plan_token())
		const int CW = SIDES ? ge.piece : kW, RG = SIDES ? ge.RS / 2 : 1; // warps that share a row; rows side by side
		const int c = SIDES ? warp % ge.piece : warp, rg = SIDES ? warp / ge.piece : 0;
		auto at_of = [&](int q) { return ((q >> 1) * ge.piece + (q & 1) * kW + c) * CH + lane * EP; }; // first element of this lane in slot q
		unsigned have = 0; // bit q: this lane holds 16 bytes of slot q
#pragma unroll
		for (int q = 0; q < SL; ++q)
			if (rg < RG && (SIDES || ((q >> 1) < ge.np && (q & 1) * kW + c < ge.piece)) && at_of(q) < n_in) have |= 1u << q;
		float4 x[SL][Q];
		{
#pragma unroll
			for (int p = 0; p < SL; ++p)
#pragma unroll
				for (int j = 0; j < Q; ++j) x[p][j] = make_float4(0.f, 0.f, 0.f, 0.f);
			mark(1);
			if (ph == 0) {
#pragma unroll
				for (int p = 0; p < SL; ++p)
					if (have >> p & 1u)
#pragma unroll
						for (int j = 0; j < Q; ++j) x[p][j] = embed4(at_of(p) + 4 * j);
			} else {
				const unsigned long long *src = k == 2 ? a.ll_att : k == 3 ? a.ll_x : k == 4 ? a.ll_hb : a.ll_x + (size_t)kLLRep * a.dim;
				src += (size_t)(cta % kLLRep) * n_in;
				constexpr int AT = SL < 16 / EP ? SL : 16 / EP; // 16 words in flight
#pragma unroll
				for (int p0 = 0; p0 < SL; p0 += AT) {
					Backoff wait;
					for (;;) {
						Words4 w[AT][Q];
#pragma unroll
						for (int p = p0; p < p0 + AT; ++p)
							if (have >> p & 1u)
#pragma unroll
								for (int j = 0; j < Q; ++j) w[p - p0][j].load(src + at_of(p) + 4 * j);
						bool good = true; // (kept whether good or not: what is not is loaded again, and no second copy of the vector is live)
#pragma unroll
						for (int p = p0; p < p0 + AT; ++p)
							if (have >> p & 1u)
#pragma unroll
								for (int j = 0; j < Q; ++j) good = good && w[p - p0][j].good(rflag), x[p][j] = w[p - p0][j].value();
						if (good || dead) break;
						dead = wait.over();
					}
				}
				dead = __any_sync(kFull, dead);
			}
			mark(2);
			if (norm) { // o = x * (1 / sqrt(mean + eps)) * w (src/infer.cpp:134-144): the scale waits for the sums, the weights come ahead of the rows
				float ss = 0.f;
#pragma unroll
				for (int p = 0; p < SL; ++p)
#pragma unroll
					for (int j = 0; j < Q; ++j) ss += x[p][j].x * x[p][j].x + x[p][j].y * x[p][j].y + x[p][j].z * x[p][j].z + x[p][j].w * x[p][j].w;
				ss = warp_sum(rg == 0 ? ss : 0.f);
				if (lane == 0) red[(ph & 1) * kW + warp] = ss;
				for (int t = 0; t * kStageBytes < n_in * 4; ++t) {
					landed(1);
#pragma unroll
					for (int p = 0; p < SL; ++p) {
						const int at = at_of(p) * 4 - t * kStageBytes;
						if ((have >> p & 1u) && at >= 0 && at < kStageBytes)
#pragma unroll
							for (int j = 0; j < Q; ++j) {
								const float4 g = lds128f(ring0 + s * kStageBytes + at + 16 * j);
								x[p][j] = make_float4(x[p][j].x * g.x, x[p][j].y * g.y, x[p][j].z * g.z, x[p][j].w * g.w);
							}
					}
					leave(1);
				}
			}
		}
		if (k == 0 && kv_sink > 0 && cta == ncta - 1) {
			// rotate each sink key forward by one position, fp16 -> fp32 -> fp16 (src/infer.cpp:303-317)
			const int hp = HD >> 1, npairs = kv_sink * a.n_kv_heads * hp;
			for (int p = tid; p < npairs; p += kCT2) {
				const int r = p / (a.n_kv_heads * hp), h = (p / hp) % a.n_kv_heads, i = (p % hp) * 2;
				__half2 *ptr = reinterpret_cast<__half2 *>(reinterpret_cast<__half *>(L.kc) + ((size_t)h * a.max_seq_len + r) * HD + i);
				float2 v = __half22float2(*ptr);
				rope_pair(v.x, v.y, i, 1, a.theta, a.rotary_dim);
				*ptr = __floats2half2_rn(v.x, v.y);
			}
		}

		// ---- the rows ----
		const int groups = (n + ge.RS - 1) / ge.RS * (k == 3 ? 2 : 1), per = kCap / ge.RS / 4 * 4; // groups whose sums are held at once
		// where this lane's 16 bytes lie in a stage; a lane that has none reads zeros instead
		const uint32_t zero = sm0 + kOffZero, near = c * kChunk + lane * 16 + (SIDES && rg < RG ? rg * (uint32_t)(n_in * B) : 0u),
		               far = near + (SIDES ? RG * (uint32_t)(n_in * B) : kW * kChunk);
		auto weights = [&](uint32_t st, uint32_t off, bool mine) { return lds128(mine ? st + off : zero); };
		for (int g0 = 0;; g0 += per, flip ^= 1) {
			const int g1 = min(groups, g0 + per);
			float *sums = part + flip * kW * kCap;
			auto keep = [&](float v, int g, int count, int lanes) { // a lane in `lanes` holds a sum; SIDES: two of each group
				const int i = lane / lanes, u = SIDES ? i >> 1 : i;
				if (lane % lanes == 0 && u < count && rg < RG) sums[c * kCap + (g + u - g0) * ge.RS + (SIDES ? rg + (i & 1) * RG : 0)] = dead ? NaN : v;
			};
			if constexpr (SL <= 2) {
				constexpr int AT = SIDES || EP == 16 ? 4 : 8, NY = SIDES ? 8 : AT; // stages whose sums are reduced together, loaded (and freed) 4 at a time; what lies past the last is not used
				bool there = false;
#pragma unroll 1
				for (int g = g0; g < g1; g += AT) {
					const int m = min(AT, g1 - g);
					uint4 w[AT][2];
#pragma unroll
					for (int v = 0; v < AT; v += 4) {
						const int part_of = max(0, min(4, m - v));
						if (!__all_sync(kFull, there)) landed(part_of);
						__syncwarp();
#pragma unroll
						for (int u = 0; u < 4; ++u) {
							const uint32_t st = stage_at(u);
							w[v + u][0] = weights(st, near, have & 1u), w[v + u][1] = weights(st, far, SIDES ? have & 1u : have & 2u);
						}
						leave(part_of);
						there = peek(min(4, g1 - g - v - 4)); // (of none: true)
					}
					float y[NY];
#pragma unroll
					for (int u = 0; u < NY; ++u) {
						if constexpr (SIDES) y[u] = stream::halves(stream::dot16<DT>(w[u >> 1][u & 1], x[0], 0ull));
						else y[u] = stream::halves(stream::dot16<DT>(w[u][0], x[0], 0ull)) + stream::halves(stream::dot16<DT>(w[u][1], x[SL - 1], 0ull));
					}
					keep(stream::sums_of<NY>(y, lane), g, m, 32 / NY);
				}
			} else {
				for (int g = g0; g < g1; g += 4) {
					const int m = min(4, g1 - g);
					float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
					for (int u = 0; u < m; ++u) { // a row, 4 of its pieces at a time (one that it has not reads zeros)
						uint64_t sum[4] = {0, 0, 0, 0};
#pragma unroll
						for (int p0 = 0; p0 < SL / 2; p0 += 4)
							if (p0 < ge.np) {
								constexpr int PC = SL / 2 < 4 ? SL / 2 : 4;
								uint4 w[PC][2];
								const int pieces = min(4, ge.np - p0);
								landed(pieces);
#pragma unroll
								for (int p = 0; p < PC; ++p) {
									const uint32_t st = stage_at(p);
									w[p][0] = weights(st, near, have >> (2 * (p0 + p)) & 1u), w[p][1] = weights(st, far, have >> (2 * (p0 + p)) & 2u);
								}
								leave(pieces);
#pragma unroll
								for (int p = 0; p < PC; ++p) sum[p] = stream::dot16<DT>(w[p][1], x[2 * (p0 + p) + 1], stream::dot16<DT>(w[p][0], x[2 * (p0 + p)], sum[p]));
							}
						y[3] = y[2], y[2] = y[1], y[1] = y[0]; // (a row's sum by its age: no index the compiler does not know)
						y[0] = (stream::halves(sum[0]) + stream::halves(sum[1])) + (stream::halves(sum[2]) + stream::halves(sum[3]));
					}
					const float v = stream::sums_of<4>(y, lane); // lane 8 i holds row m - 1 - i
					if (lane % 8 == 0 && lane / 8 < m) sums[c * kCap + g + m - 1 - lane / 8 - g0] = dead ? NaN : v;
				}
			}
			tbar();
			// ---- a thread per row, pair of rows, or gate and up: the warps' sums in order, then the phase's epilogue ----
			const int first = (k == 3 ? g0 >> 1 : g0) * ge.RS, count = min(n, (k == 3 ? g1 >> 1 : g1) * ge.RS) - first;
			const int i = (tid + flip * (kCT2 / 2)) & (kCT2 - 1);
			auto sum = [&](int at) {
				float t = 0.f;
				for (int w = 0; w < CW; ++w) t += sums[w * kCap + at];
				return t;
			};
			float f = 1.0f;
			if (norm) {
				float t = 0.f;
#pragma unroll
				for (int w = 0; w < kW; ++w) t += red[(ph & 1) * kW + w];
				f = 1.0f / sqrtf(t / n_in + a.eps);
			}
			if (k == 0) {
				if (2 * i < count) {
					int row = lo + first + 2 * i, which = 0;
					float v0 = sum(2 * i) * f, v1 = sum(2 * i + 1) * f;
					const float *sc = L.sq;
					if (row >= a.q_dim + a.kv_dim) which = 2, row -= a.q_dim + a.kv_dim, sc = L.sv;
					else if (row >= a.q_dim) which = 1, row -= a.q_dim, sc = L.sk;
					if (DT == YALM_F8E4M3 && sc) v0 *= sc[row], v1 *= sc[row + 1];
					v0 = clipf(v0, a.clip), v1 = clipf(v1, a.clip);
					const int j = row % HD;
					if (which < 2) { // interleaved-pair RoPE (src/infer.cpp:200-213)
						const float2 cs = rope[j >> 1];
						const float t0 = v0 * cs.x - v1 * cs.y, t1 = v0 * cs.y + v1 * cs.x;
						v0 = t0, v1 = t1;
					}
					if (which == 0) {
#pragma unroll
						for (int rp = 0; rp < kLLRep; ++rp) ll_store2(a.ll_q + (size_t)rp * a.q_dim + row, v0, v1, wflag);
						*reinterpret_cast<float2 *>(a.q + row) = make_float2(v0, v1);
					} else {
						const __half2 h = __floats2half2_rn(v0, v1);
						ll_store(a.ll_kv + ((which - 1) * a.kv_dim + row) / 2, __uint_as_float(*reinterpret_cast<const uint32_t *>(&h)), wflag);
						__half *cache = reinterpret_cast<__half *>(which == 1 ? L.kc : L.vc);
						*reinterpret_cast<__half2 *>(cache + ((size_t)(row / HD) * a.max_seq_len + kv_pos) * HD + j) = h;
					}
				}
			} else if (k == 3) {
				if (i < count) {
					const int at = SIDES ? i / ge.RS * 2 * ge.RS + i % ge.RS : 2 * i, row = lo + first + i;
					float gt = sum(at) * f, up = sum(at + ge.RS) * f;
					if (DT == YALM_F8E4M3 && L.s1) gt *= L.s1[row], up *= L.s3[row];
					const float v = (a.act == YALM_ACT_GELU ? act_gelu(gt) : act_silu(gt)) * up;
#pragma unroll
					for (int rp = 0; rp < kLLRep; ++rp) ll_store(a.ll_hb + (size_t)rp * a.hb_len + row, v, wflag);
					a.hb[row] = v;
				}
			} else if (i < count) {
				const int row = lo + first + i;
				float v = sum(i) * f;
				const float *sc = k == 2 ? L.so : k == 4 ? L.s2 : a.wcls_scale;
				if (DT == YALM_F8E4M3 && sc) v *= sc[row];
				if (k == 5) {
					a.logits[row] = v;
				} else { // x += W v (src/infer.cpp:335-337); the row's residual stays here
					v += xres[first + i];
					xres[first + i] = v;
					unsigned long long *dst = a.ll_x + (size_t)(k == 4 ? kLLRep : 0) * a.dim + row;
#pragma unroll
					for (int rp = 0; rp < kLLRep; ++rp) ll_store(dst + (size_t)rp * a.dim, v, wflag);
					if (k == 4) a.x[row] = v;
				}
			}
			if (g1 >= groups) break;
		}
		flip ^= 1;
		mark(3);
		};
		if (ge.RS > 1) product(std::true_type(), std::integral_constant<int, 1>());
		else if (ge.np == 1) product(std::false_type(), std::integral_constant<int, 2>());
		else product(std::false_type(), std::integral_constant<int, kFloats / EP>()); // w2 only
	}

	if (a.mode == kGreedy) { // greedy arg-max, first maximum wins (src/sampler.cpp:27-38): lanes -> warps -> CTA -> grid
		auto better = [](float ov, int oi, float &v, int &i) {
			if (ov > v || (ov == v && oi < i)) v = ov, i = oi;
		};
		float best_v = -FLT_MAX;
		int best_i = 0x7fffffff, lo, n;
		tbar(); // this CTA's rows are stored
		share(a.vocab, lo, n);
		for (int i = tid; i < n; i += kCT2) better(__ldcg(a.logits + lo + i), lo + i, best_v, best_i);
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			const float ov = __shfl_xor_sync(kFull, best_v, o);
			const int oi = __shfl_xor_sync(kFull, best_i, o);
			better(ov, oi, best_v, best_i);
		}
		tbar();
		if (lane == 0) red[warp] = best_v, misc[warp] = best_i;
		tbar();
		if (tid == 0) {
			for (int w = 1; w < kW; ++w) better(red[w], misc[w], best_v, best_i);
			a.amax_val[cta] = best_v, a.amax_idx[cta] = best_i;
		}
		grid_wait();
		if (cta == 0 && warp == 0) {
			best_v = -FLT_MAX, best_i = 0x7fffffff;
			for (int b = lane; b < ncta; b += 32) better(__ldcg(a.amax_val + b), __ldcg(a.amax_idx + b), best_v, best_i);
#pragma unroll
			for (int o = 16; o > 0; o >>= 1) {
				const float ov = __shfl_xor_sync(kFull, best_v, o);
				const int oi = __shfl_xor_sync(kFull, best_i, o);
				better(ov, oi, best_v, best_i);
			}
			if (lane == 0) {
				if (best_i == 0x7fffffff) best_i = 0;
				const int done = a.ctl[CTL_STEP], pos = misc[kMiscPos];
				if (a.tokens_out) a.tokens_out[done] = best_i;
				a.ctl[CTL_STEP] = done + 1, a.ctl[CTL_TOKEN] = best_i, a.ctl[CTL_POS] = pos + 1;
				int ks, kp, kl;
				mega::derive_ring(pos + 1, a.max_seq_len, &ks, &kp, &kl);
				a.ctl[CTL_SINK] = ks, a.ctl[CTL_KVPOS] = kp, a.ctl[CTL_KVLEN] = kl;
			}
		}
	}
	if (dead && lane == 0) { // which warp gave up, for the host
		unsigned *r = g_fault_rec;
		if (r && atomicCAS(r, 0u, (unsigned)kFaultToken) == 0u) {
			r[1] = cta, r[2] = tid, r[3] = 0, r[4] = 0;
			__threadfence_system();
		}
	}
	// the barrier words are zero again for the next launch
	tbar();
	if (tid == 0) {
		__threadfence();
		if (atomicAdd(a.sync + 1, 1u) + 1 == (unsigned)ncta) {
			a.sync[0] = 0, a.sync[1] = 0;
			__threadfence();
		}
	}
}

template <int DT>
inline const void *token_kernel_for(int head_dim, int g) {
#define YALM_TOKEN_CASE(HD, GG) \
	if (head_dim == HD && g == GG) return (const void *)decode_token_kernel<DT, HD, GG>;
	YALM_TOKEN_CASE(128, 4) YALM_TOKEN_CASE(128, 8) YALM_TOKEN_CASE(64, 4) YALM_TOKEN_CASE(32, 4) YALM_TOKEN_CASE(32, 2)
#undef YALM_TOKEN_CASE
	return nullptr;
}

} // namespace token
} // namespace mega
} // namespace yalm
