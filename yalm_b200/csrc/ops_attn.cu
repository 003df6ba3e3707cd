// Split-K flash-decode GQA attention over the fp16 KV ring buffer (sm_100a).
//
// Replaces the reference's three kernels attn_dot / attn_softmax / att_mix (src/infer.cu:338-524):
//  * one CTA serves ALL q-heads of a KV head, so every K/V row is read once, not n_heads/n_kv_heads
//    times, and each row is read as 16-byte lane-contiguous pieces (the reference walks one 256-byte
//    key row per thread);
//  * the sequence is split over gridDim.x CTAs per KV head (the reference's att_mix runs 32 CTAs on a
//    148-SM part) with an online softmax per group of lanes; the last CTA of each KV head to finish merges the
//    split partials (arrival counter in the workspace) — no second launch;
//  * no (n_heads, max_seq_len) score matrix round-trips through memory.
// Softmax order is irrelevant to the ring buffer, so sliding-window positions and the two attention
// sinks (rows 0-1) need no unrolling: the kernel just attends over rows [0, kv_len).
//
// Arithmetic follows the CPU reference (src/infer.cpp:216-248): fp32 dot over fp16 K, score /
// sqrtf(head_dim), exp(x - max) / sum, fp32 mix over fp16 V.
#include "attn_workspace.h"
#include "common.cuh"
#include "launch.h"

#include <cfloat>
#include <cstdio>
#include <mutex>

namespace yalm {

constexpr int kAttnThreads = 256;
constexpr int kAttnWarps = kAttnThreads / 32;
constexpr int kTile = 512; // most splits

struct AttnArgs {
	float *out;            // (n_heads*head_dim)
	const __half *kb, *vb; // head-major ring: (n_kv_heads, max_seq_len, head_dim)
	const float *q;        // (n_heads*head_dim)
	float *ws_acc;         // (n_kv_heads, S, G, HD) unnormalised partial outputs
	float *ws_ml;          // (n_kv_heads, S, G, 2)  running max, running sum
	unsigned *counters;    // (n_kv_heads) arrival counters, zero between launches
	int n_kv_heads, max_seq_len;
	int max_splits; // of which a context uses as many as have a batch of rows for every warp
	const int *ctl;
};

__device__ __forceinline__ void unpack8(uint4 v, float (&f)[8]) {
	float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&v.x));
	float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&v.y));
	float2 c = __half22float2(*reinterpret_cast<const __half2 *>(&v.z));
	float2 d = __half22float2(*reinterpret_cast<const __half2 *>(&v.w));
	f[0] = a.x, f[1] = a.y, f[2] = b.x, f[3] = b.y, f[4] = c.x, f[5] = c.y, f[6] = d.x, f[7] = d.y;
}

// A weight, c = 1 / sqrt(head size), d <= 0 the distance of a score from a maximum, both before that factor: of nearby scores it is exact, so a
// weight's error does not grow with the scores' size.  With 2^x of scores times a rounded log2(e) / sqrt(head size) instead the results were 3 to 10 % further from
// 64 bits below some thousand positions (37: 1.48e-7 for 1.32e-7) and lost digits with the scores' size; it took 3 % less time (4096 positions 9.9 us for 10.2).
__device__ __forceinline__ float weight(float d, float c) { return expf(d * c); }

// How a row's HD / 8 lanes share the scores of UN rows x G heads (value index u G + g): after the halving exchanges a lane holds N1
// complete values, index (sub / DUP) N1 + j.
// ONE: one CTA per SM, whose warps fetch ahead, instead of two.
template <int HD, int G, bool ONE>
struct Split {
	static constexpr int L = HD / 8;                   // lanes per K / V row (16 bytes each)
	static constexpr int RPW = 32 / L;                 // rows per warp step
	static constexpr int RPC = RPW * kAttnWarps;       // rows per CTA step
	static constexpr int UN = G >= 8 ? 2 : G >= 4 ? 4 : 8; // steps in flight per thread, keys and values
	static constexpr int CTAS = ONE ? 1 : 2;            // resident per SM (8 heads' queries and sums take 128 registers of a lane: always one)
	static constexpr bool AHEAD = ONE;                  // the next batch is fetched under this one's arithmetic: 64 / 8 heads of 128 at 4096 positions 15.3 -> 13.3 us, 32768
	                                                    // 69.7 -> 49.7
	static constexpr int NV = UN * G, N1 = NV > L ? NV / L : 1, DUP = NV < L ? L / NV : 1;
	static constexpr int NG = N1 < G ? N1 : G;         // heads that a lane's values belong to
	static constexpr int U0 = DUP * (N1 < G ? G / N1 : 1); // lanes sub and sub ^ U0, sub ^ 2 U0, .. hold the same heads of other rows
};

// Every group of HD / 8 lanes walks rows of its own with an online softmax in registers: no barrier until the CTA's end.  The scores of UN
// rows are reduced together by halving exchanges (UN G - 1 + .. shuffles for all of them, not log2 of them for each), which leaves about
// one exponential per lane and row batch.  Latency is what counts at a few thousand positions: a CTA's chain is control block, one batch
// of keys and values, one exchange of partials; short contexts use fewer splits (at least one batch per warp each), one split writes the
// result itself.  32 / 8 heads of 128, back to back, against a block-wide softmax per 512 rows: 37 positions 16 -> 3.9 us, 4096 19.6 -> 9.1 us, 32768
// 68 -> 30 us.  Of 4096 positions in 37 splits (two CTAs an SM) the join took 5 of 10.3 us; one atomic that releases and acquires for two fences around it, and
// (maximum, sum) read once, made that 9.5 (8 / 2 heads at 130: 5.7 -> 5.4); half the splits, which fetch ahead (launch_attn()), 9.1.
template <int HD, int G, bool ONE>
__global__ void __launch_bounds__(kAttnThreads, Split<HD, G, ONE>::CTAS) attn_decode_kernel(AttnArgs a) {
	using SP = Split<HD, G, ONE>;
	constexpr int L = SP::L, RPC = SP::RPC, UN = SP::UN, NV = SP::NV, N1 = SP::N1, DUP = SP::DUP, NG = SP::NG;
	extern __shared__ __align__(16) float smem[];
	float *o_s = smem;                         // [kAttnWarps][G][HD]
	float *w_s = o_s + kAttnWarps * G * HD;    // [splits][G] merge weights (splits <= kTile)
	__shared__ float m_s[kAttnWarps][G], l_s[kAttnWarps][G], l_all[G];
	__shared__ unsigned is_last;

	const int kvh = blockIdx.y, split = blockIdx.x;
	chain_wait();
	chain_next();
	const int kv_len = a.ctl[CTL_KVLEN];
	const int S = min(a.max_splits, max(1, (kv_len + RPC * UN - 1) / (RPC * UN))); // splits that have rows
	if (split >= S) return;
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, sub = lane % L, rgrp = lane / L;
	int per = (kv_len + S - 1) / S;
	per = (per + RPC - 1) / RPC * RPC;
	const int t_begin = min(split * per, kv_len), t_end = min(t_begin + per, kv_len);

	// q slice of this lane for each of the G heads: dims [sub*8, sub*8+8)
	const float c = 1.0f / sqrtf((float)HD); // maxima are of the scores before this factor
	float qr[G][8], acc[G][8];
#pragma unroll
	for (int g = 0; g < G; ++g) {
		const float *qp = a.q + (size_t)(kvh * G + g) * HD + sub * 8;
		const float4 lo = *reinterpret_cast<const float4 *>(qp), hi = *reinterpret_cast<const float4 *>(qp + 4);
		qr[g][0] = lo.x, qr[g][1] = lo.y, qr[g][2] = lo.z, qr[g][3] = lo.w;
		qr[g][4] = hi.x, qr[g][5] = hi.y, qr[g][6] = hi.z, qr[g][7] = hi.w;
#pragma unroll
		for (int j = 0; j < 8; ++j) acc[g][j] = 0.f;
	}
	float m[NG], l[NG]; // of this lane's heads, over its group's rows
#pragma unroll
	for (int j = 0; j < NG; ++j) m[j] = -INFINITY, l[j] = 0.f;
	const __half *kbase = a.kb + (size_t)kvh * a.max_seq_len * HD + sub * 8;
	const __half *vbase = a.vb + (size_t)kvh * a.max_seq_len * HD + sub * 8;

	uint4 kv[UN], vv[UN], kn[UN], vn[UN];
	auto fetch_rows = [&](uint4 (&k)[UN], uint4 (&v)[UN], int r0) {
#pragma unroll
		for (int u = 0; u < UN; ++u) k[u] = r0 + u * RPC < t_end ? ld_stream(kbase + (size_t)(r0 + u * RPC) * HD) : make_uint4(0, 0, 0, 0);
#pragma unroll
		for (int u = 0; u < UN; ++u) v[u] = r0 + u * RPC < t_end ? ld_stream(vbase + (size_t)(r0 + u * RPC) * HD) : make_uint4(0, 0, 0, 0);
	};
	const int r_first = t_begin + wid * SP::RPW + rgrp;
	if constexpr (SP::AHEAD) fetch_rows(kn, vn, r_first);
	for (int r0 = r_first; r0 - rgrp < t_end; r0 += RPC * UN) { // (warp-uniform bound: the shuffles need the whole warp)
		if constexpr (SP::AHEAD) {
#pragma unroll
			for (int u = 0; u < UN; ++u) kv[u] = kn[u], vv[u] = vn[u];
			fetch_rows(kn, vn, r0 + RPC * UN);
		} else
			fetch_rows(kv, vv, r0);
		float s[NV];
#pragma unroll
		for (int u = 0; u < UN; ++u) {
			float kf[8];
			unpack8(kv[u], kf);
#pragma unroll
			for (int g = 0; g < G; ++g) {
				float d = 0.f;
#pragma unroll
				for (int j = 0; j < 8; ++j) d = fmaf(qr[g][j], kf[j], d);
				s[u * G + g] = d;
			}
		}
		{
			int n = NV;
#pragma unroll
			for (int o = L / 2; o > 0; o >>= 1) {
				if (n > 1) { // lanes with bit o keep the upper half of the values
					n >>= 1;
#pragma unroll
					for (int i = 0; i < NV / 2; ++i)
						if (i < n) {
							const float give = (sub & o) ? s[i] : s[i + n], keep = (sub & o) ? s[i + n] : s[i];
							s[i] = keep + __shfl_xor_sync(kFull, give, o);
						}
				} else
					s[0] += __shfl_xor_sync(kFull, s[0], o);
			}
		}
		// this lane's values: index q = (sub / DUP) N1 + j, row q / G, head q % G
		float mx[NG];
#pragma unroll
		for (int j = 0; j < NG; ++j) mx[j] = -INFINITY;
#pragma unroll
		for (int j = 0; j < N1; ++j) {
			const int u = ((sub / DUP) * N1 + j) / G;
			if (r0 + u * RPC >= t_end) s[j] = -INFINITY;
			mx[j % NG] = fmaxf(mx[j % NG], s[j]);
		}
#pragma unroll
		for (int o = SP::U0; o < L; o <<= 1)
#pragma unroll
			for (int j = 0; j < NG; ++j) mx[j] = fmaxf(mx[j], __shfl_xor_sync(kFull, mx[j], o));
		bool grow = false;
#pragma unroll
		for (int j = 0; j < NG; ++j) grow |= mx[j] > m[j];
		if (__any_sync(kFull, grow)) {
			float f[NG];
#pragma unroll
			for (int j = 0; j < NG; ++j) {
				const float top = fmaxf(m[j], mx[j]);
				f[j] = m[j] == -INFINITY ? 0.f : weight(m[j] - top, c);
				m[j] = top, l[j] *= f[j];
			}
#pragma unroll
			for (int g = 0; g < G; ++g) {
				const float fg = __shfl_sync(kFull, f[g % NG], (g / N1) * DUP, L);
#pragma unroll
				for (int j = 0; j < 8; ++j) acc[g][j] *= fg;
			}
		}
#pragma unroll
		for (int j = 0; j < N1; ++j) {
			s[j] = s[j] == -INFINITY ? 0.f : weight(s[j] - m[j % NG], c);
			l[j % NG] += s[j];
		}
#pragma unroll
		for (int u = 0; u < UN; ++u) {
			float vf[8];
			unpack8(vv[u], vf);
#pragma unroll
			for (int g = 0; g < G; ++g) {
				const int q = u * G + g;
				const float p = __shfl_sync(kFull, s[q % N1], (q / N1) * DUP, L);
#pragma unroll
				for (int j = 0; j < 8; ++j) acc[g][j] = fmaf(p, vf[j], acc[g][j]);
			}
		}
	}

	// ---- the warp's row groups, then the CTA's warps ----
#pragma unroll
	for (int o = SP::U0; o < L; o <<= 1)
#pragma unroll
		for (int j = 0; j < NG; ++j) l[j] += __shfl_xor_sync(kFull, l[j], o);
	float f[NG];
#pragma unroll
	for (int j = 0; j < NG; ++j) {
		float top = m[j];
#pragma unroll
		for (int o = L; o < 32; o <<= 1) top = fmaxf(top, __shfl_xor_sync(kFull, top, o));
		f[j] = m[j] == -INFINITY ? 0.f : weight(m[j] - top, c);
		l[j] *= f[j], m[j] = top;
#pragma unroll
		for (int o = L; o < 32; o <<= 1) l[j] += __shfl_xor_sync(kFull, l[j], o);
	}
#pragma unroll
	for (int g = 0; g < G; ++g) {
		const float fg = __shfl_sync(kFull, f[g % NG], (g / N1) * DUP, L), mg = __shfl_sync(kFull, m[g % NG], (g / N1) * DUP, L),
		            lg = __shfl_sync(kFull, l[g % NG], (g / N1) * DUP, L);
#pragma unroll
		for (int j = 0; j < 8; ++j) {
			acc[g][j] *= fg;
#pragma unroll
			for (int o = L; o < 32; o <<= 1) acc[g][j] += __shfl_xor_sync(kFull, acc[g][j], o);
		}
		if (rgrp == 0) {
			float *dst = o_s + (wid * G + g) * HD + sub * 8;
			*reinterpret_cast<float4 *>(dst) = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
			*reinterpret_cast<float4 *>(dst + 4) = make_float4(acc[g][4], acc[g][5], acc[g][6], acc[g][7]);
		}
		if (lane == 0) m_s[wid][g] = mg, l_s[wid][g] = lg;
	}
	__syncthreads();
	float *my_acc = a.ws_acc + ((size_t)kvh * S + split) * G * HD;
	for (int i = threadIdx.x; i < G * HD; i += kAttnThreads) {
		const int g = i / HD;
		// lane w of 8 neighbours, which work on one head, has the factor of warp w
		constexpr unsigned kLanes = G * HD < 32 ? (1u << (G * HD % 32)) - 1u : kFull;
		const float mw = m_s[lane % kAttnWarps][g];
		float M = mw, v = 0.f;
#pragma unroll
		for (int o = kAttnWarps / 2; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(kLanes, M, o));
		const float fw = mw == -INFINITY ? 0.f : weight(mw - M, c);
		float sum = fw * l_s[lane % kAttnWarps][g];
#pragma unroll
		for (int o = kAttnWarps / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(kLanes, sum, o);
#pragma unroll
		for (int w = 0; w < kAttnWarps; ++w) v = fmaf(__shfl_sync(kLanes, fw, w, kAttnWarps), o_s[w * G * HD + i], v);
		if (S == 1) {
			a.out[(size_t)kvh * G * HD + i] = v / sum;
		} else {
			my_acc[i] = v;
			if (i % HD == 0) {
				float *ml = a.ws_ml + (((size_t)kvh * S + split) * G + g) * 2;
				ml[0] = M, ml[1] = sum;
			}
		}
	}
	if (S == 1) return;
	// ---- last CTA of this KV head merges the splits -------------------------------------------------
	__syncthreads();
	if (threadIdx.x == 0) { // releases what the barrier before it made visible, and acquires for the one after
		unsigned before;
		asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(a.counters + kvh) : "memory");
		is_last = before == (unsigned)(S - 1);
	}
	__syncthreads();
	if (!is_last) return;
	// a thread takes 4 columns of every GROUPS-th split: the partials of a batch are on their way before their weights are known
	constexpr int C4 = G * HD / 4, GROUPS = kAttnThreads / C4 > kAttnWarps ? kAttnWarps : kAttnThreads / C4, BATCH = 10;
	const int col = threadIdx.x % C4, grp = threadIdx.x / C4;
	const float4 *pa = reinterpret_cast<const float4 *>(a.ws_acc + (size_t)kvh * S * G * HD) + col;
	float4 in[BATCH], sum = make_float4(0.f, 0.f, 0.f, 0.f);
	auto fetch = [&](int s0) {
#pragma unroll
		for (int b = 0; b < BATCH; ++b)
			if (grp < GROUPS && s0 + b * GROUPS < S) in[b] = __ldcg(pa + (size_t)(s0 + b * GROUPS) * C4);
	};
	fetch(grp);
	for (int g = wid; g < G; g += kAttnWarps) {
		const float2 *ml = reinterpret_cast<const float2 *>(a.ws_ml) + (size_t)kvh * S * G + g;
		constexpr int KEPT = kTile / 32; // all at once, and once
		float2 part[KEPT];
		float M = -INFINITY, Lsum = 0.f;
#pragma unroll
		for (int i = 0; i < KEPT; ++i) {
			part[i] = make_float2(-INFINITY, 0.f);
			if (i * 32 + lane < S) part[i] = __ldcg(ml + (size_t)(i * 32 + lane) * G);
		}
#pragma unroll
		for (int i = 0; i < KEPT; ++i) M = fmaxf(M, part[i].x);
		M = warp_max(M);
#pragma unroll
		for (int i = 0; i < KEPT; ++i)
			if (i * 32 + lane < S) {
				const float w = part[i].x == -INFINITY ? 0.f : weight(part[i].x - M, c);
				w_s[(i * 32 + lane) * G + g] = w;
				Lsum += w * part[i].y;
			}
		Lsum = warp_sum(Lsum);
		if (lane == 0) l_all[g] = Lsum;
	}
	__syncthreads();
	for (int s0 = grp; s0 < S; s0 += BATCH * GROUPS) {
		if (s0 != grp) fetch(s0);
#pragma unroll
		for (int b = 0; b < BATCH; ++b)
			if (grp < GROUPS && s0 + b * GROUPS < S) {
				const float w = w_s[(s0 + b * GROUPS) * G + col / (HD / 4)];
				sum.x = fmaf(w, in[b].x, sum.x), sum.y = fmaf(w, in[b].y, sum.y), sum.z = fmaf(w, in[b].z, sum.z), sum.w = fmaf(w, in[b].w, sum.w);
			}
	}
	if (grp < GROUPS) reinterpret_cast<float4 *>(o_s)[grp * C4 + col] = sum;
	__syncthreads();
	for (int i = threadIdx.x; i < G * HD; i += kAttnThreads) {
		float v = 0.f;
#pragma unroll
		for (int k = 0; k < GROUPS; ++k) v += o_s[k * G * HD + i];
		a.out[(size_t)kvh * G * HD + i] = v / l_all[i / HD];
	}
	if (threadIdx.x == 0) a.counters[kvh] = 0; // ready for the next launch
}

// Generic path: any head_dim / group size, one CTA per q head, materialises the normalised attention
// row in `att` exactly like the reference (src/infer.cu:338-384) — used for shapes the fast path does
// not cover and by the mha test entry, which must return `att` (src/test.cpp:171-188).
// Bound by latency: a lane reads a row of keys, then a column of values, and adds in their order.  So it has 64 values of a key and 16 rows of values in
// flight: one by one, a layer whose weights had run through L2 since the last token paid the way to memory for each.
__global__ void __launch_bounds__(256) attn_generic_kernel(float *out, float *att, const __half *kb, const __half *vb,
                                                           const float *q, int head_dim, int n_heads, int n_kv_heads,
                                                           int max_seq_len, int kv_len_arg, const int *ctl) {
	__shared__ float red[36];
	const int h = blockIdx.x, kvh = h / (n_heads / n_kv_heads);
	const int kv_len = ctl ? ctl[CTL_KVLEN] : kv_len_arg;
	const __half *kh = kb + (size_t)kvh * max_seq_len * head_dim, *vh = vb + (size_t)kvh * max_seq_len * head_dim;
	const float *qh = q + (size_t)h * head_dim;
	float *atth = att + (size_t)h * max_seq_len;
	const bool wide = head_dim % 8 == 0 && ((uintptr_t)kb & 15) == 0;
	float mx = -INFINITY;
	for (int t = threadIdx.x; t < kv_len; t += blockDim.x) {
		const __half *k = kh + (size_t)t * head_dim;
		float s = 0.f;
		int i = 0;
		for (; wide && i + 64 <= head_dim; i += 64) {
			uint4 r[8];
#pragma unroll
			for (int u = 0; u < 8; ++u) r[u] = *reinterpret_cast<const uint4 *>(k + i + 8 * u);
#pragma unroll
			for (int e = 0; e < 64; ++e) s += qh[i + e] * __half2float(reinterpret_cast<const __half *>(r)[e]);
		}
		for (; i < head_dim; ++i) s += qh[i] * __half2float(k[i]);
		s /= sqrtf((float)head_dim);
		atth[t] = s;
		mx = fmaxf(mx, s);
	}
	mx = block_max(mx, red);
	float sum = 0.f;
	for (int t = threadIdx.x; t < kv_len; t += blockDim.x) {
		float e = expf(atth[t] - mx);
		atth[t] = e;
		sum += e;
	}
	sum = block_sum(sum, red);
	for (int t = threadIdx.x; t < kv_len; t += blockDim.x) atth[t] /= sum;
	__syncthreads();
	for (int i = threadIdx.x; i < head_dim; i += blockDim.x) {
		float v = 0.f;
		int t = 0;
		for (; t + 16 <= kv_len; t += 16) {
			float p[16];
			__half x[16];
#pragma unroll
			for (int u = 0; u < 16; ++u) p[u] = atth[t + u], x[u] = vh[(size_t)(t + u) * head_dim + i];
#pragma unroll
			for (int u = 0; u < 16; ++u) v += p[u] * __half2float(x[u]);
		}
		for (; t < kv_len; ++t) v += atth[t] * __half2float(vh[(size_t)t * head_dim + i]);
		out[(size_t)h * head_dim + i] = v;
	}
}

static int attn_splits(int n_kv_heads) {
	int s = 2 * device_info().sms / std::max(1, n_kv_heads);
	return std::max(1, std::min(s, kTile));
}

static bool attn_fast_shape(int head_dim, int g) {
	return (head_dim == 16 || head_dim == 32 || head_dim == 64 || head_dim == 128) &&
	       (g == 1 || g == 2 || g == 4 || g == 8);
}

template <int HD, int G, bool ONE>
static int launch_attn_of(AttnArgs &a, int splits, cudaStream_t st) {
	a.max_splits = splits;
	const size_t smem = ((size_t)a.max_splits * G + (size_t)kAttnWarps * G * HD) * sizeof(float);
	YALM_TRY(allow_smem((const void *)attn_decode_kernel<HD, G, ONE>, smem));
	return launch_chained(attn_decode_kernel<HD, G, ONE>, dim3(a.max_splits, a.n_kv_heads), dim3(kAttnThreads), smem, st, 1, a);
}
template <int HD, int G>
static int launch_attn(AttnArgs &a, int S, cudaStream_t st) {
	// all at once, and no more than a full ring has batches of rows for: the rest of a grid of 296 CTAs only begins and ends (32 / 8
	// heads of 128, a ring of 512 and 390 positions: 6.6 us -> 5.6; of 1024: 7.0 -> 5.9)
	using SP = Split<HD, G, (G >= 8)>;
	constexpr int kRows = SP::RPC * SP::UN;
	const int sms = device_info().sms, of_ring = (a.max_seq_len + kRows - 1) / kRows;
	const int splits = std::max(1, std::min({S, SP::CTAS * sms / a.n_kv_heads, of_ring}));
	// Four heads of 128 a kv head, more splits than SMs: half as many, one CTA an SM that fetches ahead, are joined sooner.  Keys and values out of memory, us with two CTAs an SM
	// against one: full rings, 32 / 8 heads 2048 8.0 7.6, 4096 9.8 9.4, 8192 13.3 13.1, 14336 18.3 17.5, 15360 18.5 18.5, 16384 18.6 19.3; 16 / 4 16384 14.8 13.1, 32768 20.0
	// 19.6; 4 / 1 32768 17.2 13.6, 131072 26.1 22.9; 56 / 14 1755 9.4 8.5, 7021 16.4 15.8, 8777 18.2 18.4, 9362 18.4 19.3; 40 / 10 11468 18.1 17.6, 12697 18.5 19.3.  With 15 kv heads
	// and more the few splits leave SMs idle or save little of the join: 60 / 15 4369 12.7 13.1, 64 / 16 4096 12.6 12.9, 160 / 40 2048 14.1 15.2.  The context is known on the
	// device only, so the ring decides, which is full at the end alone: of 16384 rows of 8 heads 37 positions take 3.5 3.7 (with one CTA an SM the next kernel's
	// wait for it), 390 6.6 6.3, 1000 7.1 6.6, 2500 9.6 8.5, 4096 10.0 9.5, 8192 13.3 13.0, 12000 16.5 15.7.  So: rings of up to 128 K rows of up to 8 kv heads, 116 K of up to 14.
	constexpr int kFewHeads = 14;
	const long few_rows = (a.n_kv_heads <= 8 ? 128 : 116) * 1024;
	if constexpr (HD == 128 && G == 4)
		if (splits * a.n_kv_heads > sms && a.n_kv_heads <= kFewHeads && (long)a.max_seq_len * a.n_kv_heads <= few_rows)
			return launch_attn_of<HD, G, true>(a, sms / a.n_kv_heads, st);
	return launch_attn_of<HD, G, (G >= 8)>(a, splits, st);
}

} // namespace yalm

using namespace yalm;

extern "C" size_t yalm_attn_workspace_bytes(int n_heads, int n_kv_heads, int head_dim) {
	if (n_heads <= 0 || n_kv_heads <= 0 || head_dim <= 0) return 0;
	return attn_workspace(0, n_kv_heads, attn_splits(n_kv_heads), n_heads / n_kv_heads, head_dim).bytes;
}

extern "C" int yalm_attn_decode(float *out, const uint16_t *key_cache, const uint16_t *value_cache, const float *q,
                                void *workspace, int n_heads, int n_kv_heads, int head_dim, int max_seq_len,
                                const int *ctl, yalm_stream_t s) {
	if (!out || !key_cache || !value_cache || !q || !workspace || !ctl) return YALM_EINVAL;
	if (n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads || max_seq_len <= 0) return YALM_EINVAL;
	const int g = n_heads / n_kv_heads;
	if (!attn_fast_shape(head_dim, g)) return YALM_EINVAL; // callers use yalm_attn_generic for odd shapes
	const int S = attn_splits(n_kv_heads);
	AttnArgs a;
	a.out = out, a.kb = (const __half *)key_cache, a.vb = (const __half *)value_cache, a.q = q;
	const AttnWorkspace w = attn_workspace((uintptr_t)workspace, n_kv_heads, S, g, head_dim);
	a.counters = (unsigned *)workspace;
	a.ws_ml = (float *)((char *)workspace + w.ml);
	a.ws_acc = (float *)((char *)workspace + w.acc);
	a.n_kv_heads = n_kv_heads, a.max_seq_len = max_seq_len, a.ctl = ctl;
	cudaStream_t st = (cudaStream_t)s;
#define YALM_ATTN_CASE(HD, G)                                                                                 \
	if (head_dim == HD && g == G) return launch_attn<HD, G>(a, S, st);
	YALM_ATTN_CASE(128, 1) YALM_ATTN_CASE(128, 2) YALM_ATTN_CASE(128, 4) YALM_ATTN_CASE(128, 8)
	YALM_ATTN_CASE(64, 1) YALM_ATTN_CASE(64, 2) YALM_ATTN_CASE(64, 4) YALM_ATTN_CASE(64, 8)
	YALM_ATTN_CASE(32, 1) YALM_ATTN_CASE(32, 2) YALM_ATTN_CASE(32, 4) YALM_ATTN_CASE(32, 8)
	YALM_ATTN_CASE(16, 1) YALM_ATTN_CASE(16, 2) YALM_ATTN_CASE(16, 4) YALM_ATTN_CASE(16, 8)
#undef YALM_ATTN_CASE
	return YALM_EINVAL;
}

// ---- yalm_attn_decode with no allocation anywhere (no counterpart in the reference; added at the request of the run's
// operators for callers that cannot call cudaMalloc: CUDA graph capture, tight serving loops, harnesses that forbid it).
// The split partials live in ONE file-scope device array per GPU that loads the library (held until exit), so:
//   * shapes whose workspace exceeds kAttnStaticBytes are refused (YALM_EINVAL + a line on stderr);
//   * every call on a device shares the array: calls that overlap on the GPU (two streams, or two host threads) race;
//   * the array keeps the last call's contents; only the arrival counters must start at zero, and they are cleared on the
//     caller's stream before each launch (a memset node under capture) — the partials are fully rewritten before being read.
// In host code `g_attn_scratch` is only a stand-in for the symbol: the device address comes from cudaGetSymbolAddress, once
// per device, with that device current.
constexpr size_t kAttnStaticBytes = 2u << 20; // 2 MiB: covers every fast shape on a <= 148-SM part (see below)
constexpr int kAttnStaticMaxDevices = 64;
static __device__ __align__(256) unsigned char g_attn_scratch[kAttnStaticBytes];

static int attn_static_scratch(void **out) {
	static std::mutex mu;
	static void *ptr[kAttnStaticMaxDevices] = {};
	int dev = -1;
	YALM_TRY(cudaGetDevice(&dev));
	if (dev < 0 || dev >= kAttnStaticMaxDevices) return YALM_EINVAL;
	std::lock_guard<std::mutex> lock(mu);
	if (!ptr[dev]) {
		void *p = nullptr;
		YALM_TRY(cudaGetSymbolAddress(&p, g_attn_scratch)); // device `dev` is current: its copy of the array
		ptr[dev] = p;
	}
	*out = ptr[dev];
	return 0;
}

extern "C" size_t yalm_attn_decode_static_max_bytes(void) {
	return kAttnStaticBytes;
}

extern "C" int yalm_attn_decode_static(float *out, const uint16_t *key_cache, const uint16_t *value_cache, const float *q,
                                       int n_heads, int n_kv_heads, int head_dim, int max_seq_len, const int *ctl,
                                       yalm_stream_t s) {
	if (!out || !key_cache || !value_cache || !q || !ctl) return YALM_EINVAL;
	if (n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads || max_seq_len <= 0) return YALM_EINVAL;
	if (!attn_fast_shape(head_dim, n_heads / n_kv_heads)) return YALM_EINVAL;
	const size_t need = yalm_attn_workspace_bytes(n_heads, n_kv_heads, head_dim);
	// the counters share the first 256-byte slot of the workspace: 64 KV heads at most
	if (need > kAttnStaticBytes || (size_t)n_kv_heads * sizeof(unsigned) > 256) {
		fprintf(stderr,
		        "yalm_attn_decode_static: n_heads %d, n_kv_heads %d, head_dim %d needs %zu bytes of split-K scratch (and at most "
		        "64 KV heads); the static scratch holds %zu — use yalm_attn_decode with a caller-owned workspace\n",
		        n_heads, n_kv_heads, head_dim, need, kAttnStaticBytes);
		return YALM_EINVAL;
	}
	void *scratch = nullptr;
	if (int rc = attn_static_scratch(&scratch)) return rc;
	YALM_TRY(cudaMemsetAsync(scratch, 0, 256, (cudaStream_t)s)); // arrival counters (a failed earlier launch may have left them)
	return yalm_attn_decode(out, key_cache, value_cache, q, scratch, n_heads, n_kv_heads, head_dim, max_seq_len, ctl, s);
}

// Not in the public header's hot-path list: generic-shape attention with a materialised `att`.
extern "C" int yalm_attn_generic(float *out, float *att, const uint16_t *key_cache, const uint16_t *value_cache,
                                 const float *q, int n_heads, int n_kv_heads, int head_dim, int max_seq_len,
                                 int kv_len, const int *ctl, yalm_stream_t s) {
	if (!out || !att || !key_cache || !value_cache || !q || n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads)
		return YALM_EINVAL;
	attn_generic_kernel<<<n_heads, 256, 0, (cudaStream_t)s>>>(out, att, (const __half *)key_cache,
	                                                          (const __half *)value_cache, q, head_dim, n_heads,
	                                                          n_kv_heads, max_seq_len, kv_len, ctl);
	return (int)cudaGetLastError();
}

extern "C" int yalm_attn_is_fast_shape(int n_heads, int n_kv_heads, int head_dim) {
	return n_kv_heads > 0 && n_heads % n_kv_heads == 0 && attn_fast_shape(head_dim, n_heads / n_kv_heads);
}
