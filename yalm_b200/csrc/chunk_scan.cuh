// The recurrence over a matrix state (ops_stack_state.cu: state_scan_kernel) for many positions, 8 at a time.
//
// One position after the other, a step is a chain - decay, M^T k, three or four exchanges, update - that takes some 400 cycles however little
// arithmetic it has.  Inside a chunk of 8 positions the same values follow from the state at its start:
//   with b_t = g_1 .. g_t (products of the decays, per channel) and M_0 the state before the chunk,
//   r_t = v_t - (b_t k_t)^T M_0,   u = T r,   y_t = (b_t q_t)^T M_0 + sum_i (B T)_ti r_i (+ skip v_t),   M_8 = b_8 M_0 + sum_i (g_{i+1} .. g_8 k_i) u_i^T
//   A_ti = k_t . (g_{i+1} .. g_t k_i) (i < t),   B_ti = q_t . (g_{i+1} .. g_t k_i) (i <= t),   T = (1 + diag(beta) A)^-1 diag(beta)
// (without the delta correction r = v and T = diag(vscale)).  Every decay enters as a product of decays, never as a quotient, so a
// decay may be 0.  All of it is fp32; what differs from the position-by-position form is the order of sums.
//
// A CTA owns 16 or 8 columns of one head.  Eight warps prepare chunks in turn - everything that the columns share: b k, b q, the update rows, T and
// B T, and the chunk's v - into a ring of shared-memory slots; four warps own NC = 4 or 2 columns each, a lane 4 (D = 128) or 2 (D = 64) rows of all of them: a
// vector of a chunk is read once for NC columns (at one column per thread the shared-memory reads were the limit), the 8 NC partial
// products meet over the 32 lanes by halving exchanges, which leave lane (t, c) with the sums of position t and column c.
// The packed fp32 instructions carry two rows each.
// Bound by the column warps, one per scheduler: of about 1550 cycles a chunk with 4 columns 600 go to the products with M_0 (shared-memory reads of four
// wavefronts each), 620 to the exchanges and T, 320 to the update.  (2 columns x 8 rows a lane, or eight warps of two columns in a CTA of 16, which
// leaves registers for four warps that prepare: no faster, 60 and 64 us for 57.)
// 512 rows, delta rule with a decay per channel: 16 heads of 128 x 128 57 -> 55 us (eight warps that prepare instead of six); 8 heads, in CTAs of 8 columns,
// 57 -> 44 us; 16 heads of 64 x 64 44 -> 34 us; without the correction 43 -> 42, 43 -> 35, 34 -> 28 us.
#pragma once

#include "tcgen.cuh"

namespace yalm {
namespace stack {

constexpr int kChunk = 8, kChunkCols = 16, kChunkSlots = 8, kPrepWarps = 8, kChunkThreads = 32 * (4 + kPrepWarps); // (kChunkCols: the most a CTA owns)

template <int D>
struct ChunkSlot { // float offsets
	static constexpr int K = 0, Q = kChunk * D, U = 2 * kChunk * D, B8 = 3 * kChunk * D, T = B8 + D, BT = T + 64, V = BT + 64, M = V + kChunk * kChunkCols, SIZE = M + 64;
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk(float lo, float hi) {
	f32x2 r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
	return r;
}
__device__ __forceinline__ float sum2(f32x2 v) {
	float lo, hi;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
	return lo + hi;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
	f32x2 r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
	f32x2 r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
	return r;
}
// N = 1 or 2 pairs of neighbouring floats
template <int N>
__device__ __forceinline__ void load_pairs(f32x2 (&r)[N], const float *p) {
	if constexpr (N == 2) {
		const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
		r[0] = v.x, r[1] = v.y;
	} else
		r[0] = *reinterpret_cast<const f32x2 *>(p);
}
template <int N>
__device__ __forceinline__ void store_pairs(float *p, const f32x2 (&r)[N]) {
	if constexpr (N == 2) *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(r[0], r[1]);
	else *reinterpret_cast<f32x2 *>(p) = r[0];
}
// N values over the 32 lanes: afterwards v[0 .. N / 32 - 1] of lane l are the sums of values l N / 32 + ..
template <int N>
__device__ __forceinline__ void exchange_sum(float (&v)[N]) {
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int o = 16, n = N / 2; o > 0; o >>= 1, n >>= 1)
#pragma unroll
		for (int i = 0; i < n; ++i) {
			const float give = (lane & o) ? v[i] : v[i + n], keep = (lane & o) ? v[i + n] : v[i];
			v[i] = keep + __shfl_xor_sync(kFull, give, o);
		}
}

// 8 NC values [position][NC] of which slot i holds position (i / NC) ^ (lane / 4): the lanes agree on who keeps what without a select (a lane always
// keeps the lower slots), but for the exchanges over the columns.  Afterwards v[0] is the sum of (position lane / 4, column lane % 4 NC / 4).
template <int NC>
__device__ __forceinline__ void exchange_chunk(float (&v)[8 * NC]) {
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int o = 16, n = 4 * NC; o >= 4; o >>= 1, n >>= 1)
#pragma unroll
		for (int i = 0; i < n; ++i) v[i] += __shfl_xor_sync(kFull, v[i + n], o);
#pragma unroll
	for (int o = 2, n = NC / 2; o > 0; o >>= 1, n >>= 1) {
#pragma unroll
		for (int i = 0; i < n; ++i) {
			const float give = (lane & o) ? v[i] : v[i + n], keep = (lane & o) ? v[i + n] : v[i];
			v[i] = keep + __shfl_xor_sync(kFull, give, o);
		}
		if (n == 0) v[0] += __shfl_xor_sync(kFull, v[0], o); // two lanes for a column
	}
}

// NC: columns of a warp
template <int D, int NC, bool DELTA, bool PER_CHANNEL>
__global__ void __launch_bounds__(kChunkThreads, 1) chunk_scan_kernel(const ScanArgs a) {
	using SL = ChunkSlot<D>;
	constexpr int NP = D / 64; // pairs of rows per lane
	extern __shared__ __align__(16) float chunk_sm[];
	__shared__ __align__(8) unsigned long long bars[2 * kChunkSlots];
	const int warp = uniform_warp(), lane = threadIdx.x & 31;
	const int h = blockIdx.y, kh = h / a.rep, c0 = blockIdx.x * 4 * NC, nchunks = (a.n + kChunk - 1) / kChunk;
	const int col_warps = min(4, (a.P - c0) / NC); // (P is a multiple of 4)
	const uint32_t full0 = s32(bars), empty0 = full0 + 8 * kChunkSlots;
	bool dead = false;
	if (threadIdx.x == 0)
		for (int i = 0; i < kChunkSlots; ++i) mbar_init(full0 + 8 * i, 1), mbar_init(empty0 + 8 * i, col_warps);
	__syncthreads();
	chain_wait();
	chain_next();

	if (warp >= 4) { // ---- prepare chunks warp - 4, warp - 4 + kPrepWarps, .. ; a lane holds rows lane D / 32 .. of every vector ----
		const int e0 = lane * 2 * NP;
		for (int ch = warp - 4; ch < nchunks; ch += kPrepWarps) {
			const int t0 = ch * kChunk, slot = ch % kChunkSlots, round = ch / kChunkSlots;
			f32x2 k[kChunk][NP], q[kChunk][NP], g[kChunk][NP];
#pragma unroll
			for (int t = 0; t < kChunk; ++t) {
				if (t0 + t < a.n) {
					load_pairs<NP>(k[t], a.k + (size_t)(t0 + t) * a.ldk + kh * D + e0);
					load_pairs<NP>(q[t], a.q + (size_t)(t0 + t) * a.ldq + kh * D + e0);
					if constexpr (PER_CHANNEL) {
						load_pairs<NP>(g[t], a.decay + (size_t)(t0 + t) * a.ldd + h * D + e0);
					} else {
						const float d = a.decay[(size_t)(t0 + t) * a.ldd + h];
#pragma unroll
						for (int p = 0; p < NP; ++p) g[t][p] = pk(d, d);
					}
				} else { // past the last position: nothing changes
#pragma unroll
					for (int p = 0; p < NP; ++p) k[t][p] = q[t][p] = 0, g[t][p] = pk(1.f, 1.f);
				}
			}
			float factor = 0.f; // lane t < 8: beta or vscale of position t
			if (lane < kChunk && t0 + lane < a.n)
				factor = DELTA ? a.beta[(size_t)(t0 + lane) * a.ldb + h] : a.vscale ? a.vscale[(size_t)(t0 + lane) * a.ldvs + h] : 1.f;
			float4 v = make_float4(0.f, 0.f, 0.f, 0.f); // position lane / 4, columns 4 (lane % 4) ..
			{
				const int t = t0 + (lane >> 2), c = c0 + (lane & 3) * 4;
				if (t < a.n && c < a.P && (lane & 3) < NC) {
					const float *src = a.v + (size_t)t * a.ldv + (size_t)h * a.P + c;
					v = make_float4(src[0], src[1], src[2], src[3]);
				}
			}
			if (round > 0) {
				mbar_wait_warp(empty0 + 8 * slot, (uint32_t)(round - 1) & 1u, dead);
				if (dead) break;
			}
			float *sm = chunk_sm + slot * SL::SIZE;
			*reinterpret_cast<float4 *>(sm + SL::V + lane * 4) = v;
			{
				f32x2 b[NP], w[NP], x[NP];
#pragma unroll
				for (int t = 0; t < kChunk; ++t) {
#pragma unroll
					for (int p = 0; p < NP; ++p) b[p] = t ? mul2(b[p], g[t][p]) : g[t][p];
					if constexpr (DELTA) {
#pragma unroll
						for (int p = 0; p < NP; ++p) x[p] = mul2(b[p], k[t][p]);
						store_pairs<NP>(sm + SL::K + t * D + e0, x);
					}
#pragma unroll
					for (int p = 0; p < NP; ++p) x[p] = mul2(b[p], q[t][p]);
					store_pairs<NP>(sm + SL::Q + t * D + e0, x);
				}
				store_pairs<NP>(sm + SL::B8 + e0, b);
#pragma unroll
				for (int t = kChunk - 1; t >= 0; --t) {
#pragma unroll
					for (int p = 0; p < NP; ++p) x[p] = t == kChunk - 1 ? k[t][p] : mul2(w[p], k[t][p]);
					store_pairs<NP>(sm + SL::U + t * D + e0, x);
#pragma unroll
					for (int p = 0; p < NP; ++p) w[p] = t == kChunk - 1 ? g[t][p] : mul2(w[p], g[t][p]);
				}
			}
			float pr[64]; // [t][i], i <= t: B_ti; [i][t], i < t: A_ti
#pragma unroll
			for (int i = 0; i < kChunk; ++i) {
				f32x2 w[NP];
#pragma unroll
				for (int p = 0; p < NP; ++p) w[p] = k[i][p];
#pragma unroll
				for (int t = i; t < kChunk; ++t) {
					f32x2 sb = 0, sa = 0;
#pragma unroll
					for (int p = 0; p < NP; ++p) {
						if (t > i) w[p] = mul2(w[p], g[t][p]);
						sb = p ? fma2(q[t][p], w[p], sb) : mul2(q[t][p], w[p]);
						if (DELTA && t > i) sa = p ? fma2(k[t][p], w[p], sa) : mul2(k[t][p], w[p]);
					}
					pr[t * 8 + i] = sum2(sb);
					if (t > i) pr[i * 8 + t] = DELTA ? sum2(sa) : 0.f;
				}
			}
			exchange_sum(pr);
			float *M = sm + SL::M;
			*reinterpret_cast<float2 *>(M + 2 * lane) = make_float2(pr[0], pr[1]);
			__syncwarp();
			float f[kChunk];
#pragma unroll
			for (int t = 0; t < kChunk; ++t) f[t] = __shfl_sync(kFull, factor, t);
			if (lane < kChunk) { // column `lane` of T, then of B T
				float x[kChunk];
#pragma unroll
				for (int t = 0; t < kChunk; ++t) {
					float s = t == lane ? 1.f : 0.f;
					if constexpr (DELTA)
#pragma unroll
						for (int i = 0; i < t; ++i) s = fmaf(-M[i * 8 + t], x[i], s);
					x[t] = f[t] * s;
					sm[SL::T + t * 8 + lane] = x[t];
				}
#pragma unroll
				for (int t = 0; t < kChunk; ++t) {
					float s = 0.f;
#pragma unroll
					for (int i = 0; i <= t; ++i) s = fmaf(M[t * 8 + i], x[i], s);
					sm[SL::BT + t * 8 + lane] = s;
				}
			}
			__syncwarp();
			if (lane == 0) mbar_arrive(full0 + 8 * slot);
		}
	} else if (warp < col_warps) { // ---- columns c0 + NC warp .. ; a lane's rows lane D / 32 .. ----
		__shared__ __align__(16) float2 u_sm[4][kChunk][NC]; // u, twice
		const int e0 = lane * 2 * NP, cw = c0 + NC * warp, t = lane >> 2, c = (lane & 3) * NC / 4;
		const bool fresh = first_pos(a.ctl, a.pos0) == 0;
		float *state = a.state + ((size_t)h * a.P + cw) * D + e0;
		f32x2 s[NC][NP];
#pragma unroll
		for (int j = 0; j < NC; ++j) {
			if (fresh) {
#pragma unroll
				for (int p = 0; p < NP; ++p) s[j][p] = 0;
			} else
				load_pairs<NP>(s[j], state + (size_t)j * D);
		}
		const float skip = a.skip ? a.skip[h] : 0.f;
		for (int ch = 0; ch < nchunks; ++ch) {
			const int slot = ch % kChunkSlots;
			mbar_wait_warp(full0 + 8 * slot, (uint32_t)(ch / kChunkSlots) & 1u, dead);
			const float *sm = chunk_sm + slot * SL::SIZE;
			float W[DELTA ? 8 * NC : 1], O[8 * NC];
#pragma unroll
			for (int tt = 0; tt < kChunk; ++tt) {
				f32x2 x[NP];
				if constexpr (DELTA) {
					load_pairs<NP>(x, sm + SL::K + (tt ^ t) * D + e0);
#pragma unroll
					for (int j = 0; j < NC; ++j) {
						f32x2 d = mul2(x[0], s[j][0]);
						if (NP == 2) d = fma2(x[NP - 1], s[j][NP - 1], d);
						W[tt * NC + j] = sum2(d);
					}
				}
				load_pairs<NP>(x, sm + SL::Q + (tt ^ t) * D + e0);
#pragma unroll
				for (int j = 0; j < NC; ++j) {
					f32x2 d = mul2(x[0], s[j][0]);
					if (NP == 2) d = fma2(x[NP - 1], s[j][NP - 1], d);
					O[tt * NC + j] = sum2(d);
				}
			}
			const float v = sm[SL::V + t * kChunkCols + warp * NC + c];
			float r = v;
			if constexpr (DELTA) {
				exchange_chunk<NC>(W);
				r = v - W[0];
			}
			exchange_chunk<NC>(O);
			float u = 0.f, y = O[0];
			float Tr[8], Br[8];
			*reinterpret_cast<float4 *>(Tr) = *reinterpret_cast<const float4 *>(sm + SL::T + t * 8), *reinterpret_cast<float4 *>(Tr + 4) = *reinterpret_cast<const float4 *>(sm + SL::T + t * 8 + 4);
			*reinterpret_cast<float4 *>(Br) = *reinterpret_cast<const float4 *>(sm + SL::BT + t * 8), *reinterpret_cast<float4 *>(Br + 4) = *reinterpret_cast<const float4 *>(sm + SL::BT + t * 8 + 4);
#pragma unroll
			for (int i = 0; i < kChunk; ++i) { // (both matrices are lower triangular, zeros included)
				const float ri = __shfl_sync(kFull, r, i * 4 + c * (4 / NC));
				if (i <= t) u = fmaf(Tr[i], ri, u), y = fmaf(Br[i], ri, y);
			}
			u_sm[warp][t][c] = make_float2(u, u); // (NC 2: two lanes, the same)
			const int pos = ch * kChunk + t;
			if (pos < a.n && (NC == 4 || !(lane & 1))) a.out[(size_t)pos * a.ldo + (size_t)h * a.P + cw + c] = dead ? __int_as_float(0x7fc00000) : fmaf(skip, v, y);
			__syncwarp();
			{
				f32x2 b[NP];
				load_pairs<NP>(b, sm + SL::B8 + e0);
#pragma unroll
				for (int j = 0; j < NC; ++j)
#pragma unroll
					for (int p = 0; p < NP; ++p) s[j][p] = mul2(s[j][p], b[p]);
#pragma unroll
				for (int i = 0; i < kChunk; ++i) {
					f32x2 x[NP], u2[NC];
					load_pairs<NP>(x, sm + SL::U + i * D + e0);
#pragma unroll
					for (int j = 0; j < NC; j += 2) {
						f32x2 two[2];
						load_pairs<2>(two, &u_sm[warp][i][j].x);
						u2[j] = two[0], u2[j + 1] = two[1];
					}
#pragma unroll
					for (int p = 0; p < NP; ++p)
#pragma unroll
						for (int j = 0; j < NC; ++j) s[j][p] = fma2(x[p], u2[j], s[j][p]);
				}
			}
			__syncwarp();
			if (lane == 0) mbar_arrive(empty0 + 8 * slot);
		}
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			if (j >= NC) break;
			if (dead)
#pragma unroll
				for (int p = 0; p < NP; ++p) s[j % NC][p] = pk(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
			store_pairs<NP>(state + (size_t)j * D, s[j % NC]);
		}
	}
}

} // namespace stack
} // namespace yalm
