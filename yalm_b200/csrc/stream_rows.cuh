// One-row products whose weights come as a stream: y = W x for one fp32 vector x, rows of W (or of w1 and w3 side by side) dealt to one CTA per SM.
//
// Bound by the bytes of W.  A warp of its own keeps a ring of some 200 KB of shared memory full with cp.async.bulk, from the first
// cycle on, so nothing that the other warps wait for - x, the norm, a row's sum - stops the stream.  Those 16 warps share every row: warp c takes the
// 512-byte chunks c, c + C, .. of it, so its part of x stays in registers for the whole kernel (read from shared memory, x costs twice the bandwidth of fp16
// weights), and a stage is done with in one chunk's latency, whatever its size: the tail after the last byte is short.  The warps'
// partial sums of up to kCap rows meet in shared memory in a fixed order.  Launched chained: while the CTAs of the kernel before are ending, this
// one's first stages are pulled into L2 (a prefetch only: whoever writes W before this kernel is seen).
//
// Feed-forward of a token (gate and up, then down), back to back, against a persistent grid of warps that load rows into registers and start
// after x is staged: 4096 x 14336 fp16 73.7 -> 55.6 us (6.3 TB/s), fp8 48.5 -> 38.7, fp32 133.2 -> 104.6; 2752 x 7040 fp16 33.1 -> 23.7, 1024 x 2816 fp16
// 15.1 -> 8.3.  What is left over the bytes at 6.9 TB/s is some 3 us a launch (barriers, x and its norm, the first bytes' latency, the last sums), and in
// fp8 the conversions, two instructions an element.  Which products come here: streamed(), ops_gemv.cu.
#pragma once

#include "gemv.cuh"
#include "launch.h"
#include "tcgen.cuh"

namespace yalm {
namespace stream {

constexpr int kWarps = 16, kThreads = 32 * (kWarps + 1), kConsumers = 32 * kWarps;
constexpr int kRing = 212992, kMaxStages = 32, kCap = 256;                    // rows whose partial sums are held at once
constexpr int kHead = 1024;                                                   // barriers, the norm's sums
constexpr int kSmem = kHead + kRing + kWarps * kCap * 4;

struct Args {
	const char *w, *w3; // w3: the second matrix (GLU), rows of both side by side
	const float *scale, *scale3, *x, *rms_w, *residual;
	float *out;
	float eps, alpha;
	int act, n, d;                      // columns, rows (of each matrix)
	int row_bytes, piece;               // 512-byte chunks of a piece (a row is NP pieces, the last may be ragged)
	int C, RG, units, stage_bytes, stages; // warps per row, rows side by side per matrix slot, rows (or row pairs) per block
};

// Weights are read once: they go first when L2 needs room.  Copies of normal priority put everything else out (loads that do not allocate in L1 do not): a
// token of the layered models took 10 to 20 % longer, attention that found none of its keys twice as long; the products themselves 2 to 5 % longer.
__device__ __forceinline__ uint64_t read_once() {
	uint64_t p;
	asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
	return p;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar, uint64_t policy) {
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy)
	             : "memory");
}
__device__ __forceinline__ void bulk_prefetch(const void *src, uint32_t bytes, uint64_t policy) {
	asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;" ::"l"(src), "r"(bytes), "l"(policy) : "memory");
}
__device__ __forceinline__ void consumer_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory"); }
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
	uint64_t r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
	return r;
}
__device__ __forceinline__ uint64_t fma2(float2 a, float lo, float hi, uint64_t c) {
	uint64_t r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pair_of(a.x, a.y)), "l"(pair_of(lo, hi)), "l"(c));
	return r;
}
__device__ __forceinline__ float halves(uint64_t v) {
	float lo, hi;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
	return lo + hi;
}
// acc += 16 bytes of weights times their x, even elements in the lower half and odd ones in the upper
template <int DT>
__device__ __forceinline__ uint64_t dot16(uint4 w, const float4 (&x)[WTraits<DT>::EP / 4], uint64_t acc) {
	const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
	if constexpr (DT == YALM_F32) {
		acc = fma2(make_float2(__uint_as_float(w.x), __uint_as_float(w.y)), x[0].x, x[0].y, acc);
		acc = fma2(make_float2(__uint_as_float(w.z), __uint_as_float(w.w)), x[0].z, x[0].w, acc);
	} else if constexpr (DT == YALM_F8E4M3) {
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			acc = fma2(WTraits<DT>::e2((uint16_t)(ww[i] & 0xffffu)), x[i].x, x[i].y, acc);
			acc = fma2(WTraits<DT>::e2((uint16_t)(ww[i] >> 16)), x[i].z, x[i].w, acc);
		}
	} else {
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			float2 v;
			if constexpr (DT == YALM_BF16) v = make_float2(WTraits<DT>::lo(ww[i]), WTraits<DT>::hi(ww[i]));
			else v = WTraits<DT>::h2(ww[i]);
			acc = i & 1 ? fma2(v, x[i >> 1].z, x[i >> 1].w, acc) : fma2(v, x[i >> 1].x, x[i >> 1].y, acc);
		}
	}
	return acc;
}

// V sums over a warp at once: each exchange halves the values a lane carries.  Lane l ends with sum l / (32 / V).
template <int V>
__device__ __forceinline__ float sums_of(float (&y)[V], int lane) {
	int n = V;
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		if (n == 1) {
			y[0] += __shfl_xor_sync(kFull, y[0], o);
			continue;
		}
		n /= 2;
		const bool up = lane & o;
#pragma unroll
		for (int i = 0; i < V / 2; ++i)
			if (i < n) y[i] = (up ? y[i + n] : y[i]) + __shfl_xor_sync(kFull, up ? y[i] : y[i + n], o);
	}
	return y[0];
}

// A block is what the warps finish together: NP == 1 and JJ == 1 (rows of up to 8 KB): 2 RG rows (GLU: RG rows of each matrix) in one stage, two of them a
// warp; longer rows: one row, NP stages of JJ chunks a warp (GLU: row i of w1, then of w3).  Its rows past the CTA's last are not copied and not used.
template <int DT, int NP, int JJ, bool GLU>
__global__ void __launch_bounds__(kThreads, 1) stream_rows_kernel(const __grid_constant__ Args a) {
	extern __shared__ __align__(128) uint8_t smem_raw[];
	constexpr int EP = WTraits<DT>::EP, CH = 32 * EP, Q = EP / 4;
	constexpr bool PAIR = NP == 1 && JJ == 1;
	constexpr float NaN = __builtin_nanf("");
	const uint32_t base = s32(smem_raw), full0 = base, empty0 = base + 8 * kMaxStages, ring0 = base + kHead;
	float *red = reinterpret_cast<float *>(smem_raw + 16 * kMaxStages), *part = reinterpret_cast<float *>(smem_raw + kHead + kRing);
	const int warp = uniform_warp(), lane = threadIdx.x & 31;
	const int r0 = (int)((long)blockIdx.x * a.d / gridDim.x), r1 = (int)((long)(blockIdx.x + 1) * a.d / gridDim.x);
	const int rows = r1 - r0, blocks = PAIR ? (rows + a.units - 1) / a.units : GLU ? 2 * rows : rows;
	const int rows_block = PAIR ? 2 * a.RG : 1; // rows of partial sums
	bool dead = false;

	if (threadIdx.x == 0) {
		for (int i = 0; i < a.stages; ++i) mbar_init(full0 + 8 * i, 1), mbar_init(empty0 + 8 * i, a.C * a.RG);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	// stage st of this CTA: its one or two ranges of global memory
	auto ranges = [&](int st, const char *(&src)[2], uint32_t &bytes) {
		if (PAIR) {
			const size_t at = (size_t)(r0 + st * a.units) * a.row_bytes;
			bytes = (uint32_t)(min(a.units, rows - st * a.units) * a.row_bytes);
			src[0] = a.w + at, src[1] = GLU ? a.w3 + at : nullptr;
		} else {
			const int b = st / NP, p = st - b * NP;
			const uint32_t off = (uint32_t)(p * a.piece) * 512u;
			src[0] = (GLU && (b & 1) ? a.w3 : a.w) + (size_t)(r0 + (GLU ? b >> 1 : b)) * a.row_bytes + off, src[1] = nullptr;
			bytes = min((uint32_t)a.piece * 512u, (uint32_t)a.row_bytes - off);
		}
	};
	const int total = blocks * NP;
	const uint64_t policy = read_once();
	if (warp == kWarps) {
		const char *src[2];
		uint32_t bytes;
		if (lane < min(a.stages, total)) {
			ranges(lane, src, bytes);
			bulk_prefetch(src[0], bytes, policy);
			if (GLU && PAIR) bulk_prefetch(src[1], bytes, policy);
		}
		__syncwarp();
	}
	__syncthreads();
	chain_wait();
	chain_next();

	if (warp == kWarps) { // ---- the stream ----
		Ring ring;
		ring.phase = 1; // the first round of every stage is free
		for (int st = 0; st < total; ++st, ring.next(a.stages)) {
			mbar_wait_warp(empty0 + 8 * ring.s, ring.phase, dead);
			if (dead) break;
			const char *src[2];
			uint32_t bytes;
			ranges(st, src, bytes);
			const uint32_t dst = ring0 + ring.s * a.stage_bytes, bar = full0 + 8 * ring.s;
			if (elect_one()) {
				mbar_expect_tx(bar, GLU && PAIR ? 2 * bytes : bytes);
				bulk_load(dst, src[0], bytes, bar, policy);
				if (GLU && PAIR) bulk_load(dst + a.RG * a.row_bytes, src[1], bytes, bar, policy);
			}
			__syncwarp();
		}
		// its own copies have landed before it leaves (the parity that a stage's last one completes is that of the round in which it would be free)
		bool late = false;
		for (int i = 0; i < a.stages; ++i, ring.next(a.stages)) mbar_wait_warp(full0 + 8 * ring.s, ring.phase, late);
		return;
	}

	// ---- this warp's chunks of x, normalised ----
	const int c = warp % a.C, rg = warp / a.C;
	const bool active = rg < a.RG;
	float4 x[NP * JJ][Q];
	bool ok[NP * JJ]; // this lane has a piece of the chunk
	float ss = 0.f;
#pragma unroll
	for (int j = 0; j < NP * JJ; ++j) {
		const int in = (j % JJ) * a.C + c, chunk = j / JJ * a.piece + in, e = chunk * CH + lane * EP;
		ok[j] = active && in < a.piece && e < a.n;
#pragma unroll
		for (int q = 0; q < Q; ++q) {
			x[j][q] = make_float4(0.f, 0.f, 0.f, 0.f);
			if (ok[j]) x[j][q] = *reinterpret_cast<const float4 *>(a.x + e + 4 * q);
			if (rg == 0) ss += x[j][q].x * x[j][q].x + x[j][q].y * x[j][q].y + x[j][q].z * x[j][q].z + x[j][q].w * x[j][q].w;
		}
	}
	if (a.rms_w) { // o = x * (1 / sqrt(mean + eps)) * w (src/infer.cpp:134-144)
		constexpr bool EARLY = NP * JJ * EP <= 32; // the norm's weights beside x in registers, loaded before the sum is known
		auto norm_weight = [&](int j, int q) {
			return ok[j] ? *reinterpret_cast<const float4 *>(a.rms_w + (j / JJ * a.piece + (j % JJ) * a.C + c) * CH + lane * EP + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
		};
		float4 nw[EARLY ? NP * JJ : 1][Q];
		if constexpr (EARLY) {
#pragma unroll
			for (int j = 0; j < NP * JJ; ++j)
#pragma unroll
				for (int q = 0; q < Q; ++q) nw[j][q] = norm_weight(j, q);
		}
		ss = warp_sum(ss);
		if (lane == 0) red[warp] = ss;
		consumer_barrier();
		float t = 0.f;
#pragma unroll
		for (int w = 0; w < kWarps; ++w) t += red[w];
		const float f = 1.0f / sqrtf(t / a.n + a.eps);
#pragma unroll
		for (int j = 0; j < NP * JJ; ++j)
#pragma unroll
			for (int q = 0; q < Q; ++q) {
				const float4 g = EARLY ? nw[EARLY ? j : 0][q] : norm_weight(j, q);
				x[j][q] = make_float4(x[j][q].x * f * g.x, x[j][q].y * f * g.y, x[j][q].z * f * g.z, x[j][q].w * f * g.w);
			}
	}

	constexpr int R = PAIR ? 2 : 1, V = PAIR ? 2 : JJ, G = NP == 1 ? 4 : 2; // rows and 16-byte loads of a lane and block, blocks at once
	Ring ring;
	// this lane's weights of the next stage, which is piece p of its row
	auto stage = [&](uint4 (&w)[V], int p) {
		mbar_wait_warp(full0 + 8 * ring.s, ring.phase, dead);
		const uint32_t at = ring0 + ring.s * a.stage_bytes + rg * a.row_bytes + c * 512 + lane * 16;
#pragma unroll
		for (int j = 0; j < V; ++j) {
			w[j] = make_uint4(0, 0, 0, 0);
			if (ok[PAIR ? 0 : p * JJ + j])
				asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[j].x), "=r"(w[j].y), "=r"(w[j].z), "=r"(w[j].w) : "r"(at + j * (PAIR ? a.RG * a.row_bytes : a.C * 512)) : "memory");
		}
		__syncwarp();
		if (lane == 0 && !dead) mbar_arrive(empty0 + 8 * ring.s); // (else it could be filled again under a copy that may still be on its way)
		ring.next(a.stages);
	};
	const int per = kCap / rows_block; // blocks whose partial sums fit
	for (int b0 = 0; b0 < blocks; b0 += per) {
		const int b1 = min(blocks, b0 + per);
		// rows of W (or row pairs) that these blocks finish
		const int first = PAIR ? b0 * a.units : GLU ? b0 >> 1 : b0, count = (PAIR ? min(rows, b1 * a.units) : GLU ? b1 >> 1 : b1) - first;
		float resid = 0.f;
		if (!GLU && a.residual && (int)threadIdx.x < count) resid = a.residual[r0 + first + threadIdx.x];
		if (active)
			for (int b = b0; b < b1; b += G) {
				// all loads of G blocks, then their products, then one reduction: block by block the shuffles' latency bounded a stage
				float y[G * R];
				if constexpr (NP == 1) {
					uint4 w[G][V];
#pragma unroll
					for (int u = 0; u < G; ++u) {
#pragma unroll
						for (int j = 0; j < V; ++j) w[u][j] = make_uint4(0, 0, 0, 0);
						if (b + u < b1) stage(w[u], 0);
					}
#pragma unroll
					for (int u = 0; u < G; ++u) {
						if constexpr (PAIR) {
							y[2 * u] = halves(dot16<DT>(w[u][0], x[0], 0ull)), y[2 * u + 1] = halves(dot16<DT>(w[u][1], x[0], 0ull));
						} else {
							y[u] = 0.f;
#pragma unroll
							for (int j = 0; j < JJ; ++j) y[u] += halves(dot16<DT>(w[u][j], x[j], 0ull));
						}
					}
				} else {
#pragma unroll
					for (int u = 0; u < G; ++u) {
						uint64_t acc[JJ] = {};
						if (b + u < b1) {
#pragma unroll
							for (int p = 0; p < NP; ++p) {
								uint4 w[V];
								stage(w, p);
#pragma unroll
								for (int j = 0; j < JJ; ++j) acc[j] = dot16<DT>(w[j], x[p * JJ + j], acc[j]);
							}
						}
						y[u] = 0.f;
#pragma unroll
						for (int j = 0; j < JJ; ++j) y[u] += halves(acc[j]);
					}
				}
				const float v = sums_of<G * R>(y, lane);
				constexpr int LANES = 32 / (G * R); // lanes that hold the same sum
				const int k = lane / LANES, u = k / R;
				if (lane % LANES == 0 && b + u < b1) part[c * kCap + (b + u - b0) * rows_block + rg + (k % R) * a.RG] = dead ? NaN : v;
			}
		consumer_barrier();
		// a thread per row: the warps' sums in order, then what the product is for
		const int i = threadIdx.x;
		if (i < count) {
			const int row = r0 + first + i;
			auto sum = [&](int at) {
				float t = 0.f;
				for (int k = 0; k < a.C; ++k) t += part[k * kCap + at];
				return t;
			};
			if constexpr (GLU) {
				const int at = PAIR ? i / a.RG * 2 * a.RG + i % a.RG : 2 * i;
				float g = sum(at), u = sum(PAIR ? at + a.RG : at + 1);
				if (DT == YALM_F8E4M3 && a.scale) g *= a.scale[row], u *= a.scale3[row];
				a.out[row] = (a.act == YALM_ACT_GELU ? act_gelu(g) : act_silu(g)) * u;
			} else {
				float v = sum(i);
				if (DT == YALM_F8E4M3 && a.scale) v *= a.scale[row];
				a.out[row] = a.residual ? resid + v : a.alpha * v;
			}
		}
		if (b1 < blocks) consumer_barrier();
	}
}

template <int DT, int NP, int JJ, bool GLU>
static int launch_as(const Args &a, cudaStream_t st) {
	auto kernel = stream_rows_kernel<DT, NP, JJ, GLU>;
	YALM_TRY(allow_smem((const void *)kernel, kSmem));
	return launch_chained(kernel, dim3(std::min(device_info().sms, a.d)), dim3(kThreads), kSmem, st, 1, a);
}
// Longest row whose part of x fits the 96 registers that 17 warps (five on one scheduler) leave a thread; longer ones take the kernels of ops_gemv.cu.
constexpr int longest(int bytes_per_element) { return (bytes_per_element == 1 ? 2 : 4) * 32 * 512 / bytes_per_element; }

// a: all but the geometry, a.n <= longest().
template <int DT, bool GLU>
static int launch(Args &a, cudaStream_t st) {
	a.row_bytes = a.n * WTraits<DT>::BYTES;
	const int chunks = (a.row_bytes + 511) / 512, pieces = (chunks + 31) / 32, NP = pieces <= 2 ? pieces : 4;
	a.piece = (chunks + NP - 1) / NP;
	const int JJ = a.piece > 16 || NP > 1 ? 2 : 1;
	a.C = (a.piece + JJ - 1) / JJ;
	a.RG = NP == 1 && JJ == 1 ? kWarps / a.C : 1, a.units = GLU ? a.RG : 2 * a.RG;
	a.stage_bytes = ((NP == 1 && JJ == 1 ? 2 * a.RG * a.row_bytes : a.piece * 512) + 511) / 512 * 512;
	a.stages = std::min(kMaxStages, kRing / a.stage_bytes);
	switch (NP * 2 + JJ) {
	case 3: return launch_as<DT, 1, 1, GLU>(a, st);
	case 4: return launch_as<DT, 1, 2, GLU>(a, st);
	case 6: return launch_as<DT, 2, 2, GLU>(a, st);
	}
	if constexpr (DT != YALM_F8E4M3) return launch_as<DT, 4, 2, GLU>(a, st);
	return YALM_EINVAL;
}

} // namespace stream
} // namespace yalm
