// Batched prefill / perplexity: n consecutive positions through the whole model in one pass.
// The reference walks a prompt token by token (src/main.cpp:91-97, 174-184); here the projections of a chunk are dense
// GEMMs on the tcgen05 tensor cores (prefill_gemm.cu), attention is a causal flash-attention over the head-major KV ring
// (prompt_attn.cu, online softmax in fp32), and the KV rows of the whole chunk are appended at once.
// Arithmetic definitions are the decode path's (rmsnorm association order, interleaved-pair RoPE with accurate
// powf/cosf/sinf, clip, gelu/silu, fp16 KV rows); what differs is the summation order inside the GEMMs and that the GEMM
// inputs (normalised x, q, attention output, GLU output) are rounded to fp16 once.  Oracle: the token loop.
#include "yalm_api.h"

#include "gemv.cuh"
#include "launch.h"
#include "mega.h"
#include "prefill.h"

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstdio>

extern "C" int yalm_gemm_f16(float *c, int ldc, const void *a, const void *w, int M, int N, int K, int accumulate, yalm_stream_t s);
extern "C" int yalm_gemm_glu_f16(void *h, int ldh, const void *a, const void *w1, const void *w3, int M, int N, int K, int act,
                                 yalm_stream_t s);

namespace yalm {
namespace prompt { // prompt_attn.cu
int causal_f16(void *out, const void *q, const void *keys, const void *values, int n, int pos0, int n_heads, int n_kv, int head_dim, int max_seq_len,
               cudaStream_t st);
}

namespace prefill {

// (cosine, sine) of every position of the portion and pair of a head's channels: the same for all layers
__global__ void turns_kernel(float2 *turns, int n, int head_dim, int rotary_dim, int pos0, float theta) {
	const int half = head_dim / 2, j = threadIdx.x % half, i = blockIdx.x * (blockDim.x / half) + threadIdx.x / half;
	float fcr, fci;
	rope_angle(fcr, fci, 2 * j, pos0 + i, theta, rotary_dim);
	chain_wait();
	chain_next();
	if (i < n) turns[(size_t)i * half + j] = make_float2(fcr, fci);
}

// x[i, :] = float(E[tokens[i], :])   (src/infer.cu:632-640, for a batch of rows)
__global__ void embed_rows_kernel(float *__restrict__ x, const __half *__restrict__ table, const int *__restrict__ tokens, int dim) {
	const __half *row = table + (size_t)tokens[blockIdx.x] * dim;
	float *dst = x + (size_t)blockIdx.x * dim;
	for (int e = threadIdx.x * 2; e < dim; e += blockDim.x * 2) {
		const float2 v = __half22float2(*reinterpret_cast<const __half2 *>(row + e));
		*reinterpret_cast<float2 *>(dst + e) = v;
	}
}

// out16[i, :] = half(x[i, :] * (1 / sqrt(mean(x^2) + eps)) * w)   (src/infer.cpp:134-144, one CTA per row)
// Rows of up to 8192 stay in registers between the sum and the scaling, all their loads in flight at once (512 rows of 4096: 6.7 -> 5.6 us).
constexpr int kNormThreads = 256, kNormKept = 8;
__global__ void __launch_bounds__(kNormThreads) rmsnorm_rows_kernel(__half *out, const float *x, const float *w, int dim, float eps) {
	__shared__ float red[33];
	chain_wait();
	chain_next();
	const float *row = x + (size_t)blockIdx.x * dim;
	const bool kept = dim <= kNormThreads * 4 * kNormKept;
	float4 v[kNormKept], gain[kNormKept];
	float ss = 0.f;
	if (kept) {
#pragma unroll
		for (int j = 0; j < kNormKept; ++j) {
			const int e = (threadIdx.x + j * kNormThreads) * 4;
			v[j] = e < dim ? *reinterpret_cast<const float4 *>(row + e) : make_float4(0.f, 0.f, 0.f, 0.f);
			if (e < dim) gain[j] = *reinterpret_cast<const float4 *>(w + e);
		}
#pragma unroll
		for (int j = 0; j < kNormKept; ++j) ss += v[j].x * v[j].x + v[j].y * v[j].y + v[j].z * v[j].z + v[j].w * v[j].w;
	} else
		for (int e = threadIdx.x * 4; e < dim; e += kNormThreads * 4) {
			const float4 t = *reinterpret_cast<const float4 *>(row + e);
			ss += t.x * t.x + t.y * t.y + t.z * t.z + t.w * t.w;
		}
	ss = block_sum(ss, red);
	const float scale = 1.0f / sqrtf(ss / dim + eps);
	__half *dst = out + (size_t)blockIdx.x * dim;
	auto put = [&](int e, float4 t, float4 g) {
		*reinterpret_cast<__half2 *>(dst + e) = __floats2half2_rn(t.x * scale * g.x, t.y * scale * g.y);
		*reinterpret_cast<__half2 *>(dst + e + 2) = __floats2half2_rn(t.z * scale * g.z, t.w * scale * g.w);
	};
	if (kept) {
#pragma unroll
		for (int j = 0; j < kNormKept; ++j) {
			const int e = (threadIdx.x + j * kNormThreads) * 4;
			if (e < dim) put(e, v[j], gain[j]);
		}
	} else
		for (int e = threadIdx.x * 4; e < dim; e += kNormThreads * 4) put(e, *reinterpret_cast<const float4 *>(row + e), *reinterpret_cast<const float4 *>(w + e));
}

// Row i of qkv (fp32: q | k | v) = position pos0 + i: clip, interleaved-pair RoPE on q and k (src/infer.cpp:200-213,
// 282-292), q -> fp16 (attention operand), k / v -> fp16 rows pos0 + i of the head-major KV ring (src/infer.cpp:294-301).
// A thread takes one pair of a head's channels through every blockDim / half-th head: the angle's power, sine and cosine, most of the work, are
// formed once per thread instead of once per pair (512 rows of 32 + 8 heads of 128: 18 -> 11 us).
__global__ void __launch_bounds__(512) rope_append_rows_kernel(__half *q16, __half *kc, __half *vc, const float *qkv, int n_heads, int n_kv, int head_dim,
                                                               int rotary_dim, int max_seq_len, int pos0, float theta, float clip) {
	const int i = blockIdx.x, pos = pos0 + i, half = head_dim / 2, at_once = blockDim.x / half, q_dim = n_heads * head_dim;
	const int j = (threadIdx.x % half) * 2, first = threadIdx.x / half;
	if (first >= at_once) return;
	chain_wait();
	chain_next();
	const float *row = qkv + (size_t)i * (q_dim + 2 * n_kv * head_dim);
	float fcr, fci;
	rope_angle(fcr, fci, j, pos, theta, rotary_dim);
	constexpr int kBatch = 4;
	const int heads = n_heads + 2 * n_kv; // q heads, k heads, v heads
	for (int h0 = first; h0 < heads; h0 += kBatch * at_once) {
		float2 v[kBatch]; // reads first, then stores
#pragma unroll
		for (int b = 0; b < kBatch; ++b)
			if (h0 + b * at_once < heads) v[b] = *reinterpret_cast<const float2 *>(row + (size_t)(h0 + b * at_once) * head_dim + j);
#pragma unroll
		for (int b = 0; b < kBatch; ++b) {
			const int h = h0 + b * at_once;
			if (h >= heads) break;
			float v0 = clipf(v[b].x, clip), v1 = clipf(v[b].y, clip);
			if (h < n_heads + n_kv) rope_turn(v0, v1, fcr, fci);
			__half *dst = h < n_heads ? q16 + (size_t)i * q_dim + h * head_dim
			                          : (h < n_heads + n_kv ? kc + ((size_t)(h - n_heads) * max_seq_len + pos) * head_dim
			                                                : vc + ((size_t)(h - n_heads - n_kv) * max_seq_len + pos) * head_dim);
			*reinterpret_cast<__half2 *>(dst + j) = __floats2half2_rn(v0, v1);
		}
	}
}

} // namespace prefill
} // namespace yalm

using namespace yalm;
using namespace yalm::prefill;

// Causal attention of n query rows (positions pos0 .. pos0 + n - 1) over the head-major fp16 KV ring.  Device pointers.
extern "C" int yalm_attn_prefill(void *out16, const void *q16, const uint16_t *key_cache, const uint16_t *value_cache, int n, int pos0,
                                 int n_heads, int n_kv_heads, int head_dim, int max_seq_len, yalm_stream_t s) {
	if (!out16 || !q16 || !key_cache || !value_cache || n < 1 || pos0 < 0 || pos0 + n > max_seq_len || n_kv_heads < 1 || n_heads % n_kv_heads)
		return YALM_EINVAL;
	return prompt::causal_f16(out16, q16, key_cache, value_cache, n, pos0, n_heads, n_kv_heads, head_dim, max_seq_len, (cudaStream_t)s);
}

// ---- Model::forward_batch ------------------------------------------------------------------------------------------
struct Model::PrefillState {
	int cap = 0;
	char *arena = nullptr;
	float *x = nullptr, *qkv = nullptr, *logits = nullptr, *probs = nullptr;
	__half *xb = nullptr, *q16 = nullptr, *att = nullptr, *hb = nullptr;
	float2 *turns = nullptr;
	int *tokens = nullptr, *targets = nullptr;
	~PrefillState() { cudaFree(arena); }
};

bool Model::supports_batch() const {
	const Config &c = *config;
	if (c.stack) return _device == Device::CUDA; // the layered executor takes any number of rows per call
	const char *env = getenv("YALM_B200_PREFILL");
	if (env && env[0] == '0') return false;
	return _device == Device::CUDA && c.weight_dtype == DType::F16 && c.n_experts == 0 && c.tp_size == 1 &&
	       (c.head_dim == 128 || c.head_dim == 64 || c.head_dim == 32) && c.dim % 8 == 0 && c.hidden_dim % 8 == 0 &&
	       (c.n_heads * c.head_dim) % 8 == 0 && (c.n_kv_heads * c.head_dim) % 8 == 0;
}

int Model::batch_capacity() const {
	if (config->stack) return supports_batch() ? config->max_seq_len : 0;
	return supports_batch() ? kPortionRows : 0;
}

int Model::forward_batch(InferenceState &s, const int *tokens, int n, int pos0, const int *targets, float *probs_out) {
	if (!supports_batch() || s.device() != Device::CUDA) return YALM_EINVAL;
	const Config &c = *config;
	if (c.stack) { // last row's logits for the samplers, or every row's probability of its target
		const int last = n - 1;
		return stack_rows(s, tokens, n, pos0, targets ? nullptr : &last, targets ? 0 : 1, nullptr, targets, probs_out);
	}
	const int cap = batch_capacity();
	if (!tokens || n < 1 || n > cap || pos0 < 0 || pos0 + n > c.max_seq_len || (targets && !probs_out)) return YALM_EINVAL;
	for (int i = 0; i < n; ++i)
		if (tokens[i] < 0 || tokens[i] >= c.vocab_size) return YALM_EINVAL;
	const int dim = c.dim, q_dim = c.n_heads * c.head_dim, kv_dim = c.n_kv_heads * c.head_dim, hid = c.hidden_dim, V = c.vocab_size;
	cudaStream_t st = s.stream();
	if (!_prefill) {
		auto ps = std::make_shared<PrefillState>();
		ps->cap = cap;
		auto pad = [](size_t b) { return (b + 255) / 256 * 256; };
		// fp32 projections and logits are stored of few rows only; of more, what the softmax of a row needs of every tile of logits
		const size_t sz[] = {pad(4ull * cap * dim), pad(4ull * kFewRows * (q_dim + 2 * kv_dim)), pad(std::max<size_t>(4ull * kFewRows * V, score_bytes(V))), pad(4ull * cap),
		                     pad(2ull * cap * std::max(dim, q_dim)), pad(2ull * cap * q_dim), pad(2ull * cap * q_dim), pad(2ull * cap * hid),
		                     pad(4ull * cap), pad(4ull * cap), pad(4ull * cap * c.head_dim)};
		size_t total = 0;
		for (size_t b : sz) total += b;
		if (cudaMalloc((void **)&ps->arena, total) != cudaSuccess) {
			cudaGetLastError();
			return (int)cudaErrorMemoryAllocation;
		}
		char *p = ps->arena;
		void **slots[] = {(void **)&ps->x, (void **)&ps->qkv, (void **)&ps->logits, (void **)&ps->probs, (void **)&ps->xb,
		                  (void **)&ps->q16, (void **)&ps->att, (void **)&ps->hb, (void **)&ps->tokens, (void **)&ps->targets,
		                  (void **)&ps->turns};
		for (int i = 0; i < 11; ++i) *slots[i] = p, p += sz[i];
		_prefill = ps;
	}
	PrefillState &P = *_prefill;
	YALM_TRY(cudaMemcpyAsync(P.tokens, tokens, sizeof(int) * n, cudaMemcpyHostToDevice, st));
	if (targets) YALM_TRY(cudaMemcpyAsync(P.targets, targets, sizeof(int) * n, cudaMemcpyHostToDevice, st));
	embed_rows_kernel<<<n, 256, 0, st>>>(P.x, static_cast<const __half *>(token_embedding_table), P.tokens, dim);
	const int act = c.act == ActivationType::SILU ? YALM_ACT_SILU : YALM_ACT_GELU;
	const bool many = n > kFewRows; // the kernels of more rows finish q, k and v, and the probabilities, themselves
	int rc;
	if (many) {
		const int per = 256 / (c.head_dim / 2);
		if ((rc = launch_chained(turns_kernel, dim3((n + per - 1) / per), dim3(256), 0, st, 1, P.turns, n, c.head_dim, c.rotary_dim, pos0, c.rope_theta))) return rc;
	}
	for (auto &bp : blocks) {
		const Block &b = *bp;
		if ((rc = launch_chained(rmsnorm_rows_kernel, dim3(n), dim3(kNormThreads), 0, st, 1, P.xb, P.x, b._rms_att_weight, dim, c.norm_eps))) return rc;
		if (many) {
			if ((rc = gemm_qkv_rotate(P.q16, b._key_cache, b._value_cache, P.turns, P.xb, b._wq, b._wk, b._wv, n, q_dim, kv_dim, dim, c.head_dim, c.max_seq_len, pos0, c.qkv_clip, st)))
				return rc;
		} else {
			// q | k | v of the chunk into one (n, q_dim + 2 kv_dim) fp32 buffer
			const int ld = q_dim + 2 * kv_dim;
			if ((rc = gemm_qkv_f16(P.qkv, ld, P.xb, b._wq, b._wk, b._wv, n, q_dim, kv_dim, dim, st))) return rc;
			if ((rc = launch_chained(rope_append_rows_kernel, dim3(n), dim3(512), 0, st, 1, P.q16, reinterpret_cast<__half *>(b._key_cache),
			                         reinterpret_cast<__half *>(b._value_cache), (const float *)P.qkv, c.n_heads, c.n_kv_heads, c.head_dim, c.rotary_dim, c.max_seq_len, pos0,
			                         c.rope_theta, c.qkv_clip)))
				return rc;
		}
		if ((rc = yalm_attn_prefill(P.att, P.q16, b._key_cache, b._value_cache, n, pos0, c.n_heads, c.n_kv_heads, c.head_dim, c.max_seq_len, st)))
			return rc;
		if ((rc = yalm_gemm_f16(P.x, dim, P.att, b._wo, n, dim, q_dim, 1, st))) return rc; // x += Wo att
		if ((rc = launch_chained(rmsnorm_rows_kernel, dim3(n), dim3(kNormThreads), 0, st, 1, P.xb, P.x, b._rms_ffn_weight, dim, c.norm_eps))) return rc;
		if ((rc = yalm_gemm_glu_f16(P.hb, hid, P.xb, b._w1, b._w3, n, hid, dim, act, st))) return rc;
		if ((rc = yalm_gemm_f16(P.x, dim, P.hb, b._w2, n, dim, hid, 1, st))) return rc; // x += W2 hb
	}
	if (targets) { // per-position logits -> probability of the given next token (Sampler::sample_prob per row)
		if ((rc = launch_chained(rmsnorm_rows_kernel, dim3(n), dim3(kNormThreads), 0, st, 1, P.xb, P.x, rms_final_weight, dim, c.norm_eps))) return rc;
		if (many) {
			if ((rc = gemm_score(P.probs, P.logits, P.targets, P.xb, wcls, n, V, dim, st))) return rc;
		} else {
			if ((rc = yalm_gemm_f16(P.logits, V, P.xb, wcls, n, V, dim, 0, st))) return rc;
			if ((rc = yalm_token_probs(P.logits, V, n, P.targets, P.probs, st))) return rc;
		}
		YALM_TRY(cudaMemcpyAsync(probs_out, P.probs, sizeof(float) * n, cudaMemcpyDeviceToHost, st));
	}
	// the LAST position's logits through the decode path's final norm + LM head (fp32 activations), as after forward()
	if ((rc = yalm_lm_head(s.logits_dev(), P.x + (size_t)(n - 1) * dim, rms_final_weight, wcls, wcls_scale, dim, V, c.norm_eps,
	                       static_cast<int>(c.weight_dtype), st)))
		return rc;
	if (s.host_logits())
		YALM_TRY(cudaMemcpyAsync(s.logits(), s.logits_dev(), sizeof(float) * V, cudaMemcpyDeviceToHost, st));
	YALM_TRY(cudaStreamSynchronize(st));
	yalm::mega::check_fault(); // (of tokens before this portion, whose keys and values it has read)
	return (int)cudaGetLastError();
}
