// The products of a prompt portion that only Model::forward_batch calls (prefill_gemm.cu).
#pragma once

#include <cuda_runtime_api.h>
#include <stddef.h>

namespace yalm {
namespace prefill {

constexpr int kFewRows = 128;     // up to here a portion's products run on the few-rows kernel, and kernels of their own rotate, append and score
constexpr int kPortionRows = 512; // most rows of a portion

// Up to kFewRows rows: the three projections of a layer as one launch, side by side in c (M, ldc) fp32.
int gemm_qkv_f16(float *c, int ldc, const void *a, const void *wq, const void *wk, const void *wv, int M, int q_dim, int kv_dim, int K, cudaStream_t st);
// More rows: the same, rotated and appended.
int gemm_qkv_rotate(void *q, void *k, void *v, const void *turns, const void *a, const void *wq, const void *wk, const void *wv, int M, int q_dim, int kv_dim, int K,
                    int head_dim, int ring, int pos0, float clip, cudaStream_t st);
// More rows: the probabilities of targets without the logits; scratch: score_bytes(N).
size_t score_bytes(int N);
int gemm_score(float *probs, void *scratch, const int *targets, const void *a, const void *w, int M, int N, int K, cudaStream_t st);

} // namespace prefill
} // namespace yalm
