// Where the split partials of one-token attention (ops_attn.cu) lie inside the caller's workspace.
#pragma once

#include <cstddef>
#include <cstdint>

namespace yalm {

// Bytes from the workspace's start: arrival counters (one per KV head, zero between launches) at 0, then the accumulators
// (KV head, split, query head of it, channel) and (maximum, sum) (KV head, split, query head, 2), fp32.  The merge reads the accumulators 16
// bytes at a time, so they start at a 16-byte boundary whatever the counts and the workspace's own alignment (4 bytes): (maximum, sum) before
// them would leave them 8 bytes off where KV heads x splits x query heads is odd (5 x 59 x 1 on 148 SMs).  The first 256 bytes of a 16-byte aligned
// workspace hold nothing but counters: calls of other shapes on the same workspace find theirs zero.
struct AttnWorkspace {
	size_t acc, ml, bytes;
};
inline AttnWorkspace attn_workspace(uintptr_t at, int n_kv, int splits, int g, int head_dim) {
	const size_t counters = (size_t)n_kv * sizeof(unsigned), rows = (size_t)n_kv * splits * g;
	AttnWorkspace w;
	w.acc = (at + counters + 256) / 16 * 16 - at;
	w.ml = w.acc + rows * head_dim * sizeof(float);
	w.bytes = rows * (head_dim + 2) * sizeof(float) + counters + 256;
	return w;
}

} // namespace yalm
