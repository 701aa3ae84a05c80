// The single-token attention kernels (attn_decode.cu).
#pragma once

#include "kernels.h"

namespace bk {

struct DecAttnParams;

// Whether this geometry fits: head sizes 64, 128 and 256, and positions (a context, or a sliding-window layer's window) whose
// probabilities fit shared memory.
bool attn_decode_fits(uint32_t dim, uint32_t positions);
// Norm, RoPE, cache store, scores, softmax and weighted sum of one token, in one kernel (fused; heads of 64 and 128) or two;
// returns how many. window: positions the token sees (0: all).
int launch_attn_decode(const DecAttnParams& a, uint32_t window, bool fused, cudaStream_t s);

}  // namespace bk
