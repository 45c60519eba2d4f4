// Argument blocks of the single-rank exchange kernels (local_exchange.cu) and of the layer calls built on them.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>
#include "../mep_types.h"

namespace mep {

struct LocalDispatchArgs {
  const __nv_bfloat16* hidden;   // [S, H]
  const float* weights;          // [S, K] or null
  __nv_bfloat16* out_hidden;     // [NvS, H]
  float* out_weights;            // [NvS]
  int32_t* out_srcinfo;          // [NvS] provenance table or null
  int32_t* dst;                  // [N]   plan (written when fresh, read otherwise)
  int32_t* zero_fill;            // [2E, 2]
  // fresh only
  const int32_t* topk;           // [N]
  const int32_t* tpe;            // [E]
  int32_t* cu_seqlens;           // [2E]
  int32_t* experts_to_copy;      // [1, E]
  int32_t* remote_stats;         // [2]
  int32_t* dup_groups;           // [NvS, 3]
  int32_t* dup_loffs;            // [NvS]
  int32_t* dup_counts;           // [2]
  uint32_t* sync;                // [0] launches completed, [1] start tickets, [2] finished CTAs, [16 + b] flag of CTA b
  int32_t* hist;                 // [grid, E] expert histogram of each CTA's tokens
  int32_t pad_step;              // 0: every padding row is cleared; else those up to the next multiple of this (a power of
                                 // two that divides token_padding), which is as far as the CTA-pair GEMMs read
  int32_t early;                 // a programmatic launch (set by the launcher)
};

struct LocalCombineArgs {
  const int32_t* dst;            // [N] plan
  const __nv_bfloat16* rows;     // [NvS, H]
  const float* weights;          // [NvS] or null
  __nv_bfloat16* out;            // [S, H]
  float* out_weights;            // [S, K] or null
};

// Everything of a single-rank MoE layer that stays the same from call to call (moe_local.cc).
struct MoeLocal {
  const MepRankCtx* ctx;         // device
  int32_t S, H, Hp, K, E, NvS;
  int32_t blocks, combine_blocks, num_ctas;      // CTAs of dispatch, combine (most) and of the GEMMs
  int32_t pdl;                   // 1: programmatic launches between the kernels of one call
  int64_t plan_off[8];           // elements from the start of a plan's allocation: dst, experts_to_copy, zero_fill,
                                 // remote_stats, dup_groups, dup_loffs, dup_counts, cu_seqlens
  const void *w_gate, *w_up, *w_down;            // [2E, in, out] bf16; these and the gradients are set for each call
  __nv_bfloat16* shard;          // [NvS, H] the Buffer's shard
  float* shard_w;                // [NvS]
  int32_t* srcinfo;              // or null
  __nv_bfloat16* x;              // [NvS, H] dispatched tokens kept for the backward pass
  float* w;                      // [NvS]
  __nv_bfloat16 *act, *gu, *dA, *dgu;
  float *dw_gate, *dw_up, *dw_down;              // [2E, in, out] fp32, or null
  uint32_t* sync;
  int32_t* hist;
  int32_t* status;
  int32_t* status_host;
  uint64_t budget_ns;
  int32_t token_padding;
  int32_t sms;                   // of the device
  int32_t in_order, reserved;    // combine call: the rows come from a saved plan's dispatch, which on a whole device goes through a large
                                 // batch in the order of the tokens (see local_combine_kernel)
};

}  // namespace mep
