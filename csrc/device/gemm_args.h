// Argument block of the grouped GEMM kernels (shared by the 1-CTA and the 2-CTA launchers).
#pragma once
#include <stdint.h>

namespace mep {

enum GemmMode { GEMM_GATE_UP = 0, GEMM_DOWN = 1, GEMM_DGRAD = 2, GEMM_DGRAD_GU = 3, GEMM_WGRAD = 4 };

struct GemmArgs {
  const int32_t* cu_seqlens;   // [G] padded end row of each group
  int32_t G;
  int32_t N;                   // output columns (GATE_UP: width of act = out dim of each weight)
  int32_t K;                   // reduction length (DGRAD_GU: 2 * inner); unused for WGRAD
  int32_t M_w;                 // WGRAD: rows of one weight matrix
  int32_t b_group_rows;        // rows one group occupies in the flattened 2-D weight tensor(s)
  int32_t accumulate;          // WGRAD: 1 -> out += acc, 0 -> out = acc
  int32_t g_begin, g_end;      // only groups in [g_begin, g_end) are computed
  int32_t zero_empty_below;    // WGRAD without accumulate: empty groups g < this get zeros
  int32_t pdl;                 // 1: programmatic launch -- the kernel right before in the stream is one of this library's that may
                               // still be running (CTA-pair kernels only)
  void* out;                   // bf16 [rows, ldo]; WGRAD: fp32 [G, M_w, N]
  void* out2;                  // GATE_UP: optional bf16 [rows, 2N] pre-activations (gate | up)
  const float* row_scale;      // GATE_UP / DOWN: optional per-row factor [rows]
  int64_t ldo;
  int32_t* status;             // [4] error word: code, site, block, tile
  uint64_t budget_ns;
  uint32_t* sched;             // [2] zero-initialised ticket counter of the dynamic tile scheduler, or null for
                               // the static strided tile order
  // DOWN / DGRAD / DGRAD_GU, optional "push" epilogue: row r of the output is not stored to `out` but sent
  // to the rank it came from: push_info[r] = src_rank * push_rows + index (or < 0 for a padding row) and the
  // row lands at push_base + src_rank * push_stride + index * N * 2 (row `index` of that rank's [push_rows, N]
  // bf16 receive area inside the symmetric heap). push_wsrc[r], if given, goes to the float at
  // push_wbase + src_rank * push_stride + index * 4.
  const int32_t* push_info;
  unsigned char* push_base;
  unsigned char* push_wbase;
  const float* push_wsrc;
  uint64_t push_stride;
  // GATE_UP / DGRAD, optional: the rows of `a` are produced by a flagged dispatch that is still running.
  // tile_done[t] holds the flag epoch at which rows [128 t, 128 t + 128) became complete; the TMA producer waits
  // (bounded) for tile_done[t] >= *tile_epoch before it loads rows of tile t. The launch must leave the dispatch
  // kernel's SMs free (num_ctas <= SMs - its CTAs), since that kernel has to be resident meanwhile.
  const uint32_t* tile_done;
  const uint32_t* tile_epoch;
  int32_t* status_host;        // optional host-mapped copy of status[0]
  // optional: the weights of groups g >= group_first are still being written by a prefetch. group_flags[g -
  // group_first] holds the prefetch epoch at which that slot became complete; the TMA producer waits (bounded)
  // for it to reach *group_epoch before it loads weights of such a group.
  const uint32_t* group_flags;
  const uint32_t* group_epoch;
  int32_t push_rows;
  int32_t push_ranks;
  int32_t group_first;
  int32_t sched_ctas;          // dynamic order: CTAs over ALL launches that draw from `sched` (several launches of
                               // one GEMM may share a counter); 0 = just this launch
  // WGRAD (CTA-pair kernel), optional optimizer in the epilogue: for a group g with upd_mask[g] != 0 the
  // gradient tile is not written to `out`; the bf16 weights upd_w[g] (same [G, M_w, N] layout) are updated in
  // place instead, w -= upd_lr * dW, with the arithmetic of the stand-alone SGD kernel. Groups with
  // upd_mask[g] == 0 (e.g. experts whose gradient still has to be reduced across ranks) are written as usual.
  void* upd_w;
  const int32_t* upd_mask;
  float upd_lr;
  int32_t sched_odd;           // CTA-pair launches on a shared counter: CTAs asked for beyond those of the grid (1: an odd number,
                               // -1: a single one, which runs as a pair)
  // optional [G, 2] table (first padding row, padding rows) of the groups, as a plan carries it: rows behind the real
  // ones, rounded up to 32, are then neither computed nor read (null: all padded rows are). CTA-pair kernels only.
  const int32_t* pad_rows;
  // CTA-pair kernels. early: what a launch reads besides the rows of `a` (WGRAD: besides both operands) and row_scale -- the tables below or cu_seqlens and
  // pad_rows, the weights, upd_mask -- was complete before the kernel right before it in the stream let its dependents launch. The launch then
  // sets up its tiles and loads the first weights while that kernel still runs. A programmatic dispatch or combine of one rank lets them in when everything
  // before it is done, so behind it that holds of whatever was queued before it; the GEMMs and the SwiGLU kernel let them in at their own
  // start, so behind those it holds of what was complete before the first of an unbroken row of them.
  // tokens, optional: token counts of groups 0 to tokens_n - 1 (the others are empty), instead of cu_seqlens and pad_rows; groups are padded to
  // multiples of token_padding rows.
  const int32_t* tokens;
  int32_t tokens_n, token_padding, early;
  // WGRAD (CTA-pair kernel): 0, or the columns of one weight matrix (a multiple of 256), N = 2 * n_each: the second half of dy's columns
  // gives the gradient (update) of another matrix of the same shape, out_b (upd_w_b).
  int32_t n_each;
  void *out_b, *upd_w_b;
  // Token-major CTA-pair kernels: groups that hold rows, as far as the caller knows, and their rows without padding; 0: all G, and the rows of `a`. They
  // only decide which kernel runs.
  int32_t held, held_rows;
};

// CTAs of a pair launch that was asked for `n`. On a counter shared with other launches the grid accounts for all `n`.
inline int pair_ctas(GemmArgs* a, int n) {
  const int grid = a->sched_ctas > 0 && n == 1 ? 2 : n & ~1;
  a->sched_odd = a->sched_ctas > 0 ? n - grid : 0;
  return grid;
}

}  // namespace mep
