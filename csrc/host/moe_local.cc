// Forward and backward pass of a single-rank MoE layer, each one call: the launches that moonep_b200/moe_layer.py issues one by
// one (about 15 us of Python each), with the weight gradients of gate and up as the last one, for callers without hooks between them.
#include "../device/gemm_args.h"
#include "../device/local_args.h"
#include "launch.h"

extern "C" {
int mep_launch_local_dispatch(const MepRankCtx*, const mep::LocalDispatchArgs*, int, int, int, int, int, int, int, int, cudaStream_t);
int mep_launch_local_combine(const MepRankCtx*, const mep::LocalCombineArgs*, int, int, int, int, int, int, cudaStream_t);
int mep_grouped_gemm_2cta(int, const void*, int64_t, int64_t, int64_t, const void*, const void*, int64_t, int64_t, int64_t,
                          const mep::GemmArgs*, int, cudaStream_t);
int mep_grouped_wgrad_2cta(const void*, int64_t, int64_t, const void*, int64_t, const mep::GemmArgs*, int, cudaStream_t);
int mep_swiglu_bwd(const void*, const void*, const float*, void*, float*, const int32_t*, int, int, int, int, cudaStream_t);
}

namespace mep {

// A pass begins with a dispatch, which lets the next launch begin when everything before it in the stream is done. Weights, and the
// plan of a backward pass, are therefore complete before any GEMM of the pass begins, and so are the token counts that a forward
// pass is given (`tpe`; its plan is written by the dispatch).
static GemmArgs gemm_args(const MoeLocal& m, const int32_t* slab, const int32_t* tpe = nullptr) {
  GemmArgs a = {};
  a.cu_seqlens = slab + m.plan_off[7];
  a.pad_rows = slab + m.plan_off[2];
  a.G = 2 * m.E; a.g_end = 2 * m.E;
  a.early = 1; a.tokens = tpe; a.tokens_n = m.E; a.token_padding = m.token_padding;
  a.pdl = m.pdl;                 // behind another kernel of the same call
  a.held = m.E; a.held_rows = m.S * m.K;
  a.status = m.status; a.status_host = m.status_host; a.budget_ns = m.budget_ns;
  return a;
}

static LocalDispatchArgs dispatch_args(const MoeLocal& m, const void* hidden, int32_t* slab) {
  LocalDispatchArgs d = {};
  d.hidden = (const __nv_bfloat16*)hidden;
  d.pad_step = 32;               // no GEMM of this layer reads further
  d.out_srcinfo = m.srcinfo;
  d.dst = slab + m.plan_off[0]; d.zero_fill = slab + m.plan_off[2];
  return d;
}

// Whether a pass's dispatch may begin while the kernel before still runs. A programmatic launch finds the SMs in the order in which that kernel leaves
// them, and the GEMM pairs behind it inherit the order; after an ordinary one neighbours in the tile list are close to each other and read the
// same lines of L2. Forward passes that begin with a programmatic / an ordinary dispatch, in us, by MiB of rows moved, six alternations: 2 (2048 x 768,
// 64 tokens) 43.5 / 47.3; 18 (512) 69.0 / 75.6; 36 (1024) 99.3 / 106.5; 39 (7168 x 2048, 320) 498 / 500; 54 (2048 x 768, 1531) 131.0 / 140.0 and
// 128.6 / 130.3 on another box; 63 (7168 x 2048, 512) 583 / 567; 126 (1024) 799 / 834 and 852 / 798; 252 (2048) 1465 / 1454; 504 (4096) 2682 / 2701 and 2782 / 2736.
// So from the line on neither is better by more than runs and boxes differ.
static int early_dispatch(const MoeLocal& m) { return m.pdl && (int64_t)m.S * (m.K + 1) * m.H * 2 < (40ll << 20); }

static void plan_into(const MoeLocal& m, const int32_t* topk, const int32_t* tpe, int32_t* slab, LocalDispatchArgs* d) {
  d->topk = topk; d->tpe = tpe;
  d->dst = slab + m.plan_off[0]; d->experts_to_copy = slab + m.plan_off[1]; d->zero_fill = slab + m.plan_off[2];
  d->remote_stats = slab + m.plan_off[3]; d->dup_groups = slab + m.plan_off[4]; d->dup_loffs = slab + m.plan_off[5];
  d->dup_counts = slab + m.plan_off[6]; d->cu_seqlens = slab + m.plan_off[7];
  d->sync = m.sync; d->hist = m.hist;
}

// x [NvS, in] times weights [2E, in, out] (or their transposes), see GemmMode
static int gemm(const MoeLocal& m, GemmMode mode, const void* a, int64_t a_cols, const void* b0, const void* b1, int64_t in, int64_t out,
                GemmArgs& g, cudaStream_t stream) {
  g.b_group_rows = (int32_t)in;
  return mep_grouped_gemm_2cta(mode, a, m.NvS, a_cols, a_cols, b0, b1, 2 * (int64_t)m.E * in, out, out, &g, m.num_ctas, stream);
}

}  // namespace mep

// Dispatch and combine alone, for a Buffer whose caller computes the experts. Dispatch plans into `slab` when `topk` is
// given and reads the plan from it otherwise; `dst` / `zero_fill` may come from another plan's tensors instead.
extern "C" int mep_local_dispatch_call(const mep::MoeLocal* mp, const void* hidden, const float* route_w, const int32_t* topk, const int32_t* tpe,
                                       int32_t* slab, int32_t* dst, int32_t* zero_fill, void* rows, float* row_w, cudaStream_t stream) {
  using namespace mep;
  const MoeLocal& m = *mp;
  LocalDispatchArgs d = {};
  d.hidden = (const __nv_bfloat16*)hidden; d.weights = route_w;
  d.out_hidden = (__nv_bfloat16*)rows; d.out_weights = row_w; d.out_srcinfo = m.srcinfo;
  d.dst = dst; d.zero_fill = zero_fill;
  if (topk) plan_into(m, topk, tpe, slab, &d);
  return mep_launch_local_dispatch(m.ctx, &d, topk ? 1 : 0, m.blocks, m.sms, m.S, m.K, m.H, m.E, m.pdl, stream);
}

extern "C" int mep_local_combine_call(const mep::MoeLocal* mp, const int32_t* dst, const void* rows, const float* row_w, void* out, float* out_w,
                                      cudaStream_t stream) {
  using namespace mep;
  const MoeLocal& m = *mp;
  LocalCombineArgs c = {dst, (const __nv_bfloat16*)rows, row_w, (__nv_bfloat16*)out, out_w};
  return mep_launch_local_combine(m.ctx, &c, m.combine_blocks, m.S, m.H, m.K, m.pdl, m.in_order && m.combine_blocks >= m.sms, stream);
}

extern "C" int mep_moe_local_forward(const mep::MoeLocal* mp, const void* hidden, const float* route_w, const int32_t* topk,
                                     const int32_t* tpe, int32_t* slab, void* out, int keep, cudaStream_t stream) {
  using namespace mep;
  const MoeLocal& m = *mp;
  __nv_bfloat16* x = keep ? m.x : m.shard;
  float* w = keep ? m.w : m.shard_w;
  LocalDispatchArgs d = dispatch_args(m, hidden, slab);
  d.weights = route_w; d.out_hidden = x; d.out_weights = w;
  plan_into(m, topk, tpe, slab, &d);
  if (mep_launch_local_dispatch(m.ctx, &d, 1, m.blocks, m.sms, m.S, m.K, m.H, m.E, early_dispatch(m), stream)) return -1;
  GemmArgs g = gemm_args(m, slab, tpe);
  g.N = m.Hp; g.K = m.H; g.out = m.act; g.out2 = keep ? m.gu : nullptr; g.row_scale = w; g.ldo = m.Hp;
  if (gemm(m, GEMM_GATE_UP, x, m.H, m.w_gate, m.w_up, m.H, m.Hp, g, stream)) return -1;
  g = gemm_args(m, slab, tpe);
  g.N = m.H; g.K = m.Hp; g.out = m.shard; g.ldo = m.H;
  if (gemm(m, GEMM_DOWN, m.act, m.Hp, m.w_down, nullptr, m.Hp, m.H, g, stream)) return -1;
  LocalCombineArgs c = {slab + m.plan_off[0], m.shard, nullptr, (__nv_bfloat16*)out, nullptr};
  return mep_launch_local_combine(m.ctx, &c, m.combine_blocks, m.S, m.H, m.K, m.pdl, 0, stream);
}

// `update`: lr and the group mask of the update in the weight-gradient epilogues, or mask = null (gradients are stored).
extern "C" int mep_moe_local_backward(const mep::MoeLocal* mp, const void* dy, int32_t* slab, void* dx, float* d_route_w, int accumulate,
                                      float lr, const int32_t* mask, cudaStream_t stream) {
  using namespace mep;
  const MoeLocal& m = *mp;
  LocalDispatchArgs d = dispatch_args(m, dy, slab);
  d.out_hidden = m.shard;
  if (mep_launch_local_dispatch(m.ctx, &d, 0, m.blocks, m.sms, m.S, m.K, m.H, m.E, early_dispatch(m), stream)) return -1;
  GemmArgs g = gemm_args(m, slab);
  g.N = m.Hp; g.K = m.H; g.out = m.dA; g.ldo = m.Hp;
  if (gemm(m, GEMM_DGRAD, m.shard, m.H, m.w_down, nullptr, m.Hp, m.H, g, stream)) return -1;
  const int32_t* cu = slab + m.plan_off[7];
  if (mep_swiglu_bwd(m.dA, m.gu, m.w, m.dgu, m.shard_w, cu, 2 * m.E, m.Hp, 4 * m.num_ctas, m.pdl, stream)) return -1;
  auto wgrad = [&](const void* x, int64_t in, const void* dyc, int64_t ld, int64_t out, float* dw, const void* w, float* dw_b, const void* w_b) {
    GemmArgs a = gemm_args(m, slab);
    a.N = (int32_t)(dw_b ? 2 * out : out); a.M_w = (int32_t)in; a.accumulate = accumulate; a.zero_empty_below = m.E; a.out = dw;
    if (dw_b) { a.n_each = (int32_t)out; a.out_b = dw_b; }
    if (mask) { a.upd_w = const_cast<void*>(w); a.upd_w_b = const_cast<void*>(w_b); a.upd_mask = mask; a.upd_lr = lr; }
    return mep_grouped_wgrad_2cta(x, m.NvS, in, dyc, ld, &a, m.num_ctas, stream);
  };
  if (wgrad(m.act, m.Hp, m.shard, m.H, m.H, m.dw_down, m.w_down, nullptr, nullptr)) return -1;
  g = gemm_args(m, slab);
  g.N = m.H; g.K = 2 * m.Hp; g.out = m.shard; g.ldo = m.H;
  if (gemm(m, GEMM_DGRAD_GU, m.dgu, 2 * (int64_t)m.Hp, m.w_gate, m.w_up, m.H, m.Hp, g, stream)) return -1;
  LocalCombineArgs c = {slab + m.plan_off[0], m.shard, m.shard_w, (__nv_bfloat16*)dx, d_route_w};
  if (mep_launch_local_combine(m.ctx, &c, m.combine_blocks, m.S, m.H, m.K, m.pdl, 0, stream)) return -1;
  // Gate and up in one launch: x is read from DRAM once and there is one ramp and one last round. 16 groups of 4096 tokens, 2048 x 768: 323 -> 307 us
  // (with the update 318 -> 302); 24 of 700, 1792 x 1280: 196 -> 181; 16 of 300, 1024 x 512: 44 -> 30. An update of their weights has to wait for dgrad(gate/up), which reads them.
  return wgrad(m.x, m.H, m.dgu, 2 * (int64_t)m.Hp, m.Hp, m.dw_gate, m.w_gate, m.dw_up, m.w_up);
}

MEP_EXPORT_SIZEOF(MoeLocal, mep::MoeLocal)
