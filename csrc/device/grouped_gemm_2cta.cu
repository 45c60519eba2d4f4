// Weight-gradient grouped GEMM on CTA pairs: dW[g] (+)= X_g^T dY_g with tcgen05.mma.cta_group::2.
//
// Two CTAs of a cluster (two SMs) compute one 256 x 256 fp32 tile: each CTA stages ITS half of both
// operands (128 weight rows of X^T and 128 of the 256 output columns of dY, 32 KB per 64-token
// k-block) with ordinary single-CTA TMA loads from local memory, and the pair's tensor cores read
// both halves. Per SM that is 32 KB of shared-memory fill per k-block instead of 48 KB for the same
// amount of math, which is what limits the single-CTA kernel (operand feed, not the tensor pipe).
// No cluster-wide copy is used: every load lands in the issuing CTA only and merely counts its bytes
// on the leader CTA's mbarrier. The M tile is over weight rows, so it never straddles experts.
// Roles per CTA: warp 0 = TMA producer, warp 1 = TMEM allocation (+ MMA issue in the leader CTA),
// warps 2-9 = epilogue (each CTA drains its own 128 accumulator rows through shared memory + TMA
// store / reduce-add).
#include "tcgen05.cuh"
#include "pair.cuh"
#include "tile_queue.cuh"
#include "gemm_args.h"
#include "tmap.h"

namespace mep {
namespace w2 {

constexpr int kBK = 64, kRing = 5, kEpiWarps = 8, kThreads = 64 + 32 * kEpiWarps;
constexpr int kHalfBytes = 128 * kBK * 2;            // 16 KB: one operand half per CTA and k-block
constexpr int kStageBytes = 2 * kHalfBytes;          // 32 KB
constexpr int kAtomBytes = 64 * kBK * 2;
constexpr int kSlabBytes = 32 * 128;
constexpr int kMaxGroups = 192;
constexpr size_t kSmem = (size_t)kRing * kStageBytes + (size_t)kEpiWarps * 2 * kSlabBytes + 1024;

using namespace pair;

constexpr int kBandElems = 9 << 20;                          // elements of x for a group, on average over all G: 18 MB

struct Tile { int g, row0, m0, n0, kblocks, ksteps; };      // ksteps: 16-row steps (a k-block has four)

__global__ void __launch_bounds__(kThreads, 1)
wgrad_2cta_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                  const __grid_constant__ CUtensorMap tma_out, const __grid_constant__ CUtensorMap tma_out_b, GemmArgs args) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[kRing], empty_bar[kRing], tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t s_tmem_base;
  __shared__ volatile int s_abort;
  __shared__ tq::Ring s_ring;
  __shared__ int s_cu[kMaxGroups], s_units[kMaxGroups];     // first row, 32-row units of a group
  __shared__ unsigned char s_act[kMaxGroups];               // groups with tiles
  __shared__ int s_total;                                   // rows of all groups
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cr = cluster_ctarank();
  const bool leader = cr == 0;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int G = args.G;
  pdl_trigger();

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < kRing; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&tfull_bar[i], 1); mbar_init(&tempty_bar[i], 2 * kEpiWarps); }
    tq::init(&s_ring, 2 * kEpiWarps + 2);      // both CTAs' epilogue warps, the MMA issuer, the peer's producer
    fence_mbar_init();
    tc::prefetch_tmap(&tma_a); tc::prefetch_tmap(&tma_b); tc::prefetch_tmap(&tma_out);
    tc::prefetch_tmap(&tma_out_b);
  }
  if (warp == 1) { tmem_alloc2(&s_tmem_base, 512); tmem_relinquish2(); }
  if (!args.early) pdl_wait();          // the tables below may come from the kernel right before
  // Tile list: a thread for each group. Groups with more tokens come first, as their tiles take longer: a launch then ends with
  // the shortest tiles, and the pairs finish together (16 groups of 4096 tokens on average and up to
  // three times as many, 2048 x 768: 164 -> 146 us).
  // The keys lie in the epilogue's slabs, which ordinary stores write first: in the ring, the first TMA loads would follow ordinary accesses
  // to the same bytes with no proxy fence between them.
  int* s_key = reinterpret_cast<int*>(smem + (size_t)kRing * kStageBytes);
  static_assert(kMaxGroups * sizeof(int) <= (size_t)kEpiWarps * 2 * kSlabBytes, "keys of all groups");
  bool act = false;
  const int tg = threadIdx.x;
  int beg, rows, units;
  group_rows(args, s_key, beg, rows, units);
  if (tg < kMaxGroups) {
    int key = -1;
    if (tg < G) {
      s_cu[tg] = beg; s_units[tg] = units;
      if (tg == G - 1) s_total = beg + rows;
      act = tg >= args.g_begin && tg < args.g_end && (rows > 0 || (!args.accumulate && tg < args.zero_empty_below));
      if (act) key = units * 256 + (255 - tg);
    }
    s_key[tg] = key;
  }
  const int nact = __syncthreads_count(act ? 1 : 0);
  if (act) s_act[rank_of(s_key[tg], s_key, G)] = (unsigned char)tg;
  tc::fence_before_sync();
  __syncthreads();
  cluster_sync();                       // both CTAs' barriers exist before anyone touches the peer's
  tc::fence_after_sync();
  const uint32_t tmem_base = s_tmem_base;
  const int ntiles = nact * (args.M_w / 256) * (args.N / 256);
  const bool dyn = args.sched != nullptr;

  auto fail = [&](int site, int tile) {
    if (atomicCAS(&args.status[0], 0, MEP_ERR_MBAR_TIMEOUT) == 0) {
      args.status[1] = 100 + site; args.status[2] = blockIdx.x; args.status[3] = tile;
      if (args.status_host) { *(volatile int32_t*)args.status_host = MEP_ERR_MBAR_TIMEOUT; __threadfence_system(); }
    }
    s_abort = 1;
  };
  // Row blocks vary fastest, all of them or, where groups are large on average, in bands of at most 8: 74 pairs then read few
  // distinct slabs of a group that L2 does not hold (8 groups of 4096 tokens, 7168 x 2048: 0.817 -> 0.793 ms, with the SGD
  // epilogue 0.806 -> 0.771). With 1024 tokens a group's rows stay in L2 anyway, and the epilogue's updates take 1 % longer in bands.
  // The mean is over all G groups; a layer passes its slots for replicas too, which are empty on one rank, and there its
  // experts have to average 36 MB.
  const int bands = (int64_t)s_total * args.M_w > (int64_t)G * kBandElems ? (args.M_w / 256 + 7) / 8 : 1;
  const int mblk = args.M_w / 256, nblk = args.N / 256, bw = (mblk + bands - 1) / bands;
  const Divisor by_group(mblk * nblk), by_band(bw * nblk), by_row(bw), by_last(mblk - (bands - 1) * bw);
  auto get_tile = [&](int t, Tile& ti) {
    const int ai = by_group(t), local = t - ai * by_group.b, band = by_band(local), in = local - band * by_band.b;
    const Divisor& rows = band + 1 == bands ? by_last : by_row;
    const int nb = rows(in), g = s_act[ai];
    ti.g = g; ti.row0 = s_cu[g]; ti.ksteps = 2 * s_units[g]; ti.kblocks = (ti.ksteps + 3) >> 2;
    ti.m0 = (band * bw + in - nb * rows.b) * 256; ti.n0 = nb * 256;
  };

  if (warp == 0) {
    // ---------------- TMA producer: this CTA's halves; bytes are counted on the LEADER's barrier. The whole warp runs the
    // loop and one elected lane issues (see grouped_gemm_pair.cu).
    Tile ti;
    uint32_t s = 0, ph = 0;
    bool any = false, ready = true;      // ready: the stage is known to be free
    tq::Scheduler<true> sched; tq::Consumer<true> follow;
    if (dyn && lane == 0) { if (leader) sched.setup(&s_ring, args.sched, ntiles); else follow.setup(&s_ring); }
    tq::Snake seq(pair, npairs, ntiles);
    const uint32_t smem0 = smem_u32(smem), full0 = mapa(smem_u32(&full_bar[0]), 0);
    if (args.early) pdl_wait();
    for (;;) {
      int t = -1;
      if (!dyn) { if (!s_abort) t = seq.next(); }
      else if (lane == 0 && !s_abort) { t = leader ? sched.next(args.budget_ns) : follow.next(args.budget_ns); if (t == -2) fail(5, -1); }
      t = __shfl_sync(0xffffffffu, t, 0);
      if (t < 0) break;
      get_tile(t, ti);
      const int am = ti.m0 + (int)cr * 128, bn = ti.n0 + (int)cr * 128;
      for (int kb = 0; kb < ti.kblocks; ++kb) {
        if (!__all_sync(0xffffffffu, ready) && !__all_sync(0xffffffffu, mbar_wait_compact(&empty_bar[s], ph ^ 1u, args.budget_ns))) { if (lane == 0) fail(1, t); break; }
        const uint32_t sn = s + 1 == kRing ? 0u : s + 1, phn = sn ? ph : ph ^ 1u;
        ready = mbar_test(&empty_bar[sn], phn ^ 1u);
        if (elect_one()) {
          const uint32_t sa = smem0 + s * kStageBytes, bar = full0 + s * 8u;
          const int k = ti.row0 + kb * kBK;
          if (leader) mbar_expect_tx(&full_bar[s], 2 * kStageBytes);     // both CTAs' bytes
          // one 2-D box for each 64-column atom: with one 3-D box for both, launches of short groups that store their gradients were
          // slower (64 groups of 256 tokens, 2048 x 1536: 212 us, with these 200), deep ones the same
          tma_load_2d_bar(sa, &tma_a, am, k, bar);
          tma_load_2d_bar(sa + kAtomBytes, &tma_a, am + 64, k, bar);
          tma_load_2d_bar(sa + kHalfBytes, &tma_b, bn, k, bar);
          tma_load_2d_bar(sa + kHalfBytes + kAtomBytes, &tma_b, bn + 64, k, bar);
        }
        __syncwarp();
        any = true;
        s = sn; ph = phn;
      }
    }
    if (leader && any) mbar_wait_compact(&full_bar[s ? s - 1 : kRing - 1], s ? ph : ph ^ 1u, args.budget_ns);     // no copy outlives the pair
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only): one instruction drives both SMs. The whole warp runs the loop so
    // that stage, phase and descriptors are warp-uniform (see grouped_gemm_pair.cu); one elected lane issues.
    if (leader) {
      constexpr uint32_t idesc = tc::instr_desc_bf16(256, 256, true, true);
      const uint64_t adesc0 = tc::smem_desc(smem_u32(smem), kAtomBytes, 1024), bdesc0 = tc::smem_desc(smem_u32(smem) + kHalfBytes, kAtomBytes, 1024);
      int tcnt = 0; Tile ti;
      uint32_t stage = 0, phase = 0;
      bool ready = false;
      tq::Consumer<true> tiles; tiles.setup(&s_ring);
      tq::Snake seq(pair, npairs, ntiles);
      if (args.early) pdl_wait();       // its waits have their limit from when the operands may come
      for (;; ++tcnt) {
        int t = -1;
        if (!dyn) { if (!s_abort) t = seq.next(); }
        else if (lane == 0 && !s_abort) { t = tiles.next(args.budget_ns); if (t == -2) fail(6, tiles.n); }
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t < 0) break;
        get_tile(t, ti);
        if (ti.kblocks == 0) { --tcnt; continue; }
        const int acc = tcnt & 1; const uint32_t aph = (uint32_t)(tcnt >> 1) & 1u;
        if (!__all_sync(0xffffffffu, mbar_wait_compact(&tempty_bar[acc], aph ^ 1u, args.budget_ns))) { if (lane == 0) fail(2, t); break; }
        tc::fence_after_sync();
        const uint32_t d_tmem = tmem_base + (uint32_t)acc * 256;
        bool ok = true;
        for (int kb = 0; kb < ti.kblocks; ++kb) {
          if (!__all_sync(0xffffffffu, ready) && !__all_sync(0xffffffffu, mbar_wait_compact(&full_bar[stage], phase, args.budget_ns))) {
            if (lane == 0) fail(3, t);
            ok = false; break;
          }
          const uint32_t sn = stage + 1 == kRing ? 0u : stage + 1, phn = sn ? phase : phase ^ 1u;
          ready = mbar_test(&full_bar[sn], phn);
          tc::fence_after_sync();
          const int steps = ti.ksteps - 4 * kb;
          if (elect_one()) {
            const uint64_t ad = adesc0 + stage * (kStageBytes >> 4), bd = bdesc0 + stage * (kStageBytes >> 4);
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              if (k < steps) mma2_bf16(d_tmem, ad + k * (2048 >> 4), bd + k * (2048 >> 4), idesc, (kb | k) ? 1u : 0u);
            mma2_commit_both(smem_u32(&empty_bar[stage]));
          }
          __syncwarp();
          stage = sn; phase = phn;
        }
        if (!ok) break;
        if (elect_one()) mma2_commit_both(smem_u32(&tfull_bar[acc]));
        __syncwarp();
      }
    }
  } else {
    // ---------------- epilogue: this CTA's 128 rows of the 256-row tile
    const int q = warp & 3, half = (warp - 2) >> 2;
    const uint32_t stg = smem_u32(smem + (size_t)kRing * kStageBytes) + (uint32_t)(warp - 2) * 2 * kSlabBytes;
    const uint32_t tempty_leader[2] = {mapa(smem_u32(&tempty_bar[0]), 0), mapa(smem_u32(&tempty_bar[1]), 0)};
    // Gradients are not read before the launch ends: with their lines first in line to leave L2, short groups, whose operands are
    // read again for every tile, took 550 us instead of 635 (48 groups of 256 tokens, 7168 x 2048), deep ones the same.
    const uint64_t streamed = tc::evict_first();
    if (args.early) pdl_wait();         // gradients and weights are written from here, and the kernel before may read them
    int tcnt = 0, chunk_no = 0; Tile ti;
    tq::Consumer<true> tiles; tiles.setup(&s_ring);
    tq::Snake seq(pair, npairs, ntiles);
    for (;; ++tcnt) {
      int t = -1;
      if (!dyn) { if (!s_abort) t = seq.next(); }
      else {
        if (lane == 0 && !s_abort) { t = tiles.next(args.budget_ns); if (t == -2) fail(7, tiles.n); }
        t = __shfl_sync(0xffffffffu, t, 0);
      }
      if (t < 0) break;
      get_tile(t, ti);
      const int orow0 = ti.g * args.M_w + ti.m0 + (int)cr * 128 + q * 32;
      const int pitch = args.n_each ? args.n_each : args.N;        // one launch may compute two matrices side by side
      const bool b = ti.n0 >= pitch;
      const int ocol0 = b ? ti.n0 - pitch : ti.n0;
      // optimizer in the epilogue: this group's weights are updated in place and no gradient is written
      const bool upd = args.upd_mask != nullptr && args.upd_mask[ti.g] != 0;
      if (ti.kblocks == 0) {           // empty group that must end with a zero gradient (nothing to update)
        if (!upd) {
          // whole 512-byte runs: with a lane per row this path ran at a third of the HBM rate
          float4* o = reinterpret_cast<float4*>((float*)(b ? args.out_b : args.out) + (size_t)orow0 * pitch + ocol0 + half * 128) + lane;
          for (int r = 0; r < 32; ++r) __stcs(o + (size_t)r * (pitch / 4), make_float4(0.f, 0.f, 0.f, 0.f));
        }
        --tcnt; continue;
      }
      // A chunk is 32 rows x 32 columns. The accumulator arrives with lane = row; the weights are read and
      // written with four lanes per row instead (16 bytes each, eight rows per instruction: whole sectors),
      // so the chunk takes the same trip through the warp's shared-memory slab as a stored gradient does.
      const __nv_bfloat16* wbase = upd ? (const __nv_bfloat16*)(b ? args.upd_w_b : args.upd_w) + (size_t)orow0 * pitch + ocol0 + (half * 4) * 32 : nullptr;
      auto wptr = [&](int i, int k) {
        return const_cast<__nv_bfloat16*>(wbase) + (size_t)((lane >> 2) + 8 * k) * pitch + i * 32 + (lane & 3) * 8;
      };
      int4 wv[4][4];
      if (upd) {                       // the tile's weights (this warp's 32 x 128 part): in flight while its MMAs finish
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int k = 0; k < 4; ++k) wv[i][k] = *reinterpret_cast<const int4*>(wptr(i, k));
      }
      const int acc = tcnt & 1; const uint32_t aph = (uint32_t)(tcnt >> 1) & 1u;
      int ok = 1;
      if (lane == 0) ok = mbar_wait_compact(&tfull_bar[acc], aph, args.budget_ns) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) { if (lane == 0) fail(4, t); break; }
      tc::fence_after_sync();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)acc * 256;
      // software pipeline over the four 32-column chunks of this warp: the TMEM load of chunk i+1 is
      // in flight while chunk i goes through shared memory; the accumulator is handed back to the
      // MMA warp as soon as the last chunk sits in registers
      uint32_t r[2][32];
      tc::tmem_ld32(taddr + (half * 4) * 32, r[0]);
#pragma unroll
      for (int i = 0; i < 4; ++i, ++chunk_no) {
        const int c = half * 4 + i;
        tc::tmem_ld_wait();
        if (i + 1 < 4) {
          tc::tmem_ld32(taddr + (c + 1) * 32, r[(i + 1) & 1]);
        } else {
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) remote_arrive(tempty_leader[acc]);
        }
        if (upd) {
          const uint32_t ubuf = stg + (uint32_t)(chunk_no & 1) * kSlabBytes;
          if (lane == 0) bulk_wait_read<0>();      // a gradient stored from this slab earlier has left it
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            tc::st_shared_v4(ubuf + lane * 128 + ((j ^ (lane & 7)) << 4), r[i & 1][4 * j], r[i & 1][4 * j + 1], r[i & 1][4 * j + 2], r[i & 1][4 * j + 3]);
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int R = (lane >> 2) + 8 * k, p2 = (lane & 3) * 2;
            const int4 g0 = tc::ld_shared_v4(ubuf + R * 128 + ((p2 ^ (R & 7)) << 4));
            const int4 g1 = tc::ld_shared_v4(ubuf + R * 128 + (((p2 + 1) ^ (R & 7)) << 4));
            const float gg[8] = {__int_as_float(g0.x), __int_as_float(g0.y), __int_as_float(g0.z), __int_as_float(g0.w),
                                 __int_as_float(g1.x), __int_as_float(g1.y), __int_as_float(g1.z), __int_as_float(g1.w)};
            int4 x = wv[i][k];
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&x);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float2 f = __bfloat1622float2(h[e]);
              f.x = fmaf(-args.upd_lr, gg[2 * e], f.x);           // as in sgd_kernel
              f.y = fmaf(-args.upd_lr, gg[2 * e + 1], f.y);
              h[e] = __floats2bfloat162_rn(f.x, f.y);
            }
            *reinterpret_cast<int4*>(wptr(i, k)) = x;
          }
          continue;
        }
        const uint32_t buf = stg + (uint32_t)(chunk_no & 1) * kSlabBytes;
        if (lane == 0) bulk_wait_read<1>();
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          tc::st_shared_v4(buf + lane * 128 + ((j ^ (lane & 7)) << 4), r[i & 1][4 * j], r[i & 1][4 * j + 1], r[i & 1][4 * j + 2], r[i & 1][4 * j + 3]);
        tc::fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (args.accumulate) tc::tma_reduce_add_2d(b ? &tma_out_b : &tma_out, buf, ocol0 + c * 32, orow0);
          else tc::tma_store_2d(b ? &tma_out_b : &tma_out, buf, ocol0 + c * 32, orow0, streamed);
          bulk_commit();
        }
      }
    }
    if (lane == 0) bulk_wait_all<0>();
  }

  // ---------------- teardown: nobody leaves while the peer may still signal into this CTA
  tc::fence_before_sync();
  __syncthreads();
  cluster_sync();
  tc::fence_after_sync();
  if (warp == 1) tmem_dealloc2(tmem_base, 512);
  if (leader && threadIdx.x == 0) tq::scheduler_done(args.sched, pair == 0 ? 2 + args.sched_odd : 2, args.sched_ctas > 0 ? args.sched_ctas : (int)gridDim.x);
}

}  // namespace w2

}  // namespace mep

// dW[g] (+)= X_g^T dY_g on CTA pairs. x: [rows, M_w] bf16 (pitch x_ld), dy: [rows, N] bf16 (pitch dy_ld),
// args.out: fp32 [G, M_w, N]. Requires M_w % 256 == 0, N % 256 == 0 and an even CTA count.
extern "C" int mep_grouped_wgrad_2cta(const void* x, int64_t rows, int64_t x_ld, const void* dy, int64_t dy_ld,
                                      const mep::GemmArgs* args_in, int num_ctas, cudaStream_t stream) {
  using namespace mep;
  GemmArgs args = *args_in;
  MEP_REQUIRE(args.G >= 1 && args.G <= w2::kMaxGroups, "wgrad: G=%d out of range", args.G);
  MEP_REQUIRE(args.M_w % 256 == 0 && args.N % 256 == 0, "wgrad (2-CTA): weight shape [%d,%d] must be multiples of 256", args.M_w, args.N);
  num_ctas = pair_ctas(&args, num_ctas);
  MEP_REQUIRE(num_ctas >= 2, "wgrad (2-CTA): needs at least two CTAs");
  MEP_REQUIRE(args.n_each == 0 || (args.N == 2 * args.n_each && args.n_each % 256 == 0 && args.out_b), "wgrad (2-CTA): two matrices of %d columns in %d", args.n_each, args.N);
  MEP_REQUIRE(!args.upd_mask || (args.upd_w && (!args.n_each || args.upd_w_b)), "wgrad (2-CTA): an update without the weights of every matrix");
  const int pitch = args.n_each ? args.n_each : args.N;
  CUtensorMap ma, mb, mo, mo_b;
  if (tmap_rows(&ma, x, rows, args.M_w, x_ld, 64, 64)) return -1;
  if (tmap_rows(&mb, dy, rows, args.N, dy_ld, 64, 64)) return -1;
  if (tmap_rows(&mo, args.out, (int64_t)args.G * args.M_w, pitch, pitch, 32, 32, true)) return -1;
  if (!args.n_each) mo_b = mo;
  else if (tmap_rows(&mo_b, args.out_b, (int64_t)args.G * args.M_w, pitch, pitch, 32, 32, true)) return -1;
  if (allow_smem((const void*)w2::wgrad_2cta_kernel, w2::kSmem)) return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(num_ctas); cfg.blockDim = dim3(w2::kThreads); cfg.dynamicSmemBytes = w2::kSmem; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = args.pdl ? 2 : 1;
  MEP_CUDA_CHECK(cudaLaunchKernelEx(&cfg, w2::wgrad_2cta_kernel, ma, mb, mo, mo_b, args));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return 0;
}

