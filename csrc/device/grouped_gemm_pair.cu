// Token-major grouped GEMMs on CTA pairs (tcgen05.mma.cta_group::2): GATE_UP, DOWN, DGRAD, DGRAD_GU.
//
// A pair computes out^T: the 256 rows of an MMA tile are WEIGHT columns (128 per CTA) and its N side is up to 256
// token rows of ONE expert (half of them staged by each CTA). Three things follow.
//   * A tile never straddles experts although groups are only multiples of 128 rows (with tokens on the M side, a pair
//     wastes half a tile for every group with an odd number of 128-row blocks), and N takes the group's real size in
//     steps of 32: padding rows cost nothing when the caller passes their table (GemmArgs.pad_rows).
//   * A CTA fills 32 KB of shared memory per 64-deep k-block for the math of a 128 x 256 x 64 block; a single CTA
//     needs 48 KB. The kernels run at the board's power limit, where the bytes that move through L2 per FLOP
//     set the clock as well.
//   * The accumulator arrives transposed. It is read in MMA-fragment layout and turned by stmatrix.trans on its way
//     into 128-byte swizzled staging rows, from where TMA stores (or, for the push epilogue, 16-byte peer stores)
//     write whole 128-byte runs of token rows.
// Roles per CTA: warp 0 = TMA producer, warp 1 = TMEM allocation (+ MMA issue in the leader), warps 2-9 = epilogue: TMEM
// lane quarter = warp % 4, the two sets of four take alternate 16-token chunks.
// GATE_UP: the M side of a CTA is 64 gate columns and the same 64 up columns, so g and u of an output sit 64 TMEM
// lanes apart: the up warps hand their fp32 fragments to the gate warps through shared memory.
#include "pair.cuh"
#include "tile_queue.cuh"
#include "gemm_args.h"
#include "tmap.h"
#include "silu.cuh"

namespace mep {
namespace tp {
using namespace pair;

constexpr int kBK = 64, kEpiWarps = 8, kThreads = 64 + 32 * kEpiWarps;
constexpr int kWBytes = 128 * kBK * 2;                 // 16 KB: a CTA's weight columns of one k-block
constexpr int kRingBytes = 6 * 2 * kWBytes, kMaxRing = 10;     // a stage is 18 KB at least
constexpr int kAtomBytes = 64 * kBK * 2;
constexpr int kChunk = 16;                             // tokens per epilogue step
constexpr int kStgBytes = kChunk * 128;                // staging: 16 tokens x 64 columns
constexpr int kXchBytes = 32 * 32;                     // half of a warp's fp32 fragments of a chunk (GATE_UP)
constexpr int kMaxGroups = 192;
// BANDED: a group with more than kXBytes of token rows is walked in bands of at most kBand token tiles, all weight columns for
// a band, then the next band. 74 pairs then read 8 + 9 operand slabs at a time and fetch each token row from DRAM once; DRAM
// traffic also costs clock, the kernels being at the power limit. One group of 32768 tokens, 7168 x 2048: gate/up 1.85 ->
// 1.55 ms, down 0.91 -> 0.74; groups of 4000, 4096 x 1024: gate/up 0.471 -> 0.440, dgrad 0.237 -> 0.226. Below the line the
// weights would be read again for nothing (4096 tokens, 4096 deep, 32 MB: 1.445 -> 1.481).
constexpr int kBand = 8, kXBytes = 36 << 20;
// Up to this many rounds of tiles over the pairs, groups with larger tiles come first, so that the launch ends with the shortest and the pairs
// finish together; with more rounds the groups keep their order. Forward passes in long loops, in us, never sorted / by this rule: 1531 tokens,
// 2048 x 768, 16 experts (5 and 6 rounds) 147.1 / 143.6; 1000, 7168 x 512, 32 (2 and 16) 285.3 / 278.6; 1000, 4096 x 1024, 24 (5 and 9) 254.1 /
// 251.7. Always sorted / by this rule: 4096, 7168 x 2048, 32 (31 and 54) 2669 / 2619, a captured training step of it 8990 / 8800; from 8 to
// 24 rounds the two are within 1 % of each other. Every round runs forwards: backwards in odd ones, the pairs that the hardware starts last
// had the tiles left over in a short last round (64 tokens, 2048 x 768, two rounds, 57.4 / 51.7).
constexpr int kSortRounds = 12;
// STREAM: weights of a group with one token tile are read once: their lines leave L2 first, so that rows, tables and above all the kernels' code, which
// every launch fetches anew, stay there. Its stages are 128 deep: one load brings a column atom's weights of both k-blocks and one pair of barriers
// serves them. What a round that does not fill the GPU takes is the producer's issue (about 450 cycles a k-block and 58 GB/s per SM before). Not for
// tiles that share weights, as pairs are not in step: gate/up of 32 experts and 4096 tokens x 8, 7168 x 2048, then reads 6.2 GB instead of 3.4 and takes 2.04
// ms instead of 1.80. Without / with, in us:
//   rows of an expert                                        32            64           128           192           256           384           512
//   2048 x 768, 16 experts, forward                 46.9 / 44.2   53.2 / 47.3   57.1 / 54.6   62.8 / 61.6   69.4 / 69.4   82.9 / 84.1  100.0 / 102.3
//   (two layers in turn)    both dgrads             45.3 / 42.9   47.1 / 43.1   51.3 / 48.7   60.1 / 57.9   61.6 / 62.6   75.9 / 78.0   87.1 / 89.6
//   4096 x 1536, 32 experts, forward                 211 / 200     222 / 208     253 / 249     309 / 301     362 / 353     479 / 502     605 / 606
//   rows of an expert, captured steps                        96           112           128           144           160
//   4096 x 1536, 32 experts                         1015 / 1008   1026 / 1016   1037 / 1028   1069 / 1069   1080 / 1089
//   with the update in the epilogue                 1166 / 1158   1179 / 1165   1213 / 1198   1220 / 1232   1238 / 1261
//   7168 x 2048, 32 experts                         2196 / 2193   2212 / 2215   2286 / 2239   2391 / 2381   2477 / 2474
//   with the update in the epilogue                 2466 / 2466   2487 / 2473   2496 / 2500   2533 / 2543   2567 / 2577
// kStreamRows: so many rows (without padding) a group that holds any has at most on average. A direct call counts the rows of `a`, which may have room for more
// (kStreamRoom): dgrads of 16 groups of 66, 2048 x 768, in a table of 320 rows for each 47.3 / 43.1.
// kStreamBytes: those groups' matrices, one for each. A smaller layer whose forward pass is called over and over keeps its weights in L2: 2048 x 768, 8 experts
// (24 MiB), 32 and 128 rows 31.8 / 31.4 and 39.9 / 41.7, 1536 x 1024, 10 (30 MiB), 10 rows 33.7 / 35.2; captured steps with the update in the epilogue, dgrads
// of 512 x 1024, 19 (19 MiB), 116 rows 120.6 / 123.1, 512 x 1280, 17 (21 MiB), 16 rows 107.2 / 105.5. Half of it for a layer's
// launches that do not start early (kStreamBytesLate): nobody has loaded their first weights for them. Passes issued from Python, 2048 x 768, 8 experts:
// backward, 4 and 64 rows 88.4 / 83.9 and 95.9 / 88.2, forward, 64 rows 38.2 / 37.1.
constexpr int64_t kStreamBytes = 32 << 20, kStreamBytesLate = 16 << 20, kStreamRows = 128, kStreamRoom = 320;
enum Kind { PLAIN, BANDED, STREAM };                   // a kernel each: code that a launch does not need costs it 1 to 2 us of 50
constexpr int kStgSet = 4 * kStgBytes;                 // GATE_UP: act twice, gate, up; else: two buffers for each 64-column side
constexpr size_t kEpiBytes = 2 * kStgSet + kEpiWarps * kXchBytes;
constexpr size_t kSmem = (size_t)kRingBytes + kEpiBytes + 1024;

struct Tile { int g, row0, n, n0; bool once; };        // n tokens from row0 (a multiple of 32, at most 256); all of their group's

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// a / b for a >= 0, b > 0 and results below 2^20, without the code of an integer division: __fdividef is off by 2 ulp at
// most, so the quotient by one at most.
__device__ __forceinline__ int quotient(int a, int b) {
  const int q = (int)__fdividef((float)a + 0.5f, (float)b), r = a - q * b;
  return q + (r >= b) - (r < 0);
}

// Bounded poll of a ready flag (see GemmArgs.tile_done / group_flags); SYS: written by another GPU.
template <bool SYS>
__device__ __forceinline__ bool wait_flag(const uint32_t* flag, uint32_t epoch, uint64_t budget_ns) {
  auto up = [&] { return (int32_t)((SYS ? ld_acquire_sys(flag) : ld_acquire_gpu(flag)) - epoch) >= 0; };
  if (up()) return true;
  const long long t0 = clock64(), lim = budget_cycles(budget_ns);
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 32; ++i) { __nanosleep(SYS ? 200 : 100); if (up()) return true; }
    if (clock64() - t0 > lim) return false;
  }
}

template <int MODE, int KIND>
__global__ void __launch_bounds__(kThreads, 1)
tok_pair_kernel(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_x64,
                const __grid_constant__ CUtensorMap tma_x16, const __grid_constant__ CUtensorMap tma_w0, const __grid_constant__ CUtensorMap tma_w1,
                const __grid_constant__ CUtensorMap tma_out, const __grid_constant__ CUtensorMap tma_out2, GemmArgs args) {
  constexpr bool W_MN = MODE == GEMM_GATE_UP || MODE == GEMM_DOWN;      // weights [k, column]: the M side is contiguous
  constexpr int kCols = MODE == GEMM_GATE_UP ? 128 : 256;               // output columns of a tile
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[kMaxRing], empty_bar[kMaxRing], tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t s_tmem_base;
  __shared__ volatile int s_abort;
  __shared__ tq::Ring s_ring;
  // groups in the order of the tile list: number, first row, 32-token units, first tile; what they are ordered by
  __shared__ int s_grp[kMaxGroups], s_beg[kMaxGroups], s_units[kMaxGroups], s_start[kMaxGroups + 1];
  __shared__ __align__(16) int s_key[kMaxGroups];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cr = cluster_ctarank();
  const bool leader = cr == 0;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  __shared__ float s_scale[2][2][128];   // [set][accumulator]: row factors of the set's chunks
  __shared__ int s_half;                 // most token rows a CTA stages for a tile of this launch
  constexpr int kSub = KIND == STREAM ? 2 : 1;           // 64-deep k-blocks of a stage
  const int G = args.G, kblocks = args.K / (kSub * kBK);
  pdl_trigger();

  if (warp == 1) {
    tmem_alloc2(&s_tmem_base, 512); tmem_relinquish2();
  } else if (threadIdx.x == 64) {
    s_abort = 0;
    for (int i = 0; i < kMaxRing; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&tfull_bar[i], 1); mbar_init(&tempty_bar[i], 2 * kEpiWarps); }
    tq::init(&s_ring, 2 * kEpiWarps + 2);      // both CTAs' epilogue warps, the MMA issuer, the peer's producer
    fence_mbar_init();
  } else if (threadIdx.x == 96) {
    tc::prefetch_tmap(&tma_x); tc::prefetch_tmap(&tma_x64); tc::prefetch_tmap(&tma_x16); tc::prefetch_tmap(&tma_w0); tc::prefetch_tmap(&tma_w1);
    tc::prefetch_tmap(&tma_out); tc::prefetch_tmap(&tma_out2);
  }
  if (!args.early) pdl_wait();           // the tables below may come from the kernel right before
  // Tile list: a thread for each group. Groups are ordered by the size of their tiles where the launch has few of them (see kSortRounds) --
  // unless the rows or weights are still arriving, in the order of the groups. A key: size, group, number of token tiles.
  const int few = kSortRounds * ((args.sched_ctas > 0 ? args.sched_ctas : (int)gridDim.x) >> 1);      // alike for all launches on one ticket
  const int tg = threadIdx.x;
  int units, beg, rows, key = 0;
  group_rows(args, s_key, beg, rows, units);
  if (tg < kMaxGroups) {
    if (tg < G) {
      if (tg < args.g_begin || tg >= args.g_end) units = 0;
      const int mt = (units + 7) >> 3;
      key = ((units && !args.tile_done && !args.group_flags ? (units + mt - 1) / mt : 0) * 256 + (255 - tg)) << 16 | min(mt, 0xffff);
    }
    s_key[tg] = key;
  }
  __syncthreads();
  if (tg < G) {
    int tiles = 0;
    const int place = rank_of(key, s_key, G, &tiles), at = (int64_t)tiles * (args.N / kCols) > few ? tg : place;
    s_grp[at] = tg; s_beg[at] = beg; s_units[at] = units;
  }
  __syncthreads();
  if (warp == 0) {                       // first tile of each: 32 groups at a time
    const int nblk = args.N / kCols;
    int run = 0, most = 0;
    for (int g0 = 0; g0 < G; g0 += 32) {
      const int i = g0 + lane, u = i < G ? s_units[i] : 0;
      const int mt = (u + 7) >> 3, tiles = mt * nblk, incl = warp_incl_scan(tiles);
      if (u) most = max(most, (u + mt - 1) / mt);
      if (i < G) s_start[i] = run + incl - tiles;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    if (lane == 0) { s_start[G] = run; s_half = 16 * most; }
  }
  tc::fence_before_sync();
  __syncthreads();
  cluster_sync();                        // both CTAs' barriers exist before anyone touches the peer's
  tc::fence_after_sync();
  const uint32_t tmem_base = s_tmem_base;
  const int ntiles = s_start[G];
  const bool dyn = args.sched != nullptr;
  // Token rows arrive in one box of 128 or 64, or in boxes of 16 where no tile of the launch has more than 48 for a CTA: a stage is then
  // little more than its weights and up to ten fit instead of six. With few tokens per expert the kernel streams
  // weights, and what an SM has in flight is its bandwidth.
  const bool small = s_half <= 48;
  const uint32_t x_bytes = small ? max(s_half, 16) * 128u : s_half <= 64 ? 8192u : 16384u;
  const uint32_t stage_bytes = kSub * (((uint32_t)kWBytes + x_bytes + 1023u) & ~1023u);
  const uint32_t nstages = min((uint32_t)kMaxRing, (uint32_t)kRingBytes / stage_bytes);

  auto note = [&](int site, int tile, int code) {
    if (atomicCAS(&args.status[0], 0, code) == 0) {
      args.status[1] = 200 + site; args.status[2] = blockIdx.x; args.status[3] = tile;
      if (args.status_host) { *(volatile int32_t*)args.status_host = code; __threadfence_system(); }
    }
  };
  auto fail = [&](int site, int tile, int code = MEP_ERR_MBAR_TIMEOUT) { note(site, tile, code); s_abort = 1; };
  // tile number -> tile; `g` is a monotone cursor over the ordered groups. The tiles of a group share its tokens evenly (in units of 32), token
  // tiles vary fastest: the weight columns they have in common are then in L2 (within a band, see kBand).
  auto get_tile = [&](int t, int& g, Tile& ti) {
    while (s_start[g + 1] <= t) ++g;
    const int units = s_units[g], mt = (units + 7) >> 3, local = t - s_start[g];
    int cb, pt;
    if (KIND == BANDED && (int64_t)mt * args.K > kXBytes / 512) {
      const int nblk = args.N / kCols, bands = quotient(mt - 1, kBand) + 1, bw = quotient(mt - 1, bands) + 1;
      const int b = quotient(local, bw * nblk), in = local - b * bw * nblk, w = min(bw, mt - b * bw);
      cb = quotient(in, w); pt = b * bw + in - cb * w;
    } else {
      cb = local / mt; pt = local - cb * mt;
    }
    const int base = units / mt, rem = units - base * mt;
    ti.g = s_grp[g]; ti.n0 = cb * kCols;
    ti.row0 = s_beg[g] + 32 * (pt * base + min(pt, rem));
    ti.n = 32 * (base + (pt < rem ? 1 : 0));
    ti.once = mt == 1;
  };

  if (warp == 0) {
    // ---------------- TMA producer: this CTA's halves; bytes are counted on the LEADER's barrier. Like the MMA issuer the
    // whole warp runs the loop and one elected lane issues: with a single diverged thread a k-block cost 640 cycles of
    // issue alone, which held an SM to 46 GB/s of weights and the tensor cores to 80 % of their rate.
    int gcur = 0; Tile ti;
    uint32_t s = 0, ph = 0;
    bool any = false, ready = true;      // ready: the stage is known to be free
    bool early = args.early != 0;        // the kernel before has not been waited for yet
    tq::Scheduler<true> sched; tq::Consumer<true> follow;
    if (dyn && lane == 0) { if (leader) sched.setup(&s_ring, args.sched, ntiles); else follow.setup(&s_ring); }
    tq::Strided seq{pair, npairs, ntiles};
    const uint32_t tile_ep = args.tile_done ? *(volatile const uint32_t*)args.tile_epoch : 0u;
    const uint32_t group_ep = args.group_flags ? *(volatile const uint32_t*)args.group_epoch : 0u;
    const uint64_t streamed = tc::evict_first(), kept = tc::evict_normal();
    int seen_row = -1, seen_group = -1;              // flags known to be up: first row of the last tile, last group
    const uint32_t smem0 = smem_u32(smem), full0 = mapa(smem_u32(&full_bar[0]), 0);
    for (;;) {
      int t = -1;
      if (!dyn) { if (!s_abort) t = seq.next(); }
      else if (lane == 0 && !s_abort) { t = leader ? sched.next(args.budget_ns) : follow.next(args.budget_ns); if (t == -2) fail(5, -1); }
      t = __shfl_sync(0xffffffffu, t, 0);
      if (t < 0) break;
      get_tile(t, gcur, ti);
      int up = 1;
      if (args.tile_done && ti.row0 != seen_row) {
        // the rows come from a dispatch that may still be running: wait until they have all landed and the
        // duplicates are expanded, then order the TMA engine's reads behind that
        if (lane == 0)
          for (int b = ti.row0 >> 7; up && b <= (ti.row0 + ti.n - 1) >> 7; ++b) up = wait_flag<false>(args.tile_done + b, tile_ep, args.budget_ns) ? 1 : 0;
        seen_row = ti.row0;
      }
      if (args.group_flags && ti.g >= args.group_first && ti.g != seen_group) {
        // the weights of this group are a prefetched expert that may still be on its way
        if (lane == 0 && up) up = wait_flag<true>(args.group_flags + (ti.g - args.group_first), group_ep, args.budget_ns) ? 1 : 0;
        seen_group = ti.g;
      }
      if (args.tile_done || args.group_flags) {
        if (!__shfl_sync(0xffffffffu, up, 0)) { if (lane == 0) fail(9, t, MEP_ERR_FLAG_TIMEOUT); break; }
        __syncwarp();
        fence_proxy_async();
      }
      const int half = ti.n >> 1, xrow = ti.row0 + (int)cr * half, wrow = ti.g * args.b_group_rows;
      const uint32_t bytes = kSub * ((uint32_t)kWBytes + (small ? (uint32_t)half * 128u : half > 64 ? 16384u : 8192u));
      const uint64_t policy = ti.once ? streamed : kept;
      auto atoms = [&](uint32_t dst, const CUtensorMap* map, int k, int atom, uint32_t bar) {
        if (KIND == STREAM) tma_load_3d_bar(dst, map, 0, k, atom, bar, policy); else tma_load_3d_bar(dst, map, 0, k, atom, bar);
      };
      auto rows = [&](uint32_t dst, const CUtensorMap* map, int k, int row, uint32_t bar) {
        if (KIND == STREAM) tma_load_2d_bar(dst, map, k, row, bar, policy); else tma_load_2d_bar(dst, map, k, row, bar);
      };
      auto load_w = [&](int kb, uint32_t st) {
        const uint32_t sw = smem0 + st * stage_bytes, bar = full0 + st * 8u;
        const int k0 = kb * kSub * kBK;
        if (leader) mbar_expect_tx(&full_bar[st], 2 * bytes);
        if (MODE == GEMM_GATE_UP) {
          atoms(sw, &tma_w0, wrow + k0, ti.n0 / 64 + (int)cr, bar);
          atoms(sw + kSub * kAtomBytes, &tma_w1, wrow + k0, ti.n0 / 64 + (int)cr, bar);
        } else if (MODE == GEMM_DOWN) {
          atoms(sw, &tma_w0, wrow + k0, ti.n0 / 64 + 2 * (int)cr, bar);
        } else {
          const int kh = args.K / 2;               // DGRAD_GU: first half of K from Wg, second from Wu
#pragma unroll
          for (int i = 0; i < kSub; ++i) {
            const int k = k0 + i * kBK;
            if (MODE == GEMM_DGRAD_GU && k >= kh) rows(sw + i * kWBytes, &tma_w1, k - kh, wrow + ti.n0 + (int)cr * 128, bar);
            else rows(sw + i * kWBytes, &tma_w0, k, wrow + ti.n0 + (int)cr * 128, bar);
          }
        }
      };
      auto load_x = [&](int kb, uint32_t st) {
        const uint32_t bar = full0 + st * 8u;
#pragma unroll
        for (int j = 0; j < kSub; ++j) {
          const uint32_t sx = smem0 + st * stage_bytes + kSub * kWBytes + j * x_bytes;
          const int k0 = (kb * kSub + j) * kBK;
          if (small) {
            for (int i = 0; i < half; i += 16) tma_load_2d_bar(sx + i * 128, &tma_x16, k0, xrow + i, bar);
          } else if (half > 64) {
            tma_load_2d_bar(sx, &tma_x, k0, xrow, bar);
          } else {
            tma_load_2d_bar(sx, &tma_x64, k0, xrow, bar);
          }
        }
      };
      int kb = 0;
      if (early) {                         // fill the ring with weights, then wait for the rows
        const int pre = min((int)nstages, kblocks);
        if (elect_one()) for (int i = 0; i < pre; ++i) load_w(i, i);
        __syncwarp();
        pdl_wait();
        early = false;
        if (elect_one()) for (int i = 0; i < pre; ++i) load_x(i, i);
        __syncwarp();
        kb = pre; any = true;
        if (pre == (int)nstages) { s = 0; ph = 1; } else s = pre;
        ready = mbar_test(&empty_bar[s], ph ^ 1u);
      }
      for (; kb < kblocks; ++kb) {
        if (!__all_sync(0xffffffffu, ready) && !__all_sync(0xffffffffu, mbar_wait_compact(&empty_bar[s], ph ^ 1u, args.budget_ns))) { if (lane == 0) fail(1, t); break; }
        const uint32_t sn = s + 1 == nstages ? 0u : s + 1, phn = sn ? ph : ph ^ 1u;
        ready = mbar_test(&empty_bar[sn], phn ^ 1u);
        if (elect_one()) { load_w(kb, s); load_x(kb, s); }
        __syncwarp();
        any = true;
        s = sn; ph = phn;
      }
    }
    if (early) pdl_wait();               // whoever waits for this launch waits for the kernel before, too
    // the leader's last barrier phase covers both CTAs' copies: nobody leaves before it (cluster_sync below)
    if (leader && any) mbar_wait_compact(&full_bar[s ? s - 1 : nstages - 1], s ? ph : ph ^ 1u, args.budget_ns);
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only): one instruction drives both SMs. The whole warp runs the loop so
    // that stage, phase and descriptors are warp-uniform; one elected lane issues. With a single diverged thread the
    // loop took 673 cycles per k-block, 512 of which the tensor cores need.
    if (leader) {
      const uint32_t smem0 = smem_u32(smem);
      const uint64_t wdesc0 = W_MN ? tc::smem_desc(smem0, kSub * kAtomBytes, 1024) : tc::smem_desc(smem0, 16, 1024);
      const uint64_t xdesc0 = tc::smem_desc(smem0 + kSub * kWBytes, 16, 1024);
      constexpr uint32_t kWSub = (W_MN ? kAtomBytes : kWBytes) >> 4;
      constexpr uint32_t kWStep = W_MN ? 2048 >> 4 : 32 >> 4, kXStep = 32 >> 4;      // one 16-deep step in a descriptor's address field
      int tcnt = 0, gcur = 0; Tile ti;
      uint32_t stage = 0, phase = 0;
      bool ready = false;
      tq::Consumer<true> tiles; tiles.setup(&s_ring);
      tq::Strided seq{pair, npairs, ntiles};
      if (args.early) pdl_wait();       // no MMA can start before; the limits of its waits run from here, as everyone's do
      for (;; ++tcnt) {
        int t = -1;
        if (!dyn) { if (!s_abort) t = seq.next(); }
        else if (lane == 0 && !s_abort) { t = tiles.next(args.budget_ns); if (t == -2) fail(6, tiles.n); }
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t < 0) break;
        get_tile(t, gcur, ti);
        const uint32_t idesc = tc::instr_desc_bf16(256, 0, W_MN, false) | ((uint32_t)(ti.n >> 3) << 17);
        const int acc = tcnt & 1; const uint32_t aph = (uint32_t)(tcnt >> 1) & 1u;
        if (!__all_sync(0xffffffffu, mbar_wait_compact(&tempty_bar[acc], aph ^ 1u, args.budget_ns))) { if (lane == 0) fail(2, t); break; }
        tc::fence_after_sync();
        const uint32_t d_tmem = tmem_base + (uint32_t)acc * 256;
        bool ok = true;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!__all_sync(0xffffffffu, ready) && !__all_sync(0xffffffffu, mbar_wait_compact(&full_bar[stage], phase, args.budget_ns))) {
            if (lane == 0) fail(3, t);
            ok = false; break;
          }
          const uint32_t sn = stage + 1 == nstages ? 0u : stage + 1, phn = sn ? phase : phase ^ 1u;
          ready = mbar_test(&full_bar[sn], phn);
          tc::fence_after_sync();
          if (elect_one()) {
            const uint64_t wd = wdesc0 + stage * (stage_bytes >> 4), xd = xdesc0 + stage * (stage_bytes >> 4);
#pragma unroll
            for (int i = 0; i < kSub; ++i)
#pragma unroll
              for (int k = 0; k < kBK / 16; ++k)
                mma2_bf16(d_tmem, wd + i * kWSub + k * kWStep, xd + i * (x_bytes >> 4) + k * kXStep, idesc, (kb | i | k) ? 1u : 0u);
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
    // ---------------- epilogue: this CTA's 128 weight columns (TMEM lanes) of every token of the tile
    if (args.early) pdl_wait();
    const int q = warp & 3, set = (warp - 2) >> 2, side = q >> 1;      // side: TMEM lanes 0-63 or 64-127 = one 64-column staging row
    const uint32_t epi = smem_u32(smem + kRingBytes);
    const uint32_t tempty_leader[2] = {mapa(smem_u32(&tempty_bar[0]), 0), mapa(smem_u32(&tempty_bar[1]), 0)};
    const int set_tid = (warp - 2 - 4 * set) * 32 + lane;
    const bool issuer = lane == 0 && (q & 1) == 0;                      // one lane per (set, side) stores the staged rows
    const bool push = MODE != GEMM_GATE_UP && args.push_info != nullptr;
    // stmatrix: thread 8i + j addresses the 8-column block i of token row j; the 128-byte swizzle is xor by (row & 7)
    const uint32_t st_row = (uint32_t)(lane & 7) * 128, st_col = (uint32_t)((((q & 1) * 4 + (lane >> 3)) ^ (lane & 7)) << 4);
    int chunk_no = 0;
    int tcnt = 0, gcur = 0; Tile ti;
    tq::Consumer<true> tiles; tiles.setup(&s_ring);
    tq::Strided seq{pair, npairs, ntiles};
    auto stage = [&](uint32_t buf, const uint32_t* lo, const uint32_t* hi, float sc[4]) {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const uint32_t* l = lo + 4 * b; const uint32_t* h = hi + 4 * b;
        const float s0 = sc[2 * b], s1 = sc[2 * b + 1];
        st_matrix_x4_trans(buf + (uint32_t)b * 1024 + st_row + st_col,
                           pack2(__uint_as_float(l[0]) * s0, __uint_as_float(l[1]) * s1), pack2(__uint_as_float(l[2]) * s0, __uint_as_float(l[3]) * s1),
                           pack2(__uint_as_float(h[0]) * s0, __uint_as_float(h[1]) * s1), pack2(__uint_as_float(h[2]) * s0, __uint_as_float(h[3]) * s1));
      }
    };
    for (;; ++tcnt) {
      int t = -1;
      if (!dyn) { if (!s_abort) t = seq.next(); }
      else {
        if (lane == 0 && !s_abort) { t = tiles.next(args.budget_ns); if (t == -2) fail(7, tiles.n); }
        t = __shfl_sync(0xffffffffu, t, 0);
      }
      const int acc = tcnt & 1; const uint32_t aph = (uint32_t)(tcnt >> 1) & 1u;
      int ok = 0;
      float rs = 1.f;
      if (t >= 0) {
        get_tile(t, gcur, ti);
        const int i = ((set_tid >> 4) * 2 + set) * kChunk + (set_tid & 15);
        const bool scaled = (MODE == GEMM_GATE_UP || MODE == GEMM_DOWN) && args.row_scale && i < ti.n;
        // in flight while the tile's MMAs finish -- unless a dispatch may still be writing the factors together with the rows:
        // then only the finished MMAs, whose loads waited for the tile's flag, say that they are there
        if (scaled && !args.tile_done) rs = __ldcg(args.row_scale + ti.row0 + i);
        if (lane == 0) { ok = mbar_wait_compact(&tfull_bar[acc], aph, args.budget_ns) ? 1 : 0; if (!ok) fail(4, t); }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (scaled && args.tile_done) rs = __ldcg(args.row_scale + ti.row0 + i);
      }
      if (MODE == GEMM_GATE_UP || MODE == GEMM_DOWN) s_scale[set][acc][set_tid] = rs;
      // the warps of a set stage rows together: they go on or stop together
      if (!named_barrier_all(1 + 4 + set, 128, ok != 0)) break;
      tc::fence_after_sync();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)acc * 256;
      const int nchunks = ti.n / kChunk;
      const int col0 = ti.n0 + (int)cr * (kCols / 2) + (MODE == GEMM_GATE_UP ? 0 : side * 64);
      for (int c = set; c < nchunks; c += 2, ++chunk_no) {
        const int row = ti.row0 + c * kChunk;
        float sc[4] = {1.f, 1.f, 1.f, 1.f};          // row factors of this thread's four tokens
        if (MODE == GEMM_GATE_UP || MODE == GEMM_DOWN) {
          const float* f = &s_scale[set][acc][(c >> 1) * kChunk + 2 * (lane & 3)];
          sc[0] = f[0]; sc[1] = f[1]; sc[2] = f[8]; sc[3] = f[9];
        }
        uint32_t lo[8], hi[8];
        tmem_ld_frag16(taddr + (uint32_t)c * kChunk, lo);
        tmem_ld_frag16(taddr + (16u << 16) + (uint32_t)c * kChunk, hi);
        tc::tmem_ld_wait();
        if (c + 2 >= nchunks) {                      // this warp has read its last chunk: hand the accumulator back
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) remote_arrive(tempty_leader[acc]);
        }
        if (MODE == GEMM_GATE_UP) {
          // The gate warps compute the first eight tokens of the chunk, the up warps the other eight: each hands the
          // partner warp (same columns, other side) the half that it needs.
          const uint32_t base = epi + (uint32_t)set * kStgSet, b_act = base + (uint32_t)(chunk_no & 1) * kStgBytes;
          const uint32_t b_mine = base + (uint32_t)(2 + side) * kStgBytes;           // gate or up
          const uint32_t xch = epi + 2 * kStgSet + (uint32_t)(set * 2 + (q & 1)) * 2 * kXchBytes + (uint32_t)lane * 16;
          uint32_t keep[8];                          // this side's eight tokens: columns 0-15, then 16-31 of the warp
#pragma unroll
          for (int i = 0; i < 4; ++i) { keep[i] = side ? lo[4 + i] : lo[i]; keep[4 + i] = side ? hi[4 + i] : hi[i]; }
          tc::st_shared_v4(xch + (uint32_t)side * kXchBytes, side ? lo[0] : lo[4], side ? lo[1] : lo[5], side ? lo[2] : lo[6], side ? lo[3] : lo[7]);
          tc::st_shared_v4(xch + (uint32_t)side * kXchBytes + 512, side ? hi[0] : hi[4], side ? hi[1] : hi[5], side ? hi[2] : hi[6], side ? hi[3] : hi[7]);
          if (issuer) { if (args.out2) bulk_wait_read<0>(); else bulk_wait_read<1>(); }     // the buffers written below have left
          named_barrier(1 + set, 128);
          if (args.out2) { float one[4] = {1.f, 1.f, 1.f, 1.f}; stage(b_mine, lo, hi, one); }
          float gv[8], uv[8];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int4 p4 = tc::ld_shared_v4(xch + (uint32_t)(side ^ 1) * kXchBytes + h * 512);
            const float p[4] = {__int_as_float(p4.x), __int_as_float(p4.y), __int_as_float(p4.z), __int_as_float(p4.w)};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float m = __uint_as_float(keep[4 * h + i]);
              gv[4 * h + i] = side ? p[i] : m; uv[4 * h + i] = side ? m : p[i];
            }
          }
          bool plain = true;
#pragma unroll
          for (int i = 0; i < 8; ++i) plain = plain && silu_plain(gv[i]);
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = silu(gv[i]);
          if (!plain) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = silu_any(gv[i]);
          }
          uint32_t o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            o[i] = pack2(v[2 * i] * uv[2 * i] * sc[2 * side], v[2 * i + 1] * uv[2 * i + 1] * sc[2 * side + 1]);
          st_matrix_x4_trans(b_act + (uint32_t)side * 1024 + st_row + st_col, o[0], o[1], o[2], o[3]);
          tc::fence_async_smem();
          named_barrier(1 + set, 128);
          if (issuer) {
            if (side == 0) tc::tma_store_2d(&tma_out, b_act, col0, row);
            if (args.out2) tc::tma_store_2d(&tma_out2, b_mine, side * args.N + col0, row);
            bulk_commit();
          }
        } else {
          const uint32_t buf = epi + (uint32_t)((set * 2 + side) * 2 + (chunk_no & 1)) * kStgBytes;
          const int bar = 1 + set * 2 + side;
          if (issuer) bulk_wait_read<1>();           // the store issued two chunks ago has read this buffer
          named_barrier(bar, 64);
          stage(buf, lo, hi, sc);
          if (!push) {
            tc::fence_async_smem();
            named_barrier(bar, 64);
            if (issuer) { tc::tma_store_2d(&tma_out, buf, col0, row); bulk_commit(); }
          } else {
            // "push": every row goes straight to the rank its token came from (peer memory, plain 16-byte stores, 8
            // lanes per 128-byte run)
            named_barrier(bar, 64);
            const int tid = (q & 1) * 32 + lane, j = tid & 7;
#pragma unroll
            for (int p = 0; p < 2; ++p) {
              const int rr = p * 8 + (tid >> 3), info = args.push_info[row + rr];
              if (info < 0) continue;
              const int src = info / args.push_rows, idx = info - src * args.push_rows;
              if (src >= args.push_ranks) { if (j == 0) note(8, row + rr, MEP_ERR_BOUNDS); continue; }
              unsigned char* base = args.push_base + (size_t)src * args.push_stride;
              st_v4(base + ((size_t)idx * args.N + col0) * 2 + j * 16, tc::ld_shared_v4(buf + rr * 128 + ((j ^ (rr & 7)) << 4)));
              if (args.push_wsrc && col0 == 0 && j == 0)
                *reinterpret_cast<float*>(args.push_wbase + (size_t)src * args.push_stride + (size_t)idx * 4) = args.push_wsrc[row + rr];
            }
          }
        }
      }
    }
    if (lane == 0) bulk_wait_all<0>();       // shared memory must outlive the stores reading it
  }

  // ---------------- teardown: nobody leaves while the peer may still signal into this CTA
  tc::fence_before_sync();
  __syncthreads();
  cluster_sync();
  tc::fence_after_sync();
  if (warp == 1) tmem_dealloc2(tmem_base, 512);
  if (leader && threadIdx.x == 0) tq::scheduler_done(args.sched, pair == 0 ? 2 + args.sched_odd : 2, args.sched_ctas > 0 ? args.sched_ctas : (int)gridDim.x);
}

}  // namespace tp
}  // namespace mep

// Which kernel a launch takes (see Kind). Group sizes are only known on the device, and the code for bands costs a launch of few tiles 1 us of 20: it is there
// where groups are half as large as the line on average, so that some may be above it. All G groups count: a layer passes its slots for replicas
// too, which hold no row on one rank, so that there the average expert has to reach the line itself.
extern "C" int mep_pair_kind(int mode, int64_t a_rows, int G, int N, int K, int held, int held_rows, int early) {
  using namespace mep;
  if (a_rows * K * 2 > (int64_t)G * (tp::kXBytes / 2)) return tp::BANDED;
  const int64_t groups = held > 0 ? held : G, bytes = groups * (mode == GEMM_DGRAD_GU ? K / 2 : K) * N * 2;
  const bool few = held > 0 ? held_rows <= groups * tp::kStreamRows : a_rows <= groups * tp::kStreamRoom;
  return K % 128 == 0 && few && bytes >= (held > 0 && !early ? tp::kStreamBytesLate : tp::kStreamBytes) ? tp::STREAM : tp::PLAIN;
}

// One grouped GEMM launch on CTA pairs; same contract as mep_grouped_gemm for modes 0-3.
extern "C" int mep_grouped_gemm_2cta(int mode, const void* a, int64_t a_rows, int64_t a_cols, int64_t a_ld,
                                     const void* b0, const void* b1, int64_t b_rows, int64_t b_cols, int64_t b_ld,
                                     const mep::GemmArgs* args_in, int num_ctas, cudaStream_t stream) {
  using namespace mep;
  GemmArgs args = *args_in;
  MEP_REQUIRE(mode >= GEMM_GATE_UP && mode <= GEMM_DGRAD_GU, "gemm (CTA pairs): mode %d not supported", mode);
  MEP_REQUIRE(args.G >= 1 && args.G <= tp::kMaxGroups, "gemm: G=%d out of range [1,%d]", args.G, tp::kMaxGroups);
  MEP_REQUIRE(args.K % 64 == 0 && args.N % (mode == GEMM_GATE_UP ? 128 : 256) == 0, "gemm (CTA pairs): K=%d N=%d not tileable", args.K, args.N);
  num_ctas = pair_ctas(&args, num_ctas);
  MEP_REQUIRE(num_ctas >= 2, "gemm (CTA pairs): needs at least two CTAs");
  const int kind = mep_pair_kind(mode, a_rows, args.G, args.N, args.K, args.held, args.held_rows, args.early), deep = kind == tp::STREAM ? 128 : 64;
  CUtensorMap mx, mx64, mx16, mw0, mw1, mo, mo2;
  if (tmap_rows(&mx, a, a_rows, a_cols, a_ld, 64, 128) || tmap_rows(&mx64, a, a_rows, a_cols, a_ld, 64, 64) ||
      tmap_rows(&mx16, a, a_rows, a_cols, a_ld, 64, 16)) return -1;
  auto weights = [&](CUtensorMap* m, const void* b) {
    if (mode == GEMM_GATE_UP) return tmap_atoms(m, b, b_rows, b_cols, b_ld, 1, deep);
    if (mode == GEMM_DOWN) return tmap_atoms(m, b, b_rows, b_cols, b_ld, 2, deep);
    return tmap_rows(m, b, b_rows, b_cols, b_ld, 64, 128);
  };
  if (weights(&mw0, b0)) return -1;
  if (b1) { if (weights(&mw1, b1)) return -1; } else mw1 = mw0;
  if (args.push_info) mo = mx;
  else if (tmap_rows(&mo, args.out, a_rows, args.N, args.ldo, 64, tp::kChunk)) return -1;
  if (mode == GEMM_GATE_UP && args.out2) { if (tmap_rows(&mo2, args.out2, a_rows, 2 * (int64_t)args.N, 2 * (int64_t)args.N, 64, tp::kChunk)) return -1; }
  else mo2 = mo;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(num_ctas); cfg.blockDim = dim3(tp::kThreads); cfg.dynamicSmemBytes = tp::kSmem; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = args.pdl ? 2 : 1;
#define MEP_TP_CASE(M)                                                                                          \
  case M: {                                                                                                     \
    auto* kernel = kind == tp::BANDED ? tp::tok_pair_kernel<M, tp::BANDED>                                                \
                   : kind == tp::STREAM ? tp::tok_pair_kernel<M, tp::STREAM> : tp::tok_pair_kernel<M, tp::PLAIN>; \
    if (allow_smem((const void*)kernel, tp::kSmem)) return -1;                                                  \
    MEP_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, mx, mx64, mx16, mw0, mw1, mo, mo2, args));                  \
    break;                                                                                                      \
  }
  switch (mode) {
    MEP_TP_CASE(GEMM_GATE_UP) MEP_TP_CASE(GEMM_DOWN) MEP_TP_CASE(GEMM_DGRAD) MEP_TP_CASE(GEMM_DGRAD_GU)
    default: return set_error("gemm (CTA pairs): unknown mode %d", mode);
  }
#undef MEP_TP_CASE
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return 0;
}
