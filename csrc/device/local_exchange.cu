// Dispatch and combine of a group of ONE rank: plan, row scatter and padding in one launch; one gather-sum launch.
//
// With a single rank every expert is at home, a token's first entry is its primary row and all others are
// duplicates on the same rank, so the whole exchange is a local permutation. The multi-rank kernels do it in
// four dependent passes (planning, dispatch of the primaries, duplicate expansion from the primaries;
// duplicate reduction into the primaries, combine), each with grid barriers and half of them on `num_sms` SMs.
// Here the traffic is the minimum: dispatch reads every token row once and writes its K rows, combine reads the
// K rows and writes one. Both are HBM bound; the tables they leave are the ones the multi-rank kernels leave.
//
// Counterpart of the reference's dispatch / combine for num_ep_ranks = 1 (moonep/dispatch.py:50-692,
// moonep/combine.py:40-511), which has no separate path for it.
#include "prims.cuh"
#include "local_args.h"
#include "../host/launch.h"

namespace mep {

// Tables and weights are read by ordinary loads: a launch may begin while the kernel that writes them still runs, and the read-only path (ld.nc) asks
// for memory that nobody writes while the kernel is there.
constexpr int kLocThreads = 256, kLocWarps = kLocThreads / 32;
constexpr int kLocEntries = 1024;          // top-k entries ranked and copied at a time by one CTA
constexpr int kLocZeroBytes = 4096;        // zeroed shared memory the padding rows are stored from
constexpr int kLocMaxSlots = 8;            // row slots per copying warp
constexpr size_t kLocAlone = 115 * 1024;   // dynamic shared memory of which an SM has no room for two CTAs

// Up to this many entries every CTA counts all entries before its own by itself, above it the CTAs hand over their
// histograms. Counting costs a CTA all entries before its own, the hand-over two round trips to L2 and CTAs x E counts. Own
// count against hand-over, a dispatch with K=8 among others of its kind (programmatic launches), in us:
//   entries                 12288         18432         24576         32768         49152         65536        131072
//   H=64,   E=64      8.5 / 15.6   10.0 / 15.7   11.8 / 17.4   13.9 / 18.6   19.4 / 22.1   23.4 / 23.9   42.8 / 35.5
//   H=512,  E=64      9.1 / 16.2   11.3 / 17.6   13.2 / 19.1   15.9 / 21.6   22.4 / 26.0   27.8 / 28.8   62.5 / 53.8
//   H=2048, E=16     13.8 / 20.3   19.0 / 24.9   25.8 / 31.9   34.8 / 39.7   51.8 / 52.5   67.4 / 69.7     135 / 127
//   H=2048, E=256    14.7 / 22.3   20.8 / 28.8   27.6 / 36.3   35.8 / 44.0   54.8 / 60.8   69.8 / 71.9     141 / 138
//   H=4096, E=60     24.2 / 31.5   35.5 / 42.1   47.0 / 51.4   61.4 / 67.6   93.3 / 97.8     122 / 124             -
//   H=7168, E=32     37.6 / 44.6   56.5 / 60.3   75.3 / 82.1     101 / 101     153 / 157     202 / 196             -
// So the line is lower for long rows, at this many elements of all rows (4096, 7168, 8, E=32 with its combine: 197.0 / 195.8).
// With few CTAs each has as many entries before it, but there are fewer histograms to add up: below two thirds of the SMs the line is at five
// eighths. K=8, E=64 with 64 and with 32 CTAs: 32768 entries, H=64 20.1 / 21.1 and 31.8 / 33.0, H=1024 33.9 / 35.9 and 59.8 / 61.3; 40960, H=64 24.6
// / 25.3 and 39.4 / 39.8, H=1024 43.7 / 44.3 and 77.6 / 76.2; 49152, H=64 28.2 / 27.7 and 46.2 / 45.4, H=1024 53.1 / 51.5 and 91.5 / 90.0; 65536,
// H=64 36.3 / 33.7 and 60.1 / 58.0, H=1024 66.4 / 65.4 and 124 / 117. With 100: 49152, H=64 22.1 / 22.6, H=1024 37.6 / 40.4; 65536 28.6 / 26.6, 49.2
// / 50.6.
constexpr int kLocDirect = 65536, kLocDepth = 16;      // kLocDepth: entries that a thread has on their way when it counts
constexpr long long kLocDirectElems = 24576ll * 7168;

// A large batch of a saved plan is copied by many short CTAs, two or three to an SM, that the hardware hands out as SMs come free: SMs
// are not equally far from memory, and with one CTA for each the last was done 10 % after the average. Bytes that a CTA moves, and
// least bytes of a large batch; a caller that wants fewer CTAs than there are SMs gets its number instead. One CTA per SM against short ones, in us: S=4096, H=7168, K=8 101.6 / 89.2; 8192, 7168, 4 109.2 /
// 95.4; 8192, 2048, 8 58.8 / 53.8. Below 200 MB the gain is gone in a combine right behind, whose rows were in L2 (3001, 4096, 6 with its
// combine 65.8 / 66.9). Not for a fresh plan: planners and copiers in one launch hand over in 10 us, which only the largest
// batches win back (4096, 7168, 8 107.6 / 103.4; 1531, 7168, 8 48.1 / 55).
constexpr long long kLocShort = 311ll << 10, kLocLarge = 200ll << 20;

// Padding rows that are cleared behind row `first` of a group's `n` (see LocalDispatchArgs.pad_step).
__device__ __forceinline__ int local_pads(int first, int n, int step) { return step ? min(n, -first & (step - 1)) : n; }

// Exclusive prefix of padded group sizes: start[e] = first row of expert e; padpre[e] = padding rows of
// experts < e. 256 threads, E / 256 consecutive experts each. Returns the number of padding rows.
__device__ __forceinline__ int local_layout(const int32_t* tpe, int E, int pad, int step, int* start, int* padpre, int* s_warp) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (E + kLocThreads - 1) / kLocThreads, e0 = tid * per, e1 = min(e0 + per, E);
  int rows = 0, pads = 0;
  for (int e = e0; e < e1; ++e) { const int n = tpe[e], p = (n + pad - 1) / pad * pad; rows += p; pads += local_pads(n, p - n, step); }
  int ri = warp_incl_scan(rows), pi = warp_incl_scan(pads);
  if (lane == 31) { s_warp[warp] = ri; s_warp[kLocWarps + warp] = pi; }
  __syncthreads();
  int rb = 0, pb = 0, total = 0;
  for (int w = 0; w < kLocWarps; ++w) {
    if (w < warp) { rb += s_warp[w]; pb += s_warp[kLocWarps + w]; }
    total += s_warp[kLocWarps + w];
  }
  rb += ri - rows; pb += pi - pads;
  for (int e = e0; e < e1; ++e) {
    const int n = tpe[e], p = (n + pad - 1) / pad * pad;
    start[e] = rb; padpre[e] = pb; rb += p; pb += local_pads(n, p - n, step);
  }
  return total;
}

// One CTA owns a contiguous range of tokens. FRESH: their entries are ranked among the same-expert entries of
// the whole batch, in flat entry order, and the plan tables are written. Up to kLocDirect entries (MODE 1) a CTA
// counts the entries before its own itself: reading them is quicker than a hand-over between CTAs, which costs two
// round trips to L2. Above that (MODE 2) CTAs publish the histogram of their tokens and add up those of the CTAs
// before them; they number themselves in the order in which they start, so a CTA only ever waits for CTAs that are
// already running and no cooperative launch is needed. Then, from `dst` alone, each row goes through a warp's slot in shared memory
// with one bulk load and K bulk stores (lane k issues the store of entry k); rows of the next tokens are in
// flight meanwhile, in the fresh case already during the ranking.
// Bound by HBM: (1 + K) rows per token; 103 us at S=4096, H=7168, K=8 (5.1 TB/s, mostly stores) where planning, dispatch
// and duplicate expansion took 185.
template <int MODE>                        // 0: saved plan
__global__ void __launch_bounds__(kLocThreads, MODE ? 1 : 3)
local_dispatch_kernel(const MepRankCtx* __restrict__ cp, LocalDispatchArgs a, int copy_warps, int slots) {
  constexpr bool FRESH = MODE != 0, SHARED = MODE == 2;
  if (!a.early) pdl_trigger();               // a GEMM behind this kernel may set itself up meanwhile
  const MepRankCtx c = *cp;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_bar[kLocWarps * kLocMaxSlots];
  __shared__ int s_slot[kLocEntries];        // row of each entry of the current chunk (-1: bad entry, skipped)
  __shared__ int s_warp[2 * kLocWarps];
  __shared__ int s_vb, s_fail;
  const int nb = gridDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = c.K, S = c.S, E = c.E, NvS = c.NvS, pad = c.token_padding;
  const uint32_t row_bytes = (uint32_t)c.H * 2u;
  unsigned char* s_zero = smem;
  unsigned char* s_ring = smem + kLocZeroBytes;
  const int ngroups = FRESH ? E : 2 * E;
  int* s_start = reinterpret_cast<int*>(s_ring + (size_t)copy_warps * slots * row_bytes);   // FRESH: first row of expert e; else: first padding row of group g
  int* s_padpre = s_start + ngroups;
  int* s_cnt = s_padpre + ngroups;           // FRESH [E]: histogram, then next free row of expert e for this CTA's entries

  if (tid < kLocWarps * kLocMaxSlots) mbar_init(&s_bar[tid], 1);
  fence_mbar_init();
  for (int i = tid; i < kLocZeroBytes / 16; i += kLocThreads) reinterpret_cast<int4*>(s_zero)[i] = make_int4(0, 0, 0, 0);
  fence_proxy_async();
  if (FRESH) for (int e = tid; e < E; e += kLocThreads) s_cnt[e] = 0;
  // Up to here the kernel right before may still run, whatever it is. A GEMM behind this kernel may set itself up and load weights as soon as that one is done.
  pdl_wait();
  if (a.early) pdl_trigger();
  if (tid == 0) {
    s_fail = 0;
    s_vb = SHARED ? (int)atomicAdd(&a.sync[1], 1u) : (int)blockIdx.x;
    trace_mark(c, MEP_K_DISPATCH, 1);
  }
  __syncthreads();
  const int vb = s_vb;
  const uint32_t ep = SHARED ? *(volatile uint32_t*)&a.sync[0] + 1u : 0u;
  const int tb = min(nb, S), tpb = (S + tb - 1) / tb;
  const int t0 = min(vb * tpb, S), t1 = min(t0 + tpb, S);

  // ---- the copying warps' first rows are on their way before anything else
  const int chunk_tok = kLocEntries / K;
  unsigned char* ring = s_ring + (size_t)warp * slots * row_bytes;
  uint64_t* bars = s_bar + warp * kLocMaxSlots;
  const bool copier = warp < copy_warps;
  const int ntok = copier && t0 + warp < t1 ? (t1 - t0 - warp + copy_warps - 1) / copy_warps : 0;   // tokens t0 + warp + i * copy_warps
  int issued = 0;
  auto load = [&](int i) {       // lane 0
    issued = i + 1;
    mbar_expect_tx(&bars[i % slots], row_bytes);
    bulk_g2s(ring + (size_t)(i % slots) * row_bytes, a.hidden + (size_t)(t0 + warp + i * copy_warps) * c.H, row_bytes, &bars[i % slots]);
  };
  if (lane == 0) for (int i = 0; i < slots - 1 && i < ntok; ++i) load(i);

  // ---- layout, histogram of this CTA's entries
  int total_pad;
  if (FRESH) {
    if (SHARED) {                            // own entries
      for (int i = t0 * K + tid; i < t1 * K; i += kLocThreads) {
        const int e = a.topk[i];
        if ((unsigned)e < (unsigned)E) atomicAdd(&s_cnt[e], 1);
        else report(c, MEP_ERR_BOUNDS, MEP_K_PLANNING, 1, i, (uint32_t)e, (uint32_t)E);
      }
    } else if (t0 < t1) {
      // All entries before them. The CTAs read the same ones: each begins at another place, else the slices of L2 that hold the first entries
      // serve 148 SMs at once and the others none. That and sixteen loads in flight instead of eight: 18432 entries, H=4096, E=60 41.1 -> 38.3 us;
      // 32768, H=2048, E=16 47 -> 35.7. (Counting by ballots over the bits of the numbers, without atomics: 39.0.)
      const int n = t0 * K, rounds = n <= 8 * kLocThreads ? 0 : (n + kLocThreads * kLocDepth - 1) / (kLocThreads * kLocDepth);
      if (!rounds) {                         // a decode batch: without the code for sixteen loads, which every launch would fetch anew
        int e[8];
#pragma unroll
        for (int d = 0; d < 8; ++d) e[d] = tid + d * kLocThreads < n ? a.topk[tid + d * kLocThreads] : -1;
#pragma unroll
        for (int d = 0; d < 8; ++d) if ((unsigned)e[d] < (unsigned)E) atomicAdd(&s_cnt[e[d]], 1);
      }
      int at = rounds ? vb % rounds : 0;
      for (int r = 0; r < rounds; ++r) {
        const int i0 = at * (kLocThreads * kLocDepth) + tid;
        if (++at == rounds) at = 0;
        int e[kLocDepth];
#pragma unroll
        for (int d = 0; d < kLocDepth; ++d) e[d] = i0 + d * kLocThreads < n ? a.topk[i0 + d * kLocThreads] : -1;
#pragma unroll
        for (int d = 0; d < kLocDepth; ++d) if ((unsigned)e[d] < (unsigned)E) atomicAdd(&s_cnt[e[d]], 1);
      }
    }
    total_pad = local_layout(a.tpe, E, pad, a.pad_step, s_start, s_padpre, s_warp);
    __syncthreads();
    if (SHARED && t0 < t1) {
      for (int e = tid; e < E; e += kLocThreads) a.hist[(size_t)vb * E + e] = s_cnt[e];
      __syncthreads();
      if (tid == 0) { __threadfence(); st_release_gpu(a.sync + 16 + vb, ep); }
    }
    if (vb == nb - 1) {          // the CTA with the least to copy writes the tables that only depend on the counts
      for (int g = tid; g < 2 * E; g += kLocThreads) {
        const int e = g < E ? g : E - 1;
        const int n = a.tpe[e], p = (n + pad - 1) / pad * pad;
        a.cu_seqlens[g] = s_start[e] + p;
        const bool has = g < E && p > n;
        a.zero_fill[2 * g] = has ? s_start[e] + n : 0;
        a.zero_fill[2 * g + 1] = has ? p - n : 0;
        if (g < E) a.experts_to_copy[g] = -1;
      }
      if (tid < 2) { a.remote_stats[tid] = 0; a.dup_counts[tid] = K > 1 ? (tid ? S * (K - 1) : S) : 0; }
    }
  } else {
    // padding rows of the saved plan: group g owns flat indices [padpre[g], padpre[g + 1])
    int run = 0;
    for (int g0 = 0; g0 < ngroups; g0 += kLocThreads) {
      const int g = g0 + tid;
      const int first = g < ngroups ? a.zero_fill[2 * g] : 0;
      const int n = g < ngroups ? local_pads(first, a.zero_fill[2 * g + 1], a.pad_step) : 0;
      if (g < ngroups) s_start[g] = first;
      const int incl = warp_incl_scan(n);
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      int base = run;
      for (int w = 0; w < kLocWarps; ++w) { if (w < warp) base += s_warp[w]; run += s_warp[w]; }
      if (g < ngroups) s_padpre[g] = base + incl - n;
      __syncthreads();
    }
    total_pad = run;
  }

  // ---- padding rows, one thread each; neighbours in the flat order go to different CTAs and warps
  {
    for (int z = (lane * kLocWarps + warp) * nb + vb; z < total_pad; z += kLocThreads * nb) {
      int lo = 0, hi = ngroups - 1;          // last group with padpre <= z
      while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (s_padpre[mid] <= z) lo = mid; else hi = mid - 1; }
      int row = s_start[lo] + (z - s_padpre[lo]);
      if (FRESH) row += a.tpe[lo];
      if ((unsigned)row >= (unsigned)NvS) report(c, MEP_ERR_BOUNDS, MEP_K_DISPATCH, 40, lo, (uint32_t)row, (uint32_t)NvS);
      else {
        char* p = (char*)a.out_hidden + (size_t)row * row_bytes;
        for (uint32_t b = 0; b < row_bytes; b += kLocZeroBytes) bulk_s2g(p + b, s_zero, min((uint32_t)kLocZeroBytes, row_bytes - b));
        if (a.weights) a.out_weights[row] = 0.f;
        if (a.out_srcinfo) a.out_srcinfo[row] = -1;
      }
    }
  }
  bulk_commit();

  // ---- entries of earlier CTAs
  if (MODE == 1) {
    for (int e = tid; e < E; e += kLocThreads) s_cnt[e] += s_start[e];
    __syncthreads();
  } else if (SHARED && t0 < t1) {
    for (int u = tid; u < vb; u += kLocThreads) {
      uint32_t seen = 0;
      const bool ok = bounded_wait(c, [&] { seen = ld_acquire_gpu(a.sync + 16 + u); return (int32_t)(seen - ep) >= 0; });
      if (!ok) { report(c, MEP_ERR_GRID_SYNC_TIMEOUT, MEP_K_PLANNING, 12, u, seen, ep); s_fail = 1; }
    }
    for (int e = tid; e < E; e += kLocThreads) s_cnt[e] = s_start[e];
    __syncthreads();
    if (E <= kLocThreads) {      // several threads per expert, each over every `parts`-th CTA
      int w = 1; while (w < E) w <<= 1;
      const int parts = kLocThreads / w, e = tid & (w - 1), part = tid / w;
      if (e < E) {
        int sum = 0;
#pragma unroll 8
        for (int u = part; u < vb; u += parts) sum += __ldcg(a.hist + (size_t)u * E + e);
        if (sum) atomicAdd(&s_cnt[e], sum);
      }
    } else {
      for (int e = tid; e < E; e += kLocThreads) {
        int sum = 0;
#pragma unroll 8
        for (int u = 0; u < vb; ++u) sum += __ldcg(a.hist + (size_t)u * E + e);
        s_cnt[e] += sum;
      }
    }
    __syncthreads();
  }

  // ---- chunk by chunk: rank (fresh), tables, rows
  int it = 0, arrived = 0;                     // tokens this warp has copied / whose load it has waited for
  uint32_t phases = 0;                         // parity of each slot's barrier
  bool ok = !(SHARED && s_fail);
  for (int c0 = t0; c0 < t1 && ok; c0 += chunk_tok) {
    const int c1 = min(c0 + chunk_tok, t1), n = (c1 - c0) * K;
    if (FRESH) {
      for (int i0 = 0; i0 < n; i0 += kLocThreads) {
        const int i = i0 + tid;
        int e = i < n ? a.topk[(size_t)c0 * K + i] : -1;
        if ((unsigned)e >= (unsigned)E) {
          if (MODE == 1 && i < n) report(c, MEP_ERR_BOUNDS, MEP_K_PLANNING, 1, c0 * K + i, (uint32_t)e, (uint32_t)E);
          e = -1;
        }
        const unsigned m = __match_any_sync(0xffffffffu, e);
        const int before = __popc(m & lanemask_lt());
        int row = -1;
        const int nw = min(kLocWarps, (n - i0 + 31) >> 5);
        for (int w = 0; w < nw; ++w) {         // warps in order: the rank is stable
          if (warp == w && e >= 0) {
            const int leader = __ffs(m) - 1;
            int old = 0;
            if (lane == leader) { old = s_cnt[e]; s_cnt[e] = old + __popc(m); }
            row = __shfl_sync(m, old, leader) + before;
          }
          __syncthreads();
        }
        if (i < n) {
          if (e >= 0 && (row >= s_start[e] + a.tpe[e] || (unsigned)row >= (unsigned)NvS)) {   // counts that are not those of topk
            report(c, MEP_ERR_BOUNDS, MEP_K_PLANNING, 2, c0 * K + i, (uint32_t)row, (uint32_t)NvS);
            row = -1;
          }
          s_slot[i] = row;
        }
      }
    } else {
      for (int i = tid; i < n; i += kLocThreads) {
        const int d = a.dst[(size_t)c0 * K + i];
        int row = d >= 0 ? d : -d - 1;
        if (row >= NvS) { report(c, MEP_ERR_BOUNDS, MEP_K_DISPATCH, 41, c0 + i / K, (uint32_t)row, (uint32_t)NvS); row = -1; }
        s_slot[i] = row;
      }
    }
    __syncthreads();
    // rows: warp w copies tokens t0 + w + i * copy_warps of this chunk
    for (; it < ntok && ok; ++it) {
      const int s = t0 + warp + it * copy_warps;
      if (s >= c1) break;
      const int st = it % slots;
      if (it + slots - 1 < ntok) {             // refill the slot of the token before: its stores must have been read
        bulk_wait_read<0>();
        __syncwarp();
        if (lane == 0) load(it + slots - 1);
      }
      bool got = true;
      if (lane == 0) got = mbar_wait_bounded(&bars[st], (phases >> st) & 1u, c.wait_budget_ns);
      got = __shfl_sync(0xffffffffu, got ? 1 : 0, 0) != 0;
      if (!got) { if (lane == 0) report(c, MEP_ERR_MBAR_TIMEOUT, MEP_K_DISPATCH, 20, s, 0, 0); ok = false; break; }
      phases ^= 1u << st;
      ++arrived;
      for (int k = lane; k < K; k += 32) {
        const int row = s_slot[(s - c0) * K + k];
        if (row >= 0) bulk_s2g((char*)a.out_hidden + (size_t)row * row_bytes, ring + (size_t)st * row_bytes, row_bytes);
      }
      bulk_commit();
    }
    for (int i = tid; i < n; i += kLocThreads) {
      const int row = s_slot[i], j = c0 * K + i;
      const int s = j / K, k = j - s * K;
      if (FRESH) {
        const int r = row < 0 ? 0 : row;
        a.dst[j] = k == 0 ? r : -r - 1;
        if (K > 1) {
          if (k == 0) { a.dup_groups[3 * s] = r; a.dup_groups[3 * s + 1] = s * (K - 1); a.dup_groups[3 * s + 2] = K - 1; }
          else a.dup_loffs[s * (K - 1) + k - 1] = r;
        }
      }
      if (row >= 0) {
        if (a.weights) a.out_weights[row] = a.weights[j];
        if (a.out_srcinfo) a.out_srcinfo[row] = j;
      }
    }
    ok = __syncthreads_and(ok ? 1 : 0) != 0;   // s_slot is free again; the warps go on or stop together
  }
  if (!ok && lane == 0)                        // do not leave while loads into this CTA's memory are in flight: they get their time (again)
    for (int i = arrived; i < issued; ++i) {
      mbar_wait_bounded(&bars[i % slots], (phases >> (i % slots)) & 1u, c.wait_budget_ns);
      phases ^= 1u << (i % slots);
    }
  bulk_wait_all<0>();
  if (vb == 0 && tid == 0) {
    count(c, MEP_CNT_DISPATCHES, 1); count(c, MEP_CNT_ROWS_SENT, (unsigned long long)S); count(c, MEP_CNT_PEER_ROWS, (unsigned long long)S);
    count(c, MEP_CNT_PAD_ROWS, (unsigned long long)total_pad);
    trace_mark(c, MEP_K_DISPATCH, 5);
  }
  if (SHARED) {                                // the last CTA out closes the launch
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      if (atomicAdd(&a.sync[2], 1u) == (uint32_t)nb - 1u) { a.sync[1] = 0u; a.sync[2] = 0u; a.sync[0] = ep; __threadfence(); }
    }
  }
}

// ------------------------------------------------------------------ combine
__device__ __forceinline__ void add_bf16x8(float* acc, const int4& x) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); acc[2 * i] += f.x; acc[2 * i + 1] += f.y; }
}

// out[s] = sum over k, ascending, of the rows of token s, in fp32, rounded once: what the duplicate reduction
// followed by the combine computes, without the intermediate row. A warp works on (token, column part) units: one
// bulk load per row brings a unit into one half of the warp's stage while the other half is summed, and the plan
// entries of the unit behind that one are already being fetched. LAST_FIRST: units come from the last to the
// first. Where nothing has touched the rows of a large batch since a saved plan's dispatch, which goes through the tokens in order,
// the last ones are still in L2 (behind a fresh plan, whose CTAs have a range of tokens each, it costs 0.6 %): saved dispatch and combine of S=4096, H=7168, K=8 187.8 -> 182.3 us.
// Bound by HBM: (K + 1) rows per token. Loading into registers instead kept too little in flight: 138 us at
// S=4096, H=7168, K=8 with 32 warps per SM and 218 us with 8 (twice the loads per lane).
constexpr int kLcWarps = 12, kLcHalf = 8192;

template <bool LAST_FIRST>
__global__ void __launch_bounds__(kLcWarps * 32, 1) local_combine_kernel(const MepRankCtx* __restrict__ cp, LocalCombineArgs a, int part_vecs, int nparts) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_bar[kLcWarps * 2];
  const int K = cp->K, NvS = cp->NvS, nvec = cp->H >> 3;
  const uint64_t budget = cp->wait_budget_ns;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < kLcWarps * 2) mbar_init(&s_bar[tid], 1);
  fence_mbar_init();
  pdl_wait();                                  // the rows may come from the kernel right before
  __syncthreads();
  unsigned char* stage = smem + (size_t)warp * 2 * kLcHalf;
  uint64_t* bars = s_bar + warp * 2;
  const int units = cp->S * nparts, step = gridDim.x * kLcWarps;
  int u = blockIdx.x * kLcWarps + warp;
  auto unit = [&](int x) { return LAST_FIRST ? units - 1 - x : x; };
  auto fetch = [&](int x) { return x < units && lane < K ? a.dst[(size_t)(unit(x) / nparts) * K + lane] : 0; };
  // loads of unit x (plan entry d in lane k) into half h; returns the lanes whose entry names a row
  auto issue = [&](int at, int d, int h) {
    const int x = unit(at);
    const int part = x % nparts, vb = part * part_vecs;
    const uint32_t bytes = (uint32_t)min(part_vecs, nvec - vb) * 16u;
    const int row = d >= 0 ? d : -d - 1;
    const unsigned valid = __ballot_sync(0xffffffffu, lane < K && row < NvS);
    if (a.out_weights && part == 0 && lane < K) a.out_weights[(size_t)(x / nparts) * K + lane] = row < NvS ? a.weights[row] : 0.f;
    if (lane == 0) mbar_expect_tx(&bars[h], bytes * (uint32_t)__popc(valid));
    __syncwarp();                              // also: every lane has finished reading this half
    if ((valid >> lane) & 1u)
      bulk_g2s(stage + (size_t)h * kLcHalf + (size_t)lane * part_vecs * 16, reinterpret_cast<const int4*>(a.rows) + (size_t)row * nvec + vb, bytes, &bars[h]);
    return valid;
  };
  const unsigned all = K >= 32 ? 0xffffffffu : (1u << K) - 1u;
  unsigned cur = 0, nxt = 0;
  int h = 0, bad = -1;
  uint32_t phase = 0;                          // parity of both halves: they are used in turn
  if (u < units) cur = issue(u, fetch(u), 0);
  int dn = fetch(u + step);
  // Only now: what an early launch behind this one reads ahead of its own wait may come from the kernel before this one, too. In front of the first loads it
  // delayed them: dispatch and combine of 3000 x 4, H=512 14.64 us instead of 14.54 (as long as from the kernel's start), 500 x 4, H=1024 10.62 instead of 10.42.
  pdl_trigger();
  bool ok = true;
  for (; u < units; u += step) {
    const int un = u + step;
    if (un < units) nxt = issue(un, dn, h ^ 1);
    dn = fetch(un + step);
    const int x = unit(u);
    if (cur != all) bad = x / nparts;
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[h], phase, budget))) { ok = false; break; }
    const int part = x % nparts, vb = part * part_vecs, n = min(part_vecs, nvec - vb);
    const unsigned char* base = stage + (size_t)h * kLcHalf;
    int4* orow = reinterpret_cast<int4*>(a.out) + (size_t)(x / nparts) * nvec + vb;
    for (int v = lane; v < n; v += 32) {
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
      for (int k = 0; k < K; ++k)
        if ((cur >> k) & 1u) add_bf16x8(acc, *reinterpret_cast<const int4*>(base + ((size_t)k * part_vecs + v) * 16));
      int4 o; __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
      st_na_v4(orow + v, o);
    }
    cur = nxt; phase ^= (uint32_t)h; h ^= 1;
  }
  if (!ok) {                                   // the other half's copies get their time too before the stage goes away
    if (u + step < units) mbar_wait_bounded(&bars[h ^ 1], phase ^ (uint32_t)h, budget);
    if (lane == 0) report(*cp, MEP_ERR_MBAR_TIMEOUT, MEP_K_COMBINE, 22, u, 0, 0);
  }
  if (bad >= 0 && lane == 0) report(*cp, MEP_ERR_BOUNDS, MEP_K_COMBINE, 20, bad, (uint32_t)NvS, (uint32_t)NvS);   // corrupt or foreign plan
  if (blockIdx.x == 0 && tid == 0) {
    trace_mark(*cp, MEP_K_COMBINE, 1);
    count(*cp, MEP_CNT_COMBINES, 1); count(*cp, MEP_CNT_ROWS_PULLED, (unsigned long long)cp->S * K);
  }
}

}  // namespace mep

// `num_blocks`: most CTAs; from `sms` on (those of the device, with a CTA for each) the launch may have more, see kLocShort. fresh: plan from
// topk / tpe as well; else a.dst / a.zero_fill are read.
extern "C" int mep_launch_local_dispatch(const MepRankCtx* ctx, const mep::LocalDispatchArgs* args, int fresh,
                                         int num_blocks, int sms, int S, int K, int H, int E, int pdl, cudaStream_t stream) {
  using namespace mep;
  LocalDispatchArgs a = *args;
  a.early = pdl;
  const size_t row = (size_t)H * 2;
  const size_t tables = (size_t)(fresh ? 3 : 4) * E * sizeof(int);
  const long long bytes = (long long)S * (K + 1) * (long long)row;
  const bool large = !fresh && num_blocks >= sms && bytes >= kLocLarge && tables + kLocZeroBytes + 2 * row <= 104 * 1024;
  const size_t budget = (large ? 104 : 208) * 1024, ring = (large ? 52 : 96) * 1024;
  MEP_REQUIRE(tables + kLocZeroBytes + 2 * row <= budget, "dispatch: H=%d rows (%zu B) with E=%d do not fit shared memory", H, row, E);
  const int all = (int)((budget - tables - kLocZeroBytes) / row);           // row slots that fit
  int warps = all / 2 < kLocWarps ? all / 2 : kLocWarps;
  int slots = all / warps < kLocMaxSlots ? all / warps : kLocMaxSlots;
  // the fewest slots that still hold `ring` bytes of rows per CTA: more buys nothing, and a smaller footprint starts sooner
  while (slots > 2 && (size_t)warps * (slots - 1) * row >= ring) --slots;
  size_t smem = kLocZeroBytes + (size_t)warps * slots * row + tables;
  // A programmatic launch is placed as the SMs of the kernel before come free: without this the first of them would get two CTAs and the last none
  // (8000 x 8, H=1024 with its combine 80.0 us instead of 65.6, 3000 x 4, H=512 17.7 instead of 14.5). It costs two Buffers on streams of their own, whose
  // dispatches then share no SM: of 3000 x 4, H=256 each with its combine 21.1 us instead of 16.9 with ordinary launches. Not with a token
  // for each CTA at most, where two CTAs on an SM are as good as one (148 x 8, H=1024 9.4 / 9.5, 64 x 8 9.3 / 9.2; beside another Buffer's 13.8 / 9.3 and 10.3 / 8.8).
  if (pdl && !large && S > num_blocks && smem < kLocAlone) smem = kLocAlone;
  if (large) {                               // the same number of tokens for each warp
    const long long each = kLocShort / ((long long)row * (K + 1) * warps);
    const int tokens = warps * (each < 1 ? 1 : (int)each);
    num_blocks = (S + tokens - 1) / tokens;
  }
  const int direct = 3ll * num_blocks >= 2ll * sms ? kLocDirect : kLocDirect / 8 * 5;
  if (fresh && S * K <= direct && (long long)S * K * H <= kLocDirectElems) return launch_plain_pdl(local_dispatch_kernel<1>, dim3(num_blocks), dim3(kLocThreads), smem, stream, pdl != 0, ctx, a, warps, slots);
  if (fresh) return launch_plain_pdl(local_dispatch_kernel<2>, dim3(num_blocks), dim3(kLocThreads), smem, stream, pdl != 0, ctx, a, warps, slots);
  return launch_plain_pdl(local_dispatch_kernel<0>, dim3(num_blocks), dim3(kLocThreads), smem, stream, pdl != 0, ctx, a, warps, slots);
}

extern "C" int mep_launch_local_combine(const MepRankCtx* ctx, const mep::LocalCombineArgs* args, int num_blocks,
                                        int S, int H, int K, int pdl, int last_first, cudaStream_t stream) {
  using namespace mep;
  const int nvec = H / 8;
  // a unit is what fits half a warp's stage, or less while that leaves warps without work
  int part = kLcHalf / 16 / K;
  if (part > 32) part &= ~31;
  if (part > nvec) part = nvec;
  while (part > 32 && (long long)S * ((nvec + part - 1) / part) < (long long)num_blocks * kLcWarps) part = (part / 2 + 31) & ~31;
  const int nparts = (nvec + part - 1) / part;
  MEP_REQUIRE((long long)S * nparts < (1ll << 30), "combine: S=%d, H=%d is too large", S, H);
  const int grid = (int)(((long long)S * nparts + kLcWarps - 1) / kLcWarps);
  const bool last = last_first && (long long)S * (K + 1) * H * 2 >= kLocLarge;
  return launch_plain_pdl(last ? local_combine_kernel<true> : local_combine_kernel<false>, dim3(grid < num_blocks ? grid : num_blocks), dim3(kLcWarps * 32), (size_t)kLcWarps * 2 * kLcHalf,
                          stream, pdl != 0, ctx, *args, part, nparts);
}
