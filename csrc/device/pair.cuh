// Thin wrappers for kernels that run on CTA pairs (a cluster of two, tcgen05 cta_group::2): one elected thread of the
// leader CTA issues MMAs that use both SMs' tensor cores, shared memory and TMEM. Every load lands in the issuing
// CTA's own shared memory; only its byte count goes to the leader's barrier. No cluster-wide copy is used.
#pragma once
#include "tcgen05.cuh"
#include "gemm_args.h"

namespace mep {
namespace pair {

__device__ __forceinline__ uint32_t cluster_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t mapa(uint32_t saddr, uint32_t rank) {
  uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank)); return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Says that this warp's tcgen05.ld are done (tcgen05.wait::ld and fence::before_thread_sync come before it) and publishes no memory,
// hence relaxed: a release at cluster scope waits until the stores that the lane has in flight have been acknowledged, about
// 1200 cycles for a lane that has just issued the tile's TMA stores. That showed wherever the epilogue sets the pace: weight
// gradients of 64 groups of 256 tokens, 2048 x 1536, 212 -> 173 us; down of 16 groups of 765 tokens, 768 x 2048, 50 -> 44.
__device__ __forceinline__ void remote_arrive(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" :: "r"(cluster_addr) : "memory");
}
// cta_group::2 form: the destination is this CTA's shared memory, the mbarrier may live in the peer CTA
__device__ __forceinline__ void tma_load_2d_bar(uint32_t smem_dst, const CUtensorMap* map, int c0, int c1, uint32_t bar_cluster_addr, uint64_t policy) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
               :: "r"(smem_dst), "l"(map), "r"(c0), "r"(c1), "r"(bar_cluster_addr), "l"(policy) : "memory");
}
__device__ __forceinline__ void tma_load_2d_bar(uint32_t smem_dst, const CUtensorMap* map, int c0, int c1, uint32_t bar_cluster_addr) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               :: "r"(smem_dst), "l"(map), "r"(c0), "r"(c1), "r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(smem_result)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void mma2_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               :: "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier at this shared-memory offset in BOTH CTAs of the pair when the pair's MMAs are done
__device__ __forceinline__ void mma2_commit_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" :: "r"(bar), "h"((uint16_t)3) : "memory");
}
// Division of a >= 0 by a launch constant, results below 2^20: the product with the rounded reciprocal is off by one at most
struct Divisor {
  int b; float r;
  __device__ __forceinline__ explicit Divisor(int d) : b(d), r(1.f / (float)d) {}
  __device__ __forceinline__ int operator()(int a) const {
    const int q = (int)(((float)a + 0.5f) * r), rem = a - q * b;
    return q + (rem >= b) - (rem < 0);
  }
};
// Place of `key` among the first `n` of `keys` in falling order (keys differ, those of groups that do not count are negative;
// `keys` 16-byte aligned and filled up to a multiple of four). `low`: the sum of the keys' low 16 bits is added there.
__device__ __forceinline__ int rank_of(int key, const int* keys, int n, int* low = nullptr) {
  int r = 0;
#pragma unroll 4
  for (int j = 0; j < n; j += 4) {
    const int4 k = *reinterpret_cast<const int4*>(keys + j);
    r += (k.x > key) + (k.y > key) + (k.z > key) + (k.w > key);
    if (low) *low += (k.x & 0xffff) + (k.y & 0xffff) + (k.z & 0xffff) + (k.w & 0xffff);
  }
  return r;
}
// First row and 32-row units of the calling thread's group (threadIdx.x; of no use to threads from G on). All threads call it;
// `scratch`: 192 ints, 16-byte aligned, free again after the next block barrier.
__device__ __forceinline__ void group_rows(const GemmArgs& args, int* scratch, int& beg, int& rows, int& units) {
  const int g = threadIdx.x, G = args.G;
  beg = 0; rows = 0; units = 0;
  if (args.tokens) {
    int n = g < args.tokens_n ? __ldg(args.tokens + g) : 0;
    rows = (n + args.token_padding - 1) / args.token_padding * args.token_padding;
    if (g < 192) scratch[g] = rows;
    __syncthreads();
    for (int j = 0; j < G; j += 4) {
      const int4 v = *reinterpret_cast<const int4*>(scratch + j);
      beg += (j < g ? v.x : 0) + (j + 1 < g ? v.y : 0) + (j + 2 < g ? v.z : 0) + (j + 3 < g ? v.w : 0);
    }
    units = max((n + 31) >> 5, 0);
    __syncthreads();                     // before the scratch is used for something else
  } else if (g < G) {
    beg = g ? args.cu_seqlens[g - 1] : 0;
    rows = args.cu_seqlens[g] - beg;
    units = max((rows - (args.pad_rows ? args.pad_rows[2 * g + 1] : 0) + 31) >> 5, 0);
  }
}
// one lane of a converged warp; the others' registers stay warp-uniform, which keeps MMA descriptors out of the vector registers
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r != 0;
}
// 3-D form of tma_load_2d_bar (MN-major operands: 64 elements, k rows, 64-wide atoms)
__device__ __forceinline__ void tma_load_3d_bar(uint32_t smem_dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               :: "r"(smem_dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d_bar(uint32_t smem_dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar, uint64_t policy) {
  asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;"
               :: "r"(smem_dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar), "l"(policy) : "memory");
}
// 16 TMEM lanes x 16 fp32 columns in the layout of an MMA fragment: register 4b + i of thread T holds lane
// T / 4 + 8 * (i / 2), column 8b + 2 * (T % 4) + i % 2. `taddr` names lane 0 or 16 of the warp's quarter.
__device__ __forceinline__ void tmem_ld_frag16(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
// Four 8 x 8 bf16 matrices held as fragments (thread T: row T / 4, columns 2 * (T % 4) and + 1), stored transposed:
// thread 8i + j names the shared-memory row that receives column j of matrix i.
__device__ __forceinline__ void st_matrix_x4_trans(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" :: "r"(saddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void named_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" :: "r"(id), "r"(threads) : "memory"); }
// The same, true for everybody if `ok` holds for everybody.
__device__ __forceinline__ bool named_barrier_all(int id, int threads, bool ok) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(r) : "r"(ok ? 1u : 0u), "r"(id), "r"(threads) : "memory");
  return r != 0;
}

}  // namespace pair
}  // namespace mep
