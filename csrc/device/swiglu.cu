// Element-wise companions of the grouped GEMM (memory-bound, one pass each):
//   swiglu_bwd: from dA (= dY Wd^T, gradient w.r.t. the weighted activation), the saved
//               pre-activations (gate | up) and the per-row route weight w it produces
//               [dGate | dUp] and the route-weight gradient dW[row] = sum_j dA[row,j] * silu(g)*u.
//   sgd_step:   p -= lr * g for bf16 parameters with fp32 gradients (benchmark optimizer).
// Only rows below cu_seqlens[G-1] are defined; rows beyond are skipped.
#include "prims.cuh"
#include "silu.cuh"
#include "../host/launch.h"

namespace mep {

__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dA, const __nv_bfloat16* __restrict__ gu,
                                                         const float* __restrict__ w, __nv_bfloat16* __restrict__ dgu,
                                                         float* __restrict__ dw, const int32_t* __restrict__ cu_seqlens,
                                                         int G, int Hp) {
  pdl_trigger();
  pdl_wait();
  const int nrows = cu_seqlens[G - 1];
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const int nvec = Hp >> 3;
  for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < nrows; row += gridDim.x * wpb) {
    const float wr = w ? w[row] : 1.f;
    const __nv_bfloat16* da = dA + (size_t)row * Hp;
    const __nv_bfloat16* g = gu + (size_t)row * 2 * Hp;
    const __nv_bfloat16* u = g + Hp;
    __nv_bfloat16* dg = dgu + (size_t)row * 2 * Hp;
    __nv_bfloat16* du = dg + Hp;
    float dot = 0.f;
    for (int v = lane; v < nvec; v += 32) {
      const int4 xa = ld_nc_v4(da + v * 8), xg = ld_nc_v4(g + v * 8), xu = ld_nc_v4(u + v * 8);
      const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&xa);
      const __nv_bfloat162* pg = reinterpret_cast<const __nv_bfloat162*>(&xg);
      const __nv_bfloat162* pu = reinterpret_cast<const __nv_bfloat162*>(&xu);
      int4 og, ou;
      __nv_bfloat162* qg = reinterpret_cast<__nv_bfloat162*>(&og);
      __nv_bfloat162* qu = reinterpret_cast<__nv_bfloat162*>(&ou);
      float gs[8], sg[8];
      bool plain = true;
#pragma unroll
      for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(pg[i]); gs[2 * i] = f.x; gs[2 * i + 1] = f.y; }
#pragma unroll
      for (int i = 0; i < 8; ++i) { plain = plain && sigmoid_plain(gs[i]); sg[i] = sigmoid(gs[i]); }
      if (!plain) {
#pragma unroll
        for (int i = 0; i < 8; ++i) sg[i] = sigmoid_any(gs[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 fa = __bfloat1622float2(pa[i]), fu = __bfloat1622float2(pu[i]);
        float rg[2], ru[2];
        const float a_[2] = {fa.x, fa.y}, u_[2] = {fu.x, fu.y};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float g = gs[2 * i + j], sig = sg[2 * i + j];
          const float silu = g * sig;
          dot += a_[j] * silu * u_[j];
          const float d = a_[j] * wr;
          rg[j] = d * u_[j] * sig * (1.f + g * (1.f - sig));
          ru[j] = d * silu;
        }
        qg[i] = __floats2bfloat162_rn(rg[0], rg[1]);
        qu[i] = __floats2bfloat162_rn(ru[0], ru[1]);
      }
      st_v4(dg + v * 8, og);
      st_v4(du + v * 8, ou);
    }
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0 && dw) dw[row] = dot;
  }
}

// A block's loads of a chunk are all in flight before the first is used, and by default a block has one chunk: short blocks
// that the hardware hands out even out the SMs' unequal distance from memory. 3 x 705 M parameters: 2324 us (7.28 TB/s), where
// 1184 blocks in a loop of single vectors took 2496; 3 x 34 M: 115 against 130. Two chunks a block take 2400, loads that are
// marked as streaming 2480. Callers that name a number of blocks run beside a GEMM: single vectors in a loop need 29 to 48
// registers instead of 62 to 72 and find room next to its CTAs.
constexpr int kSgdVecs = 4;                                  // vectors of eight parameters

template <int VECS>
__device__ __forceinline__ void sgd_range(__nv_bfloat16* __restrict__ p, const float* __restrict__ g, float lr, int64_t n8) {
  constexpr int kSgdChunk = 256 * VECS;
  const int64_t chunks = (n8 + kSgdChunk - 1) / kSgdChunk;
  for (int64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
    const int64_t base = c * kSgdChunk + threadIdx.x;
    int4 x[VECS]; float4 g0[VECS], g1[VECS];
#pragma unroll
    for (int u = 0; u < VECS; ++u) {
      const int64_t i = base + u * 256;
      if (i < n8) {
        x[u] = *reinterpret_cast<const int4*>(p + i * 8);
        g0[u] = *reinterpret_cast<const float4*>(g + i * 8); g1[u] = *reinterpret_cast<const float4*>(g + i * 8 + 4);
      }
    }
#pragma unroll
    for (int u = 0; u < VECS; ++u) {
      const int64_t i = base + u * 256;
      if (i >= n8) break;
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&x[u]);
      const float gg[8] = {g0[u].x, g0[u].y, g0[u].z, g0[u].w, g1[u].x, g1[u].y, g1[u].z, g1[u].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float2 f = __bfloat1622float2(h[k]);
        f.x = fmaf(-lr, gg[2 * k], f.x); f.y = fmaf(-lr, gg[2 * k + 1], f.y);      // the form wgrad's fused update uses
        h[k] = __floats2bfloat162_rn(f.x, f.y);
      }
      *reinterpret_cast<int4*>(p + i * 8) = x[u];
    }
  }
}

template <int VECS> __global__ void __launch_bounds__(256) sgd_kernel(__nv_bfloat16* p, const float* g, float lr, int64_t n8) { sgd_range<VECS>(p, g, lr, n8); }

struct SgdPack { __nv_bfloat16* p[4]; const float* g[4]; int64_t n8[4]; };
template <int VECS> __global__ void __launch_bounds__(256) sgd_many_kernel(SgdPack k, float lr) { sgd_range<VECS>(k.p[blockIdx.y], k.g[blockIdx.y], lr, k.n8[blockIdx.y]); }

// The same update for the groups of a [G, n] tensor whose mask word is zero (`want` = 0) or non-zero (1):
// used for the experts that the weight-gradient GEMM did not already update in its epilogue.
template <int VECS>
__global__ void __launch_bounds__(256) sgd_groups_kernel(__nv_bfloat16* __restrict__ p, const float* __restrict__ g, float lr,
                                                         int64_t n8, const int32_t* __restrict__ mask, int want) {
  const int grp = blockIdx.y;
  if ((mask[grp] != 0) != (want != 0)) return;
  sgd_range<VECS>(p + (int64_t)grp * n8 * 8, g + (int64_t)grp * n8 * 8, lr, n8);
}

// For tests: compares the branch-free forms with the division for the `n` floats whose bits start at `first`;
// bad[0] / bad[1] count the sigmoids / SiLUs that differ, seen[0] / seen[1] those that were compared.
__global__ void __launch_bounds__(256) silu_sweep_kernel(uint32_t first, uint32_t n, unsigned long long* bad, unsigned long long* seen) {
  unsigned b0 = 0, b1 = 0, s0 = 0, s1 = 0;
  for (uint64_t i = blockIdx.x * 256ull + threadIdx.x; i < n; i += gridDim.x * 256ull) {
    const float g = __uint_as_float(first + (uint32_t)i);
    if (sigmoid_plain(g)) { ++s0; b0 += __float_as_uint(sigmoid(g)) != __float_as_uint(sigmoid_any(g)); }
    if (silu_plain(g)) { ++s1; b1 += __float_as_uint(silu(g)) != __float_as_uint(silu_any(g)); }
  }
  atomicAdd(bad, b0); atomicAdd(bad + 1, b1); atomicAdd(seen, s0); atomicAdd(seen + 1, s1);
}

}  // namespace mep

extern "C" int mep_silu_sweep(uint32_t first, uint32_t n, unsigned long long* bad, unsigned long long* seen, cudaStream_t stream) {
  return mep::launch_plain(mep::silu_sweep_kernel, dim3(1184), dim3(256), 0, stream, first, n, bad, seen);
}

extern "C" int mep_swiglu_bwd(const void* dA, const void* gu, const float* w, void* dgu, float* dw,
                              const int32_t* cu_seqlens, int G, int Hp, int num_blocks, int pdl, cudaStream_t stream) {
  MEP_REQUIRE(Hp % 8 == 0, "swiglu_bwd: inner size %d must be a multiple of 8", Hp);
  return mep::launch_plain_pdl(mep::swiglu_bwd_kernel, dim3(num_blocks), dim3(256), 0, stream, pdl != 0,
                           (const __nv_bfloat16*)dA, (const __nv_bfloat16*)gu, w, (__nv_bfloat16*)dgu, dw, cu_seqlens, G, Hp);
}

// `num_blocks` of the three: blocks of a tensor or group, 0: one for each chunk.
static int sgd_blocks(int num_blocks, int64_t n) { return num_blocks > 0 ? num_blocks : (int)((n / 8 + 256 * mep::kSgdVecs - 1) / (256 * mep::kSgdVecs)); }

extern "C" int mep_sgd_step(void* p, const float* g, float lr, int64_t n, int num_blocks, cudaStream_t stream) {
  MEP_REQUIRE(n % 8 == 0, "sgd_step: element count must be a multiple of 8");
  MEP_REQUIRE(num_blocks >= 0, "sgd_step: %d blocks", num_blocks);
  if (n == 0) return 0;
  return mep::launch_plain(num_blocks > 0 ? mep::sgd_kernel<1> : mep::sgd_kernel<mep::kSgdVecs>, dim3(sgd_blocks(num_blocks, n)), dim3(256), 0, stream, (__nv_bfloat16*)p, g, lr, n / 8);
}

// sgd_step of up to four tensors in one launch.
extern "C" int mep_sgd_step_many(int count, void* const* p, const float* const* g, const int64_t* n, float lr, int num_blocks, cudaStream_t stream) {
  MEP_REQUIRE(count >= 1 && count <= 4, "sgd_step: %d tensors", count);
  MEP_REQUIRE(num_blocks >= 0, "sgd_step: %d blocks", num_blocks);
  mep::SgdPack k = {};
  int64_t most = 0;
  for (int i = 0; i < count; ++i) {
    MEP_REQUIRE(n[i] % 8 == 0, "sgd_step: element count must be a multiple of 8");
    k.p[i] = (__nv_bfloat16*)p[i]; k.g[i] = g[i]; k.n8[i] = n[i] / 8;
    if (n[i] > most) most = n[i];
  }
  if (most == 0) return 0;
  return mep::launch_plain(num_blocks > 0 ? mep::sgd_many_kernel<1> : mep::sgd_many_kernel<mep::kSgdVecs>, dim3(sgd_blocks(num_blocks, most), count), dim3(256), 0, stream, k, lr);
}

extern "C" int mep_sgd_step_groups(void* p, const float* g, float lr, int64_t n_per_group, int G, const int32_t* mask, int want,
                                   int num_blocks, cudaStream_t stream) {
  MEP_REQUIRE(n_per_group % 8 == 0 && G >= 1 && G <= 65535, "sgd_step_groups: %d groups of %lld elements", G, (long long)n_per_group);
  MEP_REQUIRE(num_blocks >= 0, "sgd_step_groups: %d blocks", num_blocks);
  if (n_per_group == 0) return 0;
  return mep::launch_plain(num_blocks > 0 ? mep::sgd_groups_kernel<1> : mep::sgd_groups_kernel<mep::kSgdVecs>, dim3(sgd_blocks(num_blocks, n_per_group), G), dim3(256), 0, stream, (__nv_bfloat16*)p, g, lr,
                           n_per_group / 8, mask, want);
}
