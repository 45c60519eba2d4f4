// Router of a MoE block around the gate GEMM: bias, softmax over the experts, top-k, renormalised weights and the
// expert histogram in one launch, and the gradient of the logits in another. As torch operators this took ten
// launches forward and twelve backward, most of them shorter than their launch.
//
// Sums are taken in the order in which torch takes them (lane l adds elements l, l + 32, ..., then lanes are
// added pairwise, half the distance each time), so that weights and gradients are those of the operators to the last
// bit: training amplifies a flipped bit of a route weight into other experts for some tokens within a few steps.
#include "prims.cuh"
#include "../host/launch.h"
#include <math.h>

namespace mep {

constexpr int kRouteMaxE = 512;

// Sort key of (logit, expert): larger first, NaN largest (as torch.topk), lower expert on ties. Never 0.
__device__ __forceinline__ unsigned long long route_key(float v, int e) {
  unsigned b = __float_as_uint(v);
  b = v != v ? 0xffffffffu : (b & 0x80000000u) ? ~b : b | 0x80000000u;
  return ((unsigned long long)b << 32) | (unsigned)(0x7fffffff - e);
}

__device__ __forceinline__ float lane_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One warp per token; lane l holds experts l, l + 32, ... Bound by latency (K rounds of a warp maximum).
template <int PER>
__global__ void __launch_bounds__(256) route_kernel(const __nv_bfloat16* __restrict__ logits, const float* __restrict__ bias, float* __restrict__ w,
                                                    int32_t* __restrict__ topk, int32_t* __restrict__ tpe, float* __restrict__ probs, int S, int E, int K) {
  __shared__ int s_cnt[kRouteMaxE];
  for (int e = threadIdx.x; e < E; e += blockDim.x) s_cnt[e] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s < S; s += gridDim.x * (blockDim.x >> 5)) {
    float v[PER], top = -INFINITY, sum = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = i * 32 + lane;
      v[i] = e < E ? __bfloat162float(logits[(size_t)s * E + e]) + bias[e] : -INFINITY;
      top = fmaxf(top, v[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
#pragma unroll
    for (int i = 0; i < PER; ++i) { v[i] = expf(v[i] - top); sum += v[i]; }
    sum = lane_sum(sum);
    unsigned long long best = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = i * 32 + lane;
      v[i] = v[i] / sum;
      if (e < E) {
        best = max(best, route_key(v[i], e));
        if (probs) probs[(size_t)s * E + e] = v[i];
      }
    }
    unsigned taken = 0;                      // bit i: expert i * 32 + lane is chosen
    float mine = 0.f;                        // lane k: the k-th largest probability
    int mine_e = 0;
    for (int k = 0; k < K; ++k) {
      unsigned long long m = best;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      const int e = 0x7fffffff - (int)(unsigned)m;
      float p = 0.f;
#pragma unroll
      for (int i = 0; i < PER; ++i) if ((e >> 5) == i) p = v[i];
      p = __shfl_sync(0xffffffffu, p, e & 31);
      if (lane == k) { mine = p; mine_e = e; }
      if (lane == (e & 31)) {
        taken |= 1u << (e >> 5);
        best = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) if (i * 32 + lane < E && !((taken >> i) & 1u)) best = max(best, route_key(v[i], i * 32 + lane));
      }
    }
    const float total = lane_sum(mine);
    if (lane < K) {
      w[(size_t)s * K + lane] = mine / total;
      topk[(size_t)s * K + lane] = mine_e;
      atomicAdd(&s_cnt[mine_e], 1);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) if (s_cnt[e]) atomicAdd(&tpe[e], s_cnt[e]);
}

// dlogits [S, E] bf16 from dw and topk [S, K] and the probabilities [S, E]; one warp per token. With v the chosen
// probabilities and t their sum: dv_k = dw_k / t - sum_j dw_j v_j / t^2, then the gradient of the softmax.
template <int PER>
__global__ void __launch_bounds__(256) route_bwd_kernel(const float* __restrict__ probs, const float* __restrict__ dw, const int32_t* __restrict__ topk,
                                                        __nv_bfloat16* __restrict__ dlogits, int S, int E, int K) {
  const int lane = threadIdx.x & 31;
  for (int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s < S; s += gridDim.x * (blockDim.x >> 5)) {
    float v = 0.f, g = 0.f; int e = -1;
    if (lane < K) { e = topk[(size_t)s * K + lane]; v = probs[(size_t)s * E + e]; g = dw[(size_t)s * K + lane]; }
    const float t = lane_sum(v);
    const float gs = lane_sum(lane < K ? -g * ((v / t) / t) : 0.f);
    const float dv = g / t + gs;
    float p[PER], d[PER], q = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      p[i] = i * 32 + lane < E ? probs[(size_t)s * E + i * 32 + lane] : 0.f;
      d[i] = 0.f;
    }
    for (int k = 0; k < K; ++k) {
      const int ek = __shfl_sync(0xffffffffu, e, k);
      const float gk = __shfl_sync(0xffffffffu, dv, k);
#pragma unroll
      for (int i = 0; i < PER; ++i) if (ek == i * 32 + lane) d[i] = gk;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) q = __fadd_rn(q, __fmul_rn(d[i], p[i]));
    q = lane_sum(q);
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (i * 32 + lane < E) dlogits[(size_t)s * E + i * 32 + lane] = __float2bfloat16(fmaf(-p[i], q, __fmul_rn(d[i], p[i])));
  }
}

// act = bf16(silu(gate)) * up for a dense [rows, 2n] matrix (gate | up), and its gradient: the shared expert's activation,
// with the roundings of the two operators it stands for
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16(x)); }

__global__ void __launch_bounds__(256) swiglu_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act, int64_t n8, int vec) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / vec; const int v = (int)(i - r * vec);
    const int4 xg = ld_nc_v4(gu + (r * 2 * vec + v) * 8), xu = ld_nc_v4(gu + (r * 2 * vec + vec + v) * 8);
    const __nv_bfloat16 *pg = reinterpret_cast<const __nv_bfloat16*>(&xg), *pu = reinterpret_cast<const __nv_bfloat16*>(&xu);
    int4 o; __nv_bfloat16* q = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float g = __bfloat162float(pg[j]);
      q[j] = __float2bfloat16(bf16_round(g / (1.f + expf(-g))) * __bfloat162float(pu[j]));
    }
    st_v4(act + i * 8, o);
  }
}

__global__ void __launch_bounds__(256) swiglu_dense_bwd_kernel(const __nv_bfloat16* __restrict__ dact, const __nv_bfloat16* __restrict__ gu,
                                                               __nv_bfloat16* __restrict__ dgu, int64_t n8, int vec) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / vec; const int v = (int)(i - r * vec);
    const int64_t og = (r * 2 * vec + v) * 8, ou = og + (int64_t)vec * 8;
    const int4 xd = ld_nc_v4(dact + i * 8), xg = ld_nc_v4(gu + og), xu = ld_nc_v4(gu + ou);
    const __nv_bfloat16 *pd = reinterpret_cast<const __nv_bfloat16*>(&xd), *pg = reinterpret_cast<const __nv_bfloat16*>(&xg),
                        *pu = reinterpret_cast<const __nv_bfloat16*>(&xu);
    int4 a, b; __nv_bfloat16 *qa = reinterpret_cast<__nv_bfloat16*>(&a), *qb = reinterpret_cast<__nv_bfloat16*>(&b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float d = __bfloat162float(pd[j]), g = __bfloat162float(pg[j]), u = __bfloat162float(pu[j]);
      const float sig = 1.f / (1.f + expf(-g));
      const float ds = bf16_round(d * u);
      qa[j] = __float2bfloat16(ds * sig * (1.f + g * (1.f - sig)));
      qb[j] = __float2bfloat16(d * bf16_round(g / (1.f + expf(-g))));
    }
    st_v4(dgu + og, a);
    st_v4(dgu + ou, b);
  }
}

}  // namespace mep

extern "C" int mep_route_max_experts() { return mep::kRouteMaxE; }

extern "C" int mep_route(const void* logits, const float* bias, float* w, int32_t* topk, int32_t* tpe, float* probs, int S, int E, int K,
                         cudaStream_t stream) {
  using namespace mep;
  MEP_REQUIRE(E <= kRouteMaxE && K <= 32 && K <= E, "route: E=%d, K=%d not supported", E, K);
  MEP_CUDA_CHECK(cudaMemsetAsync(tpe, 0, (size_t)E * 4, stream));
  const dim3 grid((S + 7) / 8 < 592 ? (S + 7) / 8 : 592), block(256);
  const __nv_bfloat16* l = (const __nv_bfloat16*)logits;
  if (E <= 32) return launch_plain(route_kernel<1>, grid, block, 0, stream, l, bias, w, topk, tpe, probs, S, E, K);
  if (E <= 64) return launch_plain(route_kernel<2>, grid, block, 0, stream, l, bias, w, topk, tpe, probs, S, E, K);
  if (E <= 128) return launch_plain(route_kernel<4>, grid, block, 0, stream, l, bias, w, topk, tpe, probs, S, E, K);
  if (E <= 256) return launch_plain(route_kernel<8>, grid, block, 0, stream, l, bias, w, topk, tpe, probs, S, E, K);
  return launch_plain(route_kernel<16>, grid, block, 0, stream, l, bias, w, topk, tpe, probs, S, E, K);
}

extern "C" int mep_route_bwd(const float* probs, const float* dw, const int32_t* topk, void* dlogits, int S, int E, int K, cudaStream_t stream) {
  using namespace mep;
  const dim3 grid((S + 7) / 8 < 592 ? (S + 7) / 8 : 592), block(256);
  __nv_bfloat16* d = (__nv_bfloat16*)dlogits;
  if (E <= 32) return launch_plain(route_bwd_kernel<1>, grid, block, 0, stream, probs, dw, topk, d, S, E, K);
  if (E <= 64) return launch_plain(route_bwd_kernel<2>, grid, block, 0, stream, probs, dw, topk, d, S, E, K);
  if (E <= 128) return launch_plain(route_bwd_kernel<4>, grid, block, 0, stream, probs, dw, topk, d, S, E, K);
  if (E <= 256) return launch_plain(route_bwd_kernel<8>, grid, block, 0, stream, probs, dw, topk, d, S, E, K);
  return launch_plain(route_bwd_kernel<16>, grid, block, 0, stream, probs, dw, topk, d, S, E, K);
}

static int dense_grid(int64_t n8) { return (int)((n8 + 255) / 256 < 1184 ? (n8 + 255) / 256 : 1184); }

extern "C" int mep_swiglu(const void* gu, void* act, int64_t rows, int n, cudaStream_t stream) {
  MEP_REQUIRE(n % 8 == 0, "swiglu: inner size %d must be a multiple of 8", n);
  const int64_t n8 = rows * (n / 8);
  return mep::launch_plain(mep::swiglu_kernel, dim3(dense_grid(n8)), dim3(256), 0, stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)act, n8, n / 8);
}

extern "C" int mep_swiglu_dense_bwd(const void* dact, const void* gu, void* dgu, int64_t rows, int n, cudaStream_t stream) {
  MEP_REQUIRE(n % 8 == 0, "swiglu: inner size %d must be a multiple of 8", n);
  const int64_t n8 = rows * (n / 8);
  return mep::launch_plain(mep::swiglu_dense_bwd_kernel, dim3(dense_grid(n8)), dim3(256), 0, stream, (const __nv_bfloat16*)dact, (const __nv_bfloat16*)gu,
                           (__nv_bfloat16*)dgu, n8, n / 8);
}
