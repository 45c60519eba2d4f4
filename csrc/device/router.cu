// Router of a MoE block around the gate GEMM: bias, softmax over the experts, top-k, renormalised weights and the
// expert histogram in one launch, and the gradient of the logits in another. As torch operators this took ten
// launches forward and twelve backward, most of them shorter than their launch.
//
// The softmax over all experts cancels when the k largest probabilities are renormalised: w_k = exp(l_k - l_max) / sum
// over the chosen ones, and only their logits have a gradient, dl_k = w_k (dw_k - sum_j w_j dw_j).
#include "prims.cuh"
#include "../host/launch.h"

namespace mep {

constexpr int kRouteMaxE = 512;

// Sort key of (logit, expert): larger first, NaN largest (as torch.topk), lower expert on ties. Never 0.
__device__ __forceinline__ unsigned long long route_key(float v, int e) {
  unsigned b = __float_as_uint(v);
  b = v != v ? 0xffffffffu : (b & 0x80000000u) ? ~b : b | 0x80000000u;
  return ((unsigned long long)b << 32) | (unsigned)(0x7fffffff - e);
}

// One warp per token; lane l holds experts l, l + 32, ... Bound by latency (K rounds of a warp maximum).
template <int PER>
__global__ void __launch_bounds__(256) route_kernel(const __nv_bfloat16* __restrict__ logits, const float* __restrict__ bias, float* __restrict__ w,
                                                    int32_t* __restrict__ topk, int32_t* __restrict__ tpe, int S, int E, int K) {
  __shared__ int s_cnt[kRouteMaxE];
  for (int e = threadIdx.x; e < E; e += blockDim.x) s_cnt[e] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s < S; s += gridDim.x * (blockDim.x >> 5)) {
    float v[PER];
    unsigned long long best = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = i * 32 + lane;
      v[i] = e < E ? __bfloat162float(logits[(size_t)s * E + e]) + bias[e] : 0.f;
      if (e < E) best = max(best, route_key(v[i], e));
    }
    unsigned taken = 0;                      // bit i: expert i * 32 + lane is chosen
    float mine = 0.f, top = 0.f, sum = 0.f;  // lane k: the k-th chosen logit, then its weight
    int mine_e = 0;
    for (int k = 0; k < K; ++k) {
      unsigned long long m = best;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      const int e = 0x7fffffff - (int)(unsigned)m;
      float l = 0.f;
#pragma unroll
      for (int i = 0; i < PER; ++i) if ((e >> 5) == i) l = v[i];
      l = __shfl_sync(0xffffffffu, l, e & 31);
      if (k == 0) top = l;
      const float p = expf(l - top);
      sum += p;
      if (lane == k) { mine = p; mine_e = e; }
      if (lane == (e & 31)) {
        taken |= 1u << (e >> 5);
        best = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) if (i * 32 + lane < E && !((taken >> i) & 1u)) best = max(best, route_key(v[i], i * 32 + lane));
      }
    }
    if (lane < K) {
      w[(size_t)s * K + lane] = mine / sum;
      topk[(size_t)s * K + lane] = mine_e;
      atomicAdd(&s_cnt[mine_e], 1);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) if (s_cnt[e]) atomicAdd(&tpe[e], s_cnt[e]);
}

// dlogits [S, E] bf16 from dw, w, topk [S, K]; one warp per token.
__global__ void __launch_bounds__(256) route_bwd_kernel(const float* __restrict__ w, const float* __restrict__ dw, const int32_t* __restrict__ topk,
                                                        __nv_bfloat16* __restrict__ dlogits, int S, int E, int K) {
  const int lane = threadIdx.x & 31;
  for (int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s < S; s += gridDim.x * (blockDim.x >> 5)) {
    float wk = 0.f, dk = 0.f; int e = -1;
    if (lane < K) { wk = w[(size_t)s * K + lane]; dk = dw[(size_t)s * K + lane]; e = topk[(size_t)s * K + lane]; }
    float dot = wk * dk;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    const float g = wk * (dk - dot);
    for (int e0 = 0; e0 < E; e0 += 32) {
      float out = 0.f;
      for (int k = 0; k < K; ++k) {
        const int ek = __shfl_sync(0xffffffffu, e, k);
        const float gk = __shfl_sync(0xffffffffu, g, k);
        if (ek == e0 + lane) out = gk;
      }
      if (e0 + lane < E) dlogits[(size_t)s * E + e0 + lane] = __float2bfloat16(out);
    }
  }
}

// act = silu(gate) * up for a dense [rows, 2 * Hp] matrix (gate | up): the shared expert's activation
__global__ void __launch_bounds__(256) swiglu_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act, int64_t n8, int vec) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / vec; const int v = (int)(i - r * vec);
    const int4 xg = ld_nc_v4(gu + (r * 2 * vec + v) * 8), xu = ld_nc_v4(gu + (r * 2 * vec + vec + v) * 8);
    const __nv_bfloat162 *pg = reinterpret_cast<const __nv_bfloat162*>(&xg), *pu = reinterpret_cast<const __nv_bfloat162*>(&xu);
    int4 o; __nv_bfloat162* q = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 g = __bfloat1622float2(pg[j]), u = __bfloat1622float2(pu[j]);
      q[j] = __floats2bfloat162_rn(g.x / (1.f + __expf(-g.x)) * u.x, g.y / (1.f + __expf(-g.y)) * u.y);
    }
    st_v4(act + i * 8, o);
  }
}

}  // namespace mep

extern "C" int mep_route_max_experts() { return mep::kRouteMaxE; }

extern "C" int mep_route(const void* logits, const float* bias, float* w, int32_t* topk, int32_t* tpe, int S, int E, int K, cudaStream_t stream) {
  using namespace mep;
  MEP_REQUIRE(E <= kRouteMaxE && K <= 32 && K <= E, "route: E=%d, K=%d not supported", E, K);
  MEP_CUDA_CHECK(cudaMemsetAsync(tpe, 0, (size_t)E * 4, stream));
  const int blocks = (S + 7) / 8 < 592 ? (S + 7) / 8 : 592;
  const __nv_bfloat16* l = (const __nv_bfloat16*)logits;
  if (E <= 32) return launch_plain(route_kernel<1>, dim3(blocks), dim3(256), 0, stream, l, bias, w, topk, tpe, S, E, K);
  if (E <= 64) return launch_plain(route_kernel<2>, dim3(blocks), dim3(256), 0, stream, l, bias, w, topk, tpe, S, E, K);
  if (E <= 128) return launch_plain(route_kernel<4>, dim3(blocks), dim3(256), 0, stream, l, bias, w, topk, tpe, S, E, K);
  if (E <= 256) return launch_plain(route_kernel<8>, dim3(blocks), dim3(256), 0, stream, l, bias, w, topk, tpe, S, E, K);
  return launch_plain(route_kernel<16>, dim3(blocks), dim3(256), 0, stream, l, bias, w, topk, tpe, S, E, K);
}

extern "C" int mep_route_bwd(const float* w, const float* dw, const int32_t* topk, void* dlogits, int S, int E, int K, cudaStream_t stream) {
  const int blocks = (S + 7) / 8 < 592 ? (S + 7) / 8 : 592;
  return mep::launch_plain(mep::route_bwd_kernel, dim3(blocks), dim3(256), 0, stream, w, dw, topk, (__nv_bfloat16*)dlogits, S, E, K);
}

extern "C" int mep_swiglu(const void* gu, void* act, int64_t rows, int Hp, cudaStream_t stream) {
  MEP_REQUIRE(Hp % 8 == 0, "swiglu: inner size %d must be a multiple of 8", Hp);
  const int64_t n8 = rows * (Hp / 8);
  const int64_t blocks = (n8 + 255) / 256 < 1184 ? (n8 + 255) / 256 : 1184;
  return mep::launch_plain(mep::swiglu_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)act, n8, Hp / 8);
}
