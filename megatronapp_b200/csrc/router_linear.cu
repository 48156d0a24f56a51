// Gradients of a mixture of experts' router logits: products with a handful of columns on one side, fp32 sums of 16-bit tokens and 16-bit or
// fp32 weights.  With so few columns the tokens' bytes are the bound, so they are read once, in 16 bits, and never widened in memory.
//   dx: a thread takes eight columns of eight tokens and walks the experts.
//   dw: a thread takes eight columns of eight experts and walks its CTA's share of the tokens; a second kernel adds the shares in order.
// The logits themselves stay the library's fp32 product of widened operands: experts of a token can lie within the rounding of a sum of each
// other, and sums in another order then choose other ones (one token of 4096 in a layer of 8 experts, whose output changes entirely).
// Forward and backward, us, with library products / with these gradients: 4096 tokens x 2048, 8 experts 147 / 73; 4096 x 4096, 32 experts
// 257 / 237; 16384 x 4096, 32 experts 662 / 625; 512 x 1024, 8 experts 33 / 29.  With 64 experts the products are work for larger tiles, so 32
// is the most that comes this way.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "b200_api.h"
#include "common.cuh"

namespace b200 {
namespace {

constexpr int kE = 8;             // experts of a pass
constexpr int kTokDx = 8, kSumGroups = 8;

__device__ __forceinline__ void get8(const float* p, float (&v)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <typename T2, float2 (*kWiden)(T2), typename T>
__device__ __forceinline__ void get8_16(const T* p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = kWiden(*reinterpret_cast<const T2*>(&w[i]));
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ float2 wide_bf16(__nv_bfloat162 v) { return __bfloat1622float2(v); }
__device__ __forceinline__ float2 wide_f16(__half2 v) { return __half22float2(v); }
__device__ __forceinline__ void get8(const __nv_bfloat16* p, float (&v)[8]) { get8_16<__nv_bfloat162, wide_bf16>(p, v); }
__device__ __forceinline__ void get8(const __half* p, float (&v)[8]) { get8_16<__half2, wide_f16>(p, v); }
__device__ __forceinline__ void put8(float* p, const float (&v)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
template <typename T2, T2 (*kNarrow)(float, float), typename T>
__device__ __forceinline__ void put8_16(T* p, const float (&v)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    T2 t = kNarrow(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<uint32_t*>(&t);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ __nv_bfloat162 narrow_bf16(float a, float b) { return __floats2bfloat162_rn(a, b); }
__device__ __forceinline__ __half2 narrow_f16(float a, float b) { return __floats2half2_rn(a, b); }
__device__ __forceinline__ void put8(__nv_bfloat16* p, const float (&v)[8]) { put8_16<__nv_bfloat162, narrow_bf16>(p, v); }
__device__ __forceinline__ void put8(__half* p, const float (&v)[8]) { put8_16<__half2, narrow_f16>(p, v); }

__device__ __forceinline__ void put4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void put4(__nv_bfloat16* p, float4 v) {
  reinterpret_cast<__nv_bfloat162*>(p)[0] = narrow_bf16(v.x, v.y);
  reinterpret_cast<__nv_bfloat162*>(p)[1] = narrow_bf16(v.z, v.w);
}
__device__ __forceinline__ void put4(__half* p, float4 v) {
  reinterpret_cast<__half2*>(p)[0] = narrow_f16(v.x, v.y);
  reinterpret_cast<__half2*>(p)[1] = narrow_f16(v.z, v.w);
}

template <typename T, typename W>
__global__ void __launch_bounds__(128) router_dx_kernel(const float* __restrict__ dl, const W* __restrict__ w, T* __restrict__ dx, int n, int h, int e_all) {
  __shared__ float s_dl[kRouterExperts][kTokDx];
  const int c = (blockIdx.y * 128 + threadIdx.x) * 8, t0 = blockIdx.x * kTokDx;
  for (int i = threadIdx.x; i < e_all * kTokDx; i += 128) {
    const int k = i / e_all, e = i % e_all;
    s_dl[e][k] = t0 + k < n ? dl[static_cast<int64_t>(t0 + k) * e_all + e] : 0.f;
  }
  __syncthreads();
  if (c >= h) return;
  float acc[kTokDx][8] = {};
#pragma unroll 8
  for (int e = 0; e < e_all; ++e) {
    float wv[8];
    get8(w + static_cast<int64_t>(e) * h + c, wv);
#pragma unroll
    for (int k = 0; k < kTokDx; ++k)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[k][q] = fmaf(s_dl[e][k], wv[q], acc[k][q]);
  }
#pragma unroll
  for (int k = 0; k < kTokDx; ++k)
    if (t0 + k < n) put8(dx + static_cast<int64_t>(t0 + k) * h + c, acc[k]);
}

// part[share][e][h]
template <typename T>
__global__ void __launch_bounds__(128) router_dw_kernel(const float* __restrict__ dl, const T* __restrict__ x, float* __restrict__ part, int n, int h, int e_all,
                                                        int per_share) {
  __shared__ float s_dl[32][kE];
  const int c = (blockIdx.x * 128 + threadIdx.x) * 8, e0 = blockIdx.z * kE, first = blockIdx.y * per_share, last = min(n, first + per_share);
  float acc[kE][8] = {};
  for (int t0 = first; t0 < last; t0 += 32) {
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * kE; i += 128) {
      const int t = t0 + i / kE, e = e0 + i % kE;
      s_dl[i / kE][i % kE] = t < last && e < e_all ? dl[static_cast<int64_t>(t) * e_all + e] : 0.f;
    }
    __syncthreads();
    if (c < h) {
      const int m = min(32, last - t0);
#pragma unroll 8
      for (int i = 0; i < m; ++i) {
        float xv[8];
        get8(x + static_cast<int64_t>(t0 + i) * h + c, xv);
#pragma unroll
        for (int e = 0; e < kE; ++e)
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[e][q] = fmaf(s_dl[i][e], xv[q], acc[e][q]);
      }
    }
  }
  if (c >= h) return;
#pragma unroll
  for (int e = 0; e < kE; ++e)
    if (e0 + e < e_all) put8(part + (static_cast<int64_t>(blockIdx.y) * e_all + e0 + e) * h + c, acc[e]);
}

template <typename W>
__global__ void __launch_bounds__(32 * kSumGroups) router_dw_sum_kernel(const float* __restrict__ part, W* __restrict__ dw, int shares, int64_t size) {
  __shared__ float4 s_acc[kSumGroups][32];
  const int lane = threadIdx.x & 31, group = threadIdx.x >> 5;
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * 32 + lane) * 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i < size) {
#pragma unroll 16
    for (int k = group; k < shares; k += kSumGroups) {
      const float4 v = *reinterpret_cast<const float4*>(part + k * size + i);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
  }
  s_acc[group][lane] = acc;
  __syncthreads();
  if (group > 0 || i >= size) return;
#pragma unroll
  for (int k = 1; k < kSumGroups; ++k) {
    const float4 v = s_acc[k][lane];
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  put4(dw + i, acc);
}

template <typename T, typename W>
void run(const RouterArgs& a, cudaStream_t s) {
  const T* x = static_cast<const T*>(a.x);
  const W* w = static_cast<const W*>(a.w);
  const int groups = (a.experts + kE - 1) / kE, octets = (a.h / 8 + 127) / 128;
  if (a.dx != nullptr) router_dx_kernel<T, W><<<dim3((a.n + kTokDx - 1) / kTokDx, octets), 128, 0, s>>>(a.dlogits, w, static_cast<T*>(a.dx), a.n, a.h, a.experts);
  if (a.dw != nullptr) {
    const int shares = router_shares(a.n), per = (a.n + shares - 1) / shares;
    router_dw_kernel<T><<<dim3(octets, shares, groups), 128, 0, s>>>(a.dlogits, x, a.part, a.n, a.h, a.experts, per);
    const int64_t size = static_cast<int64_t>(a.experts) * a.h;
    router_dw_sum_kernel<W><<<static_cast<unsigned>((size / 4 + 31) / 32), 32 * kSumGroups, 0, s>>>(a.part, static_cast<W*>(a.dw), shares, size);
  }
}

}  // namespace

// 32 tokens a share until there are 128 shares
int router_shares(int n) { return n >= 32 * 128 ? 128 : (n + 31) / 32; }

void router_linear_grad(const RouterArgs& a, cudaStream_t s) {
  if (a.bf16) {
    if (a.w_f32) run<__nv_bfloat16, float>(a, s);
    else run<__nv_bfloat16, __nv_bfloat16>(a, s);
  } else {
    if (a.w_f32) run<__half, float>(a, s);
    else run<__half, __half>(a, s);
  }
}

}  // namespace b200
