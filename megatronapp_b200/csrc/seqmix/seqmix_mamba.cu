// What stands around the Mamba-2 scan between a mixer's two projections, forward and backward: the causal convolution of four steps with
// SiLU, the step sizes' softplus, and the RMS norm of the result gated by SiLU(z), one statistic per group of channels.
//
// All of it reads the input projection's columns [z | x B C | dt] where they lie ([steps, batch, width]) and writes the gradients into one
// tensor of that shape, so nothing is split, transposed, copied or concatenated.  Intermediates stay in fp32 registers; the kernels are
// bound by HBM.  Mixer of width 2048, 2048 steps, training pass: the PyTorch form of these parts took 1.2 ms in 60 launches.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "seq_common.cuh"
#include "seqmix_api.h"

namespace b200seq {
namespace {

using namespace dev;

template <typename T> __device__ __forceinline__ void load4(const T* p, float (&v)[4]);
template <> __device__ __forceinline__ void load4<float>(const float* p, float (&v)[4]) {
  const float4 u = *reinterpret_cast<const float4*>(p);
  v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
}
template <> __device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xffff0000u);
  v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xffff0000u);
}
template <typename T> __device__ __forceinline__ void store4(T* p, const float (&v)[4]);
template <> __device__ __forceinline__ void store4<float>(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <> __device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, const float (&v)[4]) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
}

// ---- convolution.  A thread walks `kRun` steps of four channels with the window in registers.
constexpr int kFwdRun = 16, kBwdRun = 32;        // backward: 32 or a little more, see mamba_conv_run

template <typename T>
__global__ void __launch_bounds__(128) mamba_conv_kernel(const MambaArgs p) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (c >= p.conv) return;
  const int t0 = blockIdx.y * kFwdRun, b = blockIdx.z;
  const T* x = static_cast<const T*>(p.zx) + static_cast<int64_t>(b) * p.width + p.di + c;
  const int64_t step = static_cast<int64_t>(p.b) * p.width;
  T* out = static_cast<T*>(p.xbc) + (static_cast<int64_t>(b) * p.s) * p.conv + c;
  float w[4][4], bias[4], win[4][4];               // w[channel][tap]
#pragma unroll
  for (int e = 0; e < 4; ++e) load4(static_cast<const T*>(p.conv_w) + (c + e) * 4, w[e]);
  load4(static_cast<const T*>(p.conv_b) + c, bias);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int e = 0; e < 4; ++e) win[k + 1][e] = 0.f;
    if (t0 - 3 + k >= 0) load4(x + (t0 - 3 + k) * step, win[k + 1]);
  }
#pragma unroll 4
  for (int i = 0; i < kFwdRun; ++i) {
    const int t = t0 + i;
    if (t >= p.s) break;
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) win[k][e] = win[k + 1][e];
    load4(x + t * step, win[3]);
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float v = bias[e];
#pragma unroll
      for (int k = 0; k < 4; ++k) v = fmaf(w[e][k], win[k][e], v);
      o[e] = v * sigmoidf_(v);
    }
    store4(out + static_cast<int64_t>(t) * p.conv, o);
  }
}

template <typename T>
__global__ void __launch_bounds__(128, 5) mamba_conv_grad_kernel(const MambaArgs p) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (c >= p.conv) return;
  const int run = p.conv_run, t0 = blockIdx.y * run, b = blockIdx.z;
  const int64_t step = static_cast<int64_t>(p.b) * p.width, at = static_cast<int64_t>(b) * p.width + p.di + c;
  const T* x = static_cast<const T*>(p.zx) + at;
  T* dx = static_cast<T*>(p.dzx) + at;
  // the incoming gradient: x, B and C lie in tensors of their own
  const int gn = (p.conv - p.di) / 2;
  const T* dout;
  int64_t dstep;
  if (c < p.di) { dout = static_cast<const T*>(p.dxs) + c; dstep = p.di; }
  else if (c < p.di + gn) { dout = static_cast<const T*>(p.dB) + c - p.di; dstep = gn; }
  else { dout = static_cast<const T*>(p.dC) + c - p.di - gn; dstep = gn; }
  dout += static_cast<int64_t>(b) * p.s * dstep;
  float w[4][4], bias[4], win[4][4], d[4][4], dw[4][4], db[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) load4(static_cast<const T*>(p.conv_w) + (c + e) * 4, w[e]);
  load4(static_cast<const T*>(p.conv_b) + c, bias);
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      win[k][e] = d[k][e] = dw[k][e] = 0.f;
      db[e] = 0.f;
    }
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (t0 - 3 + k >= 0) load4(x + (t0 - 3 + k) * step, win[k + 1]);
#pragma unroll 1
  for (int i = 0; i < run + 3; ++i) {
    const int t = t0 + i;
    float g[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        win[k][e] = win[k + 1][e];
        d[k][e] = d[k + 1][e];
      }
    if (t < p.s) {
      load4(x + t * step, win[3]);
      load4(dout + t * dstep, g);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float v = bias[e];
#pragma unroll
      for (int k = 0; k < 4; ++k) v = fmaf(w[e][k], win[k][e], v);
      const float sg = sigmoidf_(v), pre = g[e] * (sg * fmaf(v, 1.f - sg, 1.f));
      d[3][e] = t < p.s ? pre : 0.f;
      if (i < run) {
#pragma unroll
        for (int k = 0; k < 4; ++k) dw[k][e] = fmaf(d[3][e], win[k][e], dw[k][e]);
        db[e] += d[3][e];
      }
    }
    // step t - 3 has now seen the four outputs that it enters
    if (i >= 3 && t - 3 < p.s) {
      float o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = fmaf(w[e][3], d[0][e], fmaf(w[e][2], d[1][e], fmaf(w[e][1], d[2][e], w[e][0] * d[3][e])));
      store4(dx + (t - 3) * step, o);
    }
  }
  float* part = p.conv_part + (static_cast<int64_t>(b) * gridDim.y + blockIdx.y) * 5 * p.conv + c;
#pragma unroll
  for (int k = 0; k < 4; ++k) store4(part + static_cast<int64_t>(k) * p.conv, dw[k]);
  store4(part + static_cast<int64_t>(4) * p.conv, db);
}

// ---- step sizes: dt = softplus(columns + bias), [b, s, heads] fp32
template <typename T, bool kGrad>
__global__ void __launch_bounds__(256) mamba_dt_kernel(const MambaArgs p) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x, n = static_cast<int64_t>(p.b) * p.s * p.heads;
  if (i >= n) return;
  const int h = static_cast<int>(i % p.heads);
  const int64_t row = i / p.heads;
  const int t = static_cast<int>(row % p.s), b = static_cast<int>(row / p.s);
  const int64_t at = (static_cast<int64_t>(t) * p.b + b) * p.width + p.di + p.conv + h;
  const float v = ld(static_cast<const T*>(p.zx) + at) + p.dt_bias[h];
  if (!kGrad) {
    p.dt[i] = v > 20.f ? v : log1pf(expf(v));
  } else {
    const float d = p.ddt[i] * (v > 20.f ? 1.f : sigmoidf_(v));
    p.ddt[i] = d;
    st(static_cast<T*>(p.dzx) + at, d);
  }
}

// ---- gated norm: u = y silu(z), out = u / sqrt(mean_group(u^2) + eps) * w.  One warp per (step, batch, group).
template <typename T>
__global__ void __launch_bounds__(128) mamba_norm_kernel(const MambaArgs p) {
  const int64_t item = static_cast<int64_t>(blockIdx.x) * 4 + (threadIdx.x >> 5), n = static_cast<int64_t>(p.s) * p.b * p.groups;
  if (item >= n) return;
  const int lane = threadIdx.x & 31, W = p.di / p.groups, g = static_cast<int>(item % p.groups);
  const int64_t row = item / p.groups;             // t * b + batch
  const int t = static_cast<int>(row / p.b), b = static_cast<int>(row % p.b);
  const T* y = static_cast<const T*>(p.y) + (static_cast<int64_t>(b) * p.s + t) * p.di + g * W;
  const T* z = static_cast<const T*>(p.zx) + row * p.width + g * W;
  float s = 0.f;
#pragma unroll 4
  for (int c = lane * 4; c < W; c += 128) {
    float yv[4], zv[4];
    load4(y + c, yv);
    load4(z + c, zv);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float u = yv[e] * zv[e] * sigmoidf_(zv[e]);
      s = fmaf(u, u, s);
    }
  }
  s = warp_sum(s);
  const float r = rsqrtf(s / W + p.eps);
  if (lane == 0) p.rstd[item] = r;
  const T* w = static_cast<const T*>(p.norm_w) + g * W;
  T* out = static_cast<T*>(p.out) + row * p.di + g * W;
#pragma unroll 4
  for (int c = lane * 4; c < W; c += 128) {
    float yv[4], zv[4], wv[4], o[4];
    load4(y + c, yv);
    load4(z + c, zv);
    load4(w + c, wv);
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = yv[e] * zv[e] * sigmoidf_(zv[e]) * r * wv[e];
    store4(out + c, o);
  }
}

// four warps of a CTA share kNormRows rows of one group; kVec: groups of four channels per lane
constexpr int kNormRows = 16;      // four to a warp, each two dependent passes: latency, so many CTAs (2048 x 4096: 52 us with 32 rows, 33 with 16)
template <typename T, int kVec>
__global__ void __launch_bounds__(128) mamba_norm_grad_kernel(const MambaArgs p) {
  extern __shared__ float s_dw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = p.di / p.groups, g = blockIdx.y;
  const int64_t n_rows = static_cast<int64_t>(p.s) * p.b;
  const T* w = static_cast<const T*>(p.norm_w) + g * W;
  float dw[kVec][4];
#pragma unroll
  for (int i = 0; i < kVec; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) dw[i][e] = 0.f;
  for (int k = warp; k < kNormRows; k += 4) {
    const int64_t row = static_cast<int64_t>(blockIdx.x) * kNormRows + k;
    if (row >= n_rows) break;
    const int t = static_cast<int>(row / p.b), b = static_cast<int>(row % p.b);
    const int64_t at_y = (static_cast<int64_t>(b) * p.s + t) * p.di + g * W, at_z = row * p.width + g * W, at_o = row * p.di + g * W;
    const float r = p.rstd[row * p.groups + g];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int c = (i * 32 + lane) * 4;
      if (c < W) {
        float yv[4], zv[4], wv[4], gv[4];
        load4(static_cast<const T*>(p.y) + at_y + c, yv);
        load4(static_cast<const T*>(p.zx) + at_z + c, zv);
        load4(w + c, wv);
        load4(static_cast<const T*>(p.dout) + at_o + c, gv);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float u = yv[e] * zv[e] * sigmoidf_(zv[e]);
          dot = fmaf(gv[e] * wv[e], u, dot);
          dw[i][e] = fmaf(gv[e], u * r, dw[i][e]);
        }
      }
    }
    dot = warp_sum(dot) * r * r / W;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int c = (i * 32 + lane) * 4;
      if (c < W) {
        float yv[4], zv[4], wv[4], gv[4], dy[4], dz[4];
        load4(static_cast<const T*>(p.y) + at_y + c, yv);
        load4(static_cast<const T*>(p.zx) + at_z + c, zv);
        load4(w + c, wv);
        load4(static_cast<const T*>(p.dout) + at_o + c, gv);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float sg = sigmoidf_(zv[e]), a = zv[e] * sg, du = r * fmaf(-yv[e] * a, dot, gv[e] * wv[e]);
          dy[e] = du * a;
          dz[e] = du * yv[e] * sg * fmaf(zv[e], 1.f - sg, 1.f);
        }
        store4(static_cast<T*>(p.dy) + at_y + c, dy);
        store4(static_cast<T*>(p.dzx) + at_z + c, dz);
      }
    }
  }
  // the warps add up in turn
  for (int k = 0; k < 4; ++k) {
    if (warp == k) {
#pragma unroll
      for (int i = 0; i < kVec; ++i) {
        const int c = (i * 32 + lane) * 4;
        if (c < W) {
          float v[4] = {dw[i][0], dw[i][1], dw[i][2], dw[i][3]};
          if (k > 0) {
            float o[4];
            load4(s_dw + c, o);
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] += o[e];
          }
          store4(k < 3 ? s_dw + c : p.norm_part + (static_cast<int64_t>(blockIdx.x) * p.groups + g) * W + c, v);
        }
      }
    }
    __syncthreads();
  }
}

template <typename T>
void norm_grad(const MambaArgs& p, cudaStream_t s) {
  const int W = p.di / p.groups, vec = (W / 4 + 31) / 32;
  const dim3 grid(mamba_norm_parts(p.s, p.b), p.groups);
  const int smem = W * 4;
  if (vec <= 1) mamba_norm_grad_kernel<T, 1><<<grid, 128, smem, s>>>(p);
  else if (vec <= 2) mamba_norm_grad_kernel<T, 2><<<grid, 128, smem, s>>>(p);
  else if (vec <= 4) mamba_norm_grad_kernel<T, 4><<<grid, 128, smem, s>>>(p);
  else if (vec <= 8) mamba_norm_grad_kernel<T, 8><<<grid, 128, smem, s>>>(p);
  else if (vec <= 16) mamba_norm_grad_kernel<T, 16><<<grid, 128, smem, s>>>(p);
  else mamba_norm_grad_kernel<T, 32><<<grid, 128, smem, s>>>(p);
}

template <typename T>
void before_scan(const MambaArgs& p, cudaStream_t s) {
  const int64_t n = static_cast<int64_t>(p.b) * p.s * p.heads;
  mamba_conv_kernel<T><<<dim3((p.conv / 4 + 127) / 128, (p.s + kFwdRun - 1) / kFwdRun, p.b), 128, 0, s>>>(p);
  mamba_dt_kernel<T, false><<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(p);
}
template <typename T>
void before_scan_grad(const MambaArgs& p, cudaStream_t s) {
  const int64_t n = static_cast<int64_t>(p.b) * p.s * p.heads;
  mamba_conv_grad_kernel<T><<<dim3((p.conv / 4 + 127) / 128, mamba_conv_parts(p.s, p.conv_run), p.b), 128, 0, s>>>(p);
  mamba_dt_kernel<T, true><<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(p);
}
template <typename T>
void norm(const MambaArgs& p, cudaStream_t s) {
  const int64_t n = static_cast<int64_t>(p.s) * p.b * p.groups;
  mamba_norm_kernel<T><<<static_cast<unsigned>((n + 3) / 4), 128, 0, s>>>(p);
}

}  // namespace

// Steps of a backward run.  A CTA takes long for what it does (35 dependent steps), so a last wave of a few CTAs costs as much as a full one:
// the runs are lengthened until the last full wave holds them all (2048 steps x 6144 channels: 768 CTAs on 592 places 73 us, 588 with runs
// of 42 steps 50; 96 registers instead of 104 make it 740 places, and 732 CTAs with runs of 34 steps take 44).
int mamba_conv_run(int steps, int batch, int conv, bool bf16) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bf16 ? mamba_conv_grad_kernel<__nv_bfloat16> : mamba_conv_grad_kernel<float>, 128, 0) != cudaSuccess)
    return kBwdRun;
  const int64_t rows = static_cast<int64_t>((conv / 4 + 127) / 128) * batch, ctas = rows * ((steps + kBwdRun - 1) / kBwdRun);
  const int64_t places = static_cast<int64_t>(sms) * per_sm, parts = ctas / (places > 0 ? places : 1) * places / rows;
  return parts < 1 ? kBwdRun : static_cast<int>((steps + parts - 1) / parts < kBwdRun ? kBwdRun : (steps + parts - 1) / parts);
}
int mamba_conv_parts(int steps, int run) { return (steps + run - 1) / run; }
int mamba_norm_parts(int steps, int batch) { return static_cast<int>((static_cast<int64_t>(steps) * batch + kNormRows - 1) / kNormRows); }

void mamba_before_scan(const MambaArgs& p, bool bf16, cudaStream_t s) { bf16 ? before_scan<__nv_bfloat16>(p, s) : before_scan<float>(p, s); }
void mamba_before_scan_grad(const MambaArgs& p, bool bf16, cudaStream_t s) { bf16 ? before_scan_grad<__nv_bfloat16>(p, s) : before_scan_grad<float>(p, s); }
void mamba_gated_norm(const MambaArgs& p, bool bf16, cudaStream_t s) { bf16 ? norm<__nv_bfloat16>(p, s) : norm<float>(p, s); }
void mamba_gated_norm_grad(const MambaArgs& p, bool bf16, cudaStream_t s) { bf16 ? norm_grad<__nv_bfloat16>(p, s) : norm_grad<float>(p, s); }

}  // namespace b200seq
