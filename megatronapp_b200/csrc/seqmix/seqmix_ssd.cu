// Mamba-2 state-space scan in blocks of 64 steps, forward and backward, everything in fp32:
//
//   S_t = exp(dt_t A) S_{t-1} + dt_t x_t B_t^T,   y_t = S_t C_t + D x_t          (per head; B and C per group of heads)
//
// Within a block (cum_t: running sum of dt A)
//   y_t = sum_{u <= t} exp(cum_t - cum_u) (C_t . B_u) dt_u x_u + exp(cum_t) S C_t + D x_t
// so the work is small products of 64-row tiles.  Forward: the scores C B^T once per group, what every block adds to the state, a pass over
// the blocks that turns this into the state each block starts from, and the outputs.  Backward: the same two state kernels for the
// gradient that enters each block's starting state, walked in reverse, then one kernel for all gradients of a block, whose CTA walks the
// heads of a group so that the gradients of B and C add up in registers.  Exponents above the diagonal are never taken (they can overflow).
//
// fp32 inputs: tiles in fp32 in shared memory, 4 x 4 or 4 x 8 results per thread, bound by fp32 multiply-adds (2.1 M per head and block
// backward, 1.3 M forward) and the shared-memory reads that feed them.  bf16 inputs: block states, outputs and gradients on the tensor
// instructions (64 heads x 2048 steps x 64 x 128: outputs 140 -> 56 us, states 57 -> 34 and 59 -> 34, gradients 383 -> 191; errors of the final
// state, the gradients of dt and of the initial state 1.8e-7, 3.2e-7 and 1.2e-7 of their size at 65 steps, with multiply-adds 1.9e-7, 3.5e-7
// and 1.9e-7).  The block-by-block PyTorch form took some 2900 launches and 14 ms of
// device time for 64 heads x 2048 steps.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "seq_common.cuh"
#include "seqmix_api.h"

namespace b200seq {
namespace {

constexpr int kT = 64;          // steps of a block
constexpr int kP = 64;          // head width
constexpr int kPitchT = kT + 4;  // padded rows: 16-byte aligned, conflict-free when 8 threads read 8 rows
constexpr int kThreads = 256;

template <typename T> __device__ __forceinline__ float4 ld4(const T* p);
template <> __device__ __forceinline__ float4 ld4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 ld4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
template <typename T> __device__ __forceinline__ void st4(T* p, float4 v);
template <> __device__ __forceinline__ void st4<float>(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
template <> __device__ __forceinline__ void st4<__nv_bfloat16>(__nv_bfloat16* p, float4 v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
}

// acc[i][j] += sum_k A(m_i, k) B(n_j, k).  An operand lies with k contiguous (X[m][k]; the thread's rows are t, t + 16, ...) or with
// its own index contiguous (X[k][m]; groups of four: 4 t .. 4 t + 3, then 64 further on)
template <int MI, int NI, bool AK, bool BK>
__device__ __forceinline__ void mm(float (&acc)[MI][NI], const float* A, int pa, const float* B, int pb, int K, int ty, int tx) {
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    float a[MI][4], b[NI][4];
    if constexpr (AK) {
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(A + (ty + 16 * i) * pa + k);
        a[i][0] = v.x; a[i][1] = v.y; a[i][2] = v.z; a[i][3] = v.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < MI / 4; ++q)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const float4 v = *reinterpret_cast<const float4*>(A + (k + kk) * pa + q * 64 + ty * 4);
          a[q * 4][kk] = v.x; a[q * 4 + 1][kk] = v.y; a[q * 4 + 2][kk] = v.z; a[q * 4 + 3][kk] = v.w;
        }
    }
    if constexpr (BK) {
#pragma unroll
      for (int j = 0; j < NI; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(B + (tx + 16 * j) * pb + k);
        b[j][0] = v.x; b[j][1] = v.y; b[j][2] = v.z; b[j][3] = v.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < NI / 4; ++q)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const float4 v = *reinterpret_cast<const float4*>(B + (k + kk) * pb + q * 64 + tx * 4);
          b[q * 4][kk] = v.x; b[q * 4 + 1][kk] = v.y; b[q * 4 + 2][kk] = v.z; b[q * 4 + 3][kk] = v.w;
        }
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) acc[i][j] = fmaf(a[i][kk], b[j][kk], acc[i][j]);
  }
}
template <int MI, int NI>
__device__ __forceinline__ void zero(float (&a)[MI][NI]) {
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j) a[i][j] = 0.f;
}
__device__ __forceinline__ float half_warp_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// column of result j of a thread whose operand has its own index contiguous
__device__ __forceinline__ int col4(int t, int j) { return (j >> 2) * 64 + t * 4 + (j & 3); }

// 64 rows of W columns into padded fp32 rows; rows from `rows` on are zeros.  f(row): factor of the row
template <int W, int kBy = kThreads, typename T, typename F>
__device__ __forceinline__ void load_rows(float* dst, int pitch, const T* src, int64_t stride, int rows, F f) {
#pragma unroll 8
  for (int i = threadIdx.x & (kBy - 1); i < kT * (W / 4); i += kBy) {
    const int r = i / (W / 4), c = (i % (W / 4)) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) {
      v = ld4(src + r * stride + c);
      const float s = f(r);
      v.x *= s; v.y *= s; v.z *= s; v.w *= s;
    }
    *reinterpret_cast<float4*>(dst + r * pitch + c) = v;
  }
}
struct One { __device__ float operator()(int) const { return 1.f; } };

// dt and the running sum of dt * A of one block (dt = 0 from `rows` on); all threads call it.  The sum goes step by step: neighbours then share
// what was rounded before them, and the exponentials of their differences keep it out (a scan over the lanes left 2^-24 of the sum in each).
__device__ __forceinline__ void block_decay(float* s_dt, float* s_cum, const float* dt, int64_t stride, int rows, float a) {
  if (threadIdx.x < 32) {
    const int l = threadIdx.x;
    const float d0 = l < rows ? dt[l * stride] : 0.f, d1 = l + 32 < rows ? dt[(l + 32) * stride] : 0.f;
    s_dt[l] = d0;
    s_dt[l + 32] = d1;
    s_cum[l] = d0 * a;
    s_cum[l + 32] = d1 * a;
    __syncwarp();
    if (l == 0) {
      float run = 0.f;
#pragma unroll 1
      for (float4* q = reinterpret_cast<float4*>(s_cum); q < reinterpret_cast<float4*>(s_cum + kT); q += 4) {
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = q[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          run += v[i].x; v[i].x = run;
          run += v[i].y; v[i].y = run;
          run += v[i].z; v[i].z = run;
          run += v[i].w; v[i].w = run;
          q[i] = v[i];
        }
      }
    }
  }
  __syncthreads();
}

// scores of a group's block: G[t][u] = C_t . B_u
template <int N, typename T>
__global__ void __launch_bounds__(kThreads) ssd_scores_kernel(const SsdArgs p) {
  extern __shared__ __align__(16) float sm[];
  constexpr int kPitchN = N + 4;
  float *sC = sm, *sB = sm + kT * kPitchN;
  const int c = blockIdx.x, g = blockIdx.y, b = blockIdx.z, t0 = c * kT, rows = min(kT, p.l - t0);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  load_rows<N>(sC, kPitchN, static_cast<const T*>(p.C) + b * p.c_sb + t0 * p.c_sl + g * N, p.c_sl, rows, One{});
  load_rows<N>(sB, kPitchN, static_cast<const T*>(p.B) + b * p.b_sb + t0 * p.b_sl + g * N, p.b_sl, rows, One{});
  __syncthreads();
  float acc[4][4];
  zero(acc);
  mm<4, 4, true, true>(acc, sC, kPitchN, sB, kPitchN, N, ty, tx);
  float* out = p.scores + ((static_cast<int64_t>(b) * p.n_chunks + c) * p.g + g) * (kT * kT);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) out[(ty + 16 * i) * kT + tx + 16 * j] = acc[i][j];
}

// kGrad = false: what a block adds to the state, sum_u exp(cum_end - cum_u) dt_u x_u B_u^T
// kGrad = true : what its outputs' gradients put on its starting state, sum_t exp(cum_t) dy_t C_t^T
template <int N, typename T, bool kGrad>
__global__ void __launch_bounds__(kThreads) ssd_state_kernel(const SsdArgs p) {
  extern __shared__ __align__(16) float sm[];
  constexpr int kPitchN = N + 4;
  float *sX = sm, *sB = sX + kT * kPitchT, *s_dt = sB + kT * kPitchN, *s_cum = s_dt + kT;
  const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z, t0 = c * kT, rows = min(kT, p.l - t0), g = h / (p.h / p.g);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  block_decay(s_dt, s_cum, p.dt + (static_cast<int64_t>(b) * p.l + t0) * p.h + h, p.h, rows, p.A[h]);
  const float end = s_cum[kT - 1];
  if constexpr (kGrad) {
    load_rows<kP>(sX, kPitchT, static_cast<const T*>(p.dy) + ((static_cast<int64_t>(b) * p.l + t0) * p.h + h) * kP, static_cast<int64_t>(p.h) * kP, rows,
                  [&](int r) { return expf(s_cum[r]); });
    load_rows<N>(sB, kPitchN, static_cast<const T*>(p.C) + b * p.c_sb + t0 * p.c_sl + g * N, p.c_sl, rows, One{});
  } else {
    load_rows<kP>(sX, kPitchT, static_cast<const T*>(p.x) + b * p.x_sb + t0 * p.x_sl + h * kP, p.x_sl, rows,
                  [&](int r) { return expf(end - s_cum[r]) * s_dt[r]; });
    load_rows<N>(sB, kPitchN, static_cast<const T*>(p.B) + b * p.b_sb + t0 * p.b_sl + g * N, p.b_sl, rows, One{});
    if (threadIdx.x == 0) p.decay[(static_cast<int64_t>(b) * p.h + h) * p.n_chunks + c] = expf(end);
  }
  __syncthreads();
  float acc[4][N / 16];
  zero(acc);
  mm<4, N / 16, false, false>(acc, sX, kPitchT, sB, kPitchN, kT, ty, tx);
  float* out = (kGrad ? p.dstates : p.states) + ((static_cast<int64_t>(b) * p.h + h) * p.n_chunks + c) * (kP * N);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < N / 64; ++q)
      *reinterpret_cast<float4*>(out + (ty * 4 + i) * N + q * 64 + tx * 4) = make_float4(acc[i][q * 4], acc[i][q * 4 + 1], acc[i][q * 4 + 2], acc[i][q * 4 + 3]);
}

// ---- bf16 operands on the tensor instructions.  A bf16 operand enters as it is; an fp32 one as three bf16 parts that add up to it exactly
// (truncated, so 8 + 8 + 8 bits and no part overflows).  The products of parts are exact; the first parts' are summed by themselves, since
// these instructions cut their sums off where a multiply-add rounds, and a third of the additions at full size leaves a third of that error.
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t shared_at(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(shared_at(p)) : "memory");
}
__device__ __forceinline__ void ldm4_trans(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(shared_at(p)) : "memory");
}
__device__ __forceinline__ void ldm2_trans(uint32_t& r0, uint32_t& r1, const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(shared_at(p)) : "memory");
}
__device__ __forceinline__ float high_part(float v) { return __uint_as_float(__float_as_uint(v) & 0xffff0000u); }
__device__ __forceinline__ float rest_of(float v, float high) { return v == high ? 0.f : v - high; }   // an infinity has no rest
__device__ __forceinline__ uint32_t pack_high(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }
__device__ __forceinline__ void split3(float x, float y, uint32_t (&part)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    part[i] = pack_high(x, y);
    x = rest_of(x, high_part(x));
    y = rest_of(y, high_part(y));
  }
}
constexpr int kPitchH = 72;                     // bf16 rows of 64, 16 bytes further on in each: ldmatrix without conflicts
constexpr int kPlane = kT * kPitchH;
// 64 rows of W columns as they are
template <int W>
__device__ __forceinline__ void copy_rows(__nv_bfloat16* dst, int pitch, const __nv_bfloat16* src, int64_t stride, int rows) {
#pragma unroll
  for (int k = 0; k < kT * (W / 4) / kThreads; ++k) {
    const int i = (threadIdx.x & (kThreads - 1)) + k * kThreads, r = i / (W / 4), c = (i % (W / 4)) * 4;
    *reinterpret_cast<uint2*>(dst + r * pitch + c) = r < rows ? *reinterpret_cast<const uint2*>(src + r * stride + c) : make_uint2(0u, 0u);
  }
}
__device__ __forceinline__ void store_split(__nv_bfloat16* plane, float4 v) {
  uint32_t lo[3], hi[3];
  split3(v.x, v.y, lo);
  split3(v.z, v.w, hi);
#pragma unroll
  for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(plane + k * kPlane) = make_uint2(lo[k], hi[k]);
}

// ssd_state_kernel for bf16: a warp takes 16 (N = 64: 8) columns n and all 64 rows p
template <int N, bool kGrad>
__global__ void __launch_bounds__(kThreads) ssd_state_mma_kernel(const SsdArgs p) {
  extern __shared__ __align__(16) float sm[];
  using H = __nv_bfloat16;
  constexpr int kPitchB = N + 8, NT = N / 64;
  H *sX = reinterpret_cast<H*>(sm), *sB = sX + 3 * kPlane;
  float *s_dt = reinterpret_cast<float*>(sB + kT * kPitchB), *s_cum = s_dt + kT;
  const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z, t0 = c * kT, rows = min(kT, p.l - t0), g = h / (p.h / p.g);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr (kGrad) copy_rows<N>(sB, kPitchB, static_cast<const H*>(p.C) + b * p.c_sb + t0 * p.c_sl + g * N, p.c_sl, rows);
  else copy_rows<N>(sB, kPitchB, static_cast<const H*>(p.B) + b * p.b_sb + t0 * p.b_sl + g * N, p.b_sl, rows);
  const int64_t stride = kGrad ? static_cast<int64_t>(p.h) * kP : p.x_sl;
  const H* x = kGrad ? static_cast<const H*>(p.dy) + ((static_cast<int64_t>(b) * p.l + t0) * p.h + h) * kP : static_cast<const H*>(p.x) + b * p.x_sb + t0 * p.x_sl + h * kP;
  float4 v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = threadIdx.x + k * kThreads, r = i / 16;
    v[k] = r < rows ? ld4(x + r * stride + (i % 16) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  block_decay(s_dt, s_cum, p.dt + (static_cast<int64_t>(b) * p.l + t0) * p.h + h, p.h, rows, p.A[h]);
  const float end = s_cum[kT - 1];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = threadIdx.x + k * kThreads, r = i / 16;
    const float f = r >= rows ? 0.f : kGrad ? expf(s_cum[r]) : expf(end - s_cum[r]) * s_dt[r];
    store_split(sX + r * kPitchH + (i % 16) * 4, make_float4(v[k].x * f, v[k].y * f, v[k].z * f, v[k].w * f));
  }
  if (!kGrad && threadIdx.x == 0) p.decay[(static_cast<int64_t>(b) * p.h + h) * p.n_chunks + c] = expf(end);
  __syncthreads();
  const int n0 = warp * (8 * NT);
  float acc[4][NT][4], low[4][NT][4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][n][e] = low[m][n][e] = 0.f;
#pragma unroll
  for (int k = 0; k < kT / 16; ++k) {
    uint32_t fb[4];
    const H* bp = sB + (k * 16 + (lane & 15)) * kPitchB + n0;
    if constexpr (NT == 2) ldm4_trans(fb, bp + (lane >> 4) * 8);
    else ldm2_trans(fb[0], fb[1], bp);
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        uint32_t fa[4];
        ldm4_trans(fa, sX + q * kPlane + (k * 16 + (lane & 7) + (lane >> 4) * 8) * kPitchH + m * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int n = 0; n < NT; ++n) mma16816(q == 0 ? acc[m][n] : low[m][n], fa, fb[2 * n], fb[2 * n + 1]);
      }
  }
  float* out = (kGrad ? p.dstates : p.states) + ((static_cast<int64_t>(b) * p.h + h) * p.n_chunks + c) * (kP * N);
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float* o = out + (m * 16 + (lane >> 2)) * N + n0 + n * 8 + (lane & 3) * 2;
      *reinterpret_cast<float2*>(o) = make_float2(acc[m][n][0] + low[m][n][0], acc[m][n][1] + low[m][n][1]);
      *reinterpret_cast<float2*>(o + 8 * N) = make_float2(acc[m][n][2] + low[m][n][2], acc[m][n][3] + low[m][n][3]);
    }
}

// ssd_out_kernel for bf16: a warp takes 8 columns p and all 64 rows t.  Its rows of the state come straight from memory into the operand's
// registers: a thread's four neighbouring values stand for the k slots 2i, 2i + 1, 2i + 8, 2i + 9 in both operands.
template <int N>
__global__ void __launch_bounds__(kThreads, 3) ssd_out_mma_kernel(const SsdArgs p) {
  extern __shared__ __align__(16) float sm[];
  using H = __nv_bfloat16;
  constexpr int kPitchC = N + 16;
  H *sM = reinterpret_cast<H*>(sm), *sX = sM + 3 * kPlane, *sC = sX + kPlane;
  float *s_dt = reinterpret_cast<float*>(sC + kT * kPitchC), *s_cum = s_dt + kT;
  const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z, t0 = c * kT, rows = min(kT, p.l - t0), g = h / (p.h / p.g);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tg = lane & 3;
  const float* S = p.states + ((static_cast<int64_t>(b) * p.h + h) * p.n_chunks + c) * (kP * N) + (warp * 8 + gr) * N + tg * 4;
  float4 st[N / 16];
#pragma unroll
  for (int k = 0; k < N / 16; ++k) st[k] = *reinterpret_cast<const float4*>(S + k * 16);
  const float* G = p.scores + ((static_cast<int64_t>(b) * p.n_chunks + c) * p.g + g) * (kT * kT);
  float4 v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = *reinterpret_cast<const float4*>(G + (threadIdx.x + k * kThreads) * 4);
  copy_rows<N>(sC, kPitchC, static_cast<const H*>(p.C) + b * p.c_sb + t0 * p.c_sl + g * N, p.c_sl, rows);
  copy_rows<kP>(sX, kPitchH, static_cast<const H*>(p.x) + b * p.x_sb + t0 * p.x_sl + h * kP, p.x_sl, rows);
  block_decay(s_dt, s_cum, p.dt + (static_cast<int64_t>(b) * p.l + t0) * p.h + h, p.h, rows, p.A[h]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = threadIdx.x + k * kThreads, t = i / 16, u = (i % 16) * 4;
    float e[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q] = u + q <= t ? e[q] * expf(s_cum[t] - s_cum[u + q]) * s_dt[u + q] : 0.f;
    store_split(sM + t * kPitchH + u, make_float4(e[0], e[1], e[2], e[3]));
  }
  __syncthreads();
  float acc[4][4], low[4][4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[m][e] = low[m][e] = 0.f;
#pragma unroll
  for (int k = 0; k < N / 16; ++k) {
    uint32_t b0[3], b1[3];
    split3(st[k].x, st[k].y, b0);
    split3(st[k].z, st[k].w, b1);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const H* cp = sC + (m * 16 + gr) * kPitchC + k * 16 + tg * 4;
      const uint2 r0 = *reinterpret_cast<const uint2*>(cp), r1 = *reinterpret_cast<const uint2*>(cp + 8 * kPitchC);
      const uint32_t fa[4] = {r0.x, r1.x, r0.y, r1.y};
#pragma unroll
      for (int q = 0; q < 3; ++q) mma16816(q == 0 ? acc[m] : low[m], fa, b0[q], b1[q]);
    }
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const float e0 = expf(s_cum[m * 16 + gr]), e1 = expf(s_cum[m * 16 + gr + 8]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc[m][e] = (acc[m][e] + low[m][e]) * (e < 2 ? e0 : e1);
      low[m][e] = 0.f;
    }
  }
#pragma unroll
  for (int k = 0; k < kT / 16; ++k) {
    uint32_t x0, x1;
    ldm2_trans(x0, x1, sX + (k * 16 + (lane & 15)) * kPitchH + warp * 8);
#pragma unroll
    for (int m = k; m < 4; ++m)                 // nothing above the diagonal
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        uint32_t fa[4];
        ldm4(fa, sM + q * kPlane + (m * 16 + (lane & 15)) * kPitchH + k * 16 + (lane >> 4) * 8);
        mma16816(q == 0 ? acc[m] : low[m], fa, x0, x1);
      }
  }
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[m][e] += low[m][e];
  const float d = p.D[h];
  __syncthreads();
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int at = (m * 16 + gr + 8 * e) * kPitchH + warp * 8 + tg * 2;
      const float2 xv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sX + at));
      *reinterpret_cast<__nv_bfloat162*>(sM + at) = __floats2bfloat162_rn(fmaf(d, xv.x, acc[m][2 * e]), fmaf(d, xv.y, acc[m][2 * e + 1]));
    }
  __syncthreads();
  H* y = static_cast<H*>(p.y) + ((static_cast<int64_t>(b) * p.l + t0) * p.h + h) * kP;
  for (int i = threadIdx.x; i < rows * (kP / 8); i += kThreads) {
    const int t = i / (kP / 8), q = (i % (kP / 8)) * 8;
    *reinterpret_cast<uint4*>(y + static_cast<int64_t>(t) * p.h * kP + q) = *reinterpret_cast<const uint4*>(sM + t * kPitchH + q);
  }
}

// along the blocks, in place.  Forward: each block's contribution becomes the state it starts from.  Reverse: the gradient of each block's
// starting state (its own outputs' part) becomes the gradient of the state it ends with.  Bound by bytes: eight blocks are read before any
// of them is written, which the compiler cannot do by itself within one buffer (64 heads x 2048 x 64 x 128: 53 to 81 us before, 21 after).
template <bool kReverse>
__global__ void __launch_bounds__(kThreads) ssd_pass_kernel(float4* __restrict__ s, const float* __restrict__ decay, const float4* __restrict__ first,
                                                            float4* __restrict__ last, int n_chunks, int per_head) {
  const int64_t bh = blockIdx.y;
  const int e = blockIdx.x * kThreads + threadIdx.x;
  if (e >= per_head) return;
  float4 run = first != nullptr ? first[bh * per_head + e] : make_float4(0.f, 0.f, 0.f, 0.f);
  float4* base = s + bh * n_chunks * per_head + e;
  const float* d = decay + bh * n_chunks;
  constexpr int kAhead = 8;                    // blocks read before the first of them is written (they lie in one buffer)
  for (int i0 = 0; i0 < n_chunks; i0 += kAhead) {
    float4 v[kAhead];
    float f[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const int i = min(i0 + k, n_chunks - 1), c = kReverse ? n_chunks - 1 - i : i;
      v[k] = base[static_cast<int64_t>(c) * per_head];
      f[k] = d[c];
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      if (i0 + k >= n_chunks) break;
      const int c = kReverse ? n_chunks - 1 - (i0 + k) : i0 + k;
      base[static_cast<int64_t>(c) * per_head] = run;
      run.x = fmaf(run.x, f[k], v[k].x); run.y = fmaf(run.y, f[k], v[k].y); run.z = fmaf(run.z, f[k], v[k].z); run.w = fmaf(run.w, f[k], v[k].w);
    }
  }
  if (last != nullptr) last[bh * per_head + e] = run;
}

template <int N, typename T>
__global__ void __launch_bounds__(kThreads) ssd_out_kernel(const SsdArgs p) {
  extern __shared__ __align__(16) float sm[];
  constexpr int kPitchN = N + 4;
  float *sM = sm, *sXT = sM + kT * kPitchT, *sC = sXT + kP * kPitchT, *sS = sC + kT * kPitchN, *s_dt = sS + kP * kPitchN, *s_cum = s_dt + kT;
  const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z, t0 = c * kT, rows = min(kT, p.l - t0), g = h / (p.h / p.g);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  block_decay(s_dt, s_cum, p.dt + (static_cast<int64_t>(b) * p.l + t0) * p.h + h, p.h, rows, p.A[h]);
  const float* G = p.scores + ((static_cast<int64_t>(b) * p.n_chunks + c) * p.g + g) * (kT * kT);
  for (int i = threadIdx.x; i < kT * kT / 4; i += kThreads) {
    const int t = i / (kT / 4), u = (i % (kT / 4)) * 4;
    float4 v = *reinterpret_cast<const float4*>(G + t * kT + u);
    float* e = reinterpret_cast<float*>(&v);
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q] = u + q <= t ? e[q] * expf(s_cum[t] - s_cum[u + q]) * s_dt[u + q] : 0.f;
    *reinterpret_cast<float4*>(sM + t * kPitchT + u) = v;
  }
  const T* x = static_cast<const T*>(p.x) + b * p.x_sb + t0 * p.x_sl + h * kP;
  for (int i = threadIdx.x; i < kT * (kP / 4); i += kThreads) {
    const int u = i % kT, q = (i / kT) * 4;
    const float4 v = u < rows ? ld4(x + u * p.x_sl + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    sXT[q * kPitchT + u] = v.x;
    sXT[(q + 1) * kPitchT + u] = v.y;
    sXT[(q + 2) * kPitchT + u] = v.z;
    sXT[(q + 3) * kPitchT + u] = v.w;
  }
  load_rows<N>(sC, kPitchN, static_cast<const T*>(p.C) + b * p.c_sb + t0 * p.c_sl + g * N, p.c_sl, rows, [&](int r) { return expf(s_cum[r]); });
  load_rows<N>(sS, kPitchN, p.states + ((static_cast<int64_t>(b) * p.h + h) * p.n_chunks + c) * (kP * N), static_cast<int64_t>(N), kP, One{});
  __syncthreads();
  float acc[4][4];
  zero(acc);
  mm<4, 4, true, true>(acc, sM, kPitchT, sXT, kPitchT, kT, ty, tx);
  mm<4, 4, true, true>(acc, sC, kPitchN, sS, kPitchN, N, ty, tx);
  const float d = p.D[h];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sM[(ty + 16 * i) * kPitchT + tx + 16 * j] = fmaf(d, sXT[(tx + 16 * j) * kPitchT + ty + 16 * i], acc[i][j]);
  __syncthreads();
  T* y = static_cast<T*>(p.y) + ((static_cast<int64_t>(b) * p.l + t0) * p.h + h) * kP;
  for (int i = threadIdx.x; i < rows * (kP / 4); i += kThreads) {
    const int t = i / (kP / 4), q = (i % (kP / 4)) * 4;
    st4(y + static_cast<int64_t>(t) * p.h * kP + q, *reinterpret_cast<const float4*>(sM + t * kPitchT + q));
  }
}

// all gradients of one block for `per` heads of one group.  The first half of the threads takes the scores, C and x, the second half what
// goes through the state at the block's end, B among it: half of the multiply-adds each, and four warps per scheduler instead of two.
// While the first half finishes dx the second fetches the next head's states.  64 heads x 2048 steps x 64 x 128: 485 us with 256 threads that
// took one product after the other, 375 now.
template <int N, typename T>
__global__ void __launch_bounds__(2 * kThreads, 1) ssd_grad_kernel(const SsdArgs p) {
  extern __shared__ __align__(16) float sm[];
  constexpr int kPitchN = N + 4, NI = N / 16;
  float* sC = sm;                              // [t][n]
  float* sB = sC + kT * kPitchN;               // [u][n]
  float* sS = sB + kT * kPitchN;               // [p][n] state at the block's start
  float* sR = sS + kP * kPitchN;               // [p][n] gradient of the state at its end
  float* sG = sR + kP * kPitchN;               // [t][u]
  float* sX = sG + kT * kPitchT;               // [u][p]
  float* sY = sX + kT * kPitchT;               // [t][p] dy
  float* sM = sY + kT * kPitchT;               // [t][u] decayed scores, then the group's score gradients
  float* sQ = sM + kT * kPitchT;               // [u][p] the end state's part of dx, then the score gradients transposed
  float* s_dt = sQ + kT * kPitchT;
  float *s_cum = s_dt + kT, *s_row = s_cum + kT, *s_end = s_row + kT, *s_dir = s_end + kT, *s_col = s_dir + kT, *s_red = s_col + 8 * kT;
  const int c = blockIdx.x, b = blockIdx.z, t0 = c * kT, rows = min(kT, p.l - t0), hpg = p.h / p.g;
  const int g = blockIdx.y / p.n_sub, sub = blockIdx.y % p.n_sub, per = hpg / p.n_sub;
  const bool second = threadIdx.x >= kThreads;
  const int tid = threadIdx.x & (kThreads - 1), tx = tid & 15, ty = tid >> 4, warp = tid >> 5, lane = tid & 31;
  load_rows<N, 2 * kThreads>(sC, kPitchN, static_cast<const T*>(p.C) + b * p.c_sb + t0 * p.c_sl + g * N, p.c_sl, rows, One{});
  load_rows<N, 2 * kThreads>(sB, kPitchN, static_cast<const T*>(p.B) + b * p.b_sb + t0 * p.b_sl + g * N, p.b_sl, rows, One{});
  load_rows<kT, 2 * kThreads>(sG, kPitchT, p.scores + ((static_cast<int64_t>(b) * p.n_chunks + c) * p.g + g) * (kT * kT), static_cast<int64_t>(kT), kT, One{});
  const int h0 = g * hpg + sub * per;
  auto state_at = [&](int h) { return ((static_cast<int64_t>(b) * p.h + h) * p.n_chunks + c) * (kP * N); };
  load_rows<N, 2 * kThreads>(sS, kPitchN, p.states + state_at(h0), static_cast<int64_t>(N), kP, One{});
  load_rows<N, 2 * kThreads>(sR, kPitchN, p.dstates + state_at(h0), static_cast<int64_t>(N), kP, One{});
  float acc[4][NI], dG[4][4];                  // dC in the first half, dB in the second
  zero(acc);
  zero(dG);
  for (int hi = 0; hi < per; ++hi) {
    const int h = h0 + hi;
    const float a = p.A[h];
    const int64_t row0 = (static_cast<int64_t>(b) * p.l + t0) * p.h + h;
    __syncthreads();                           // the head before is done with its tiles
    load_rows<kP, 2 * kThreads>(sX, kPitchT, static_cast<const T*>(p.x) + b * p.x_sb + t0 * p.x_sl + h * kP, p.x_sl, rows, One{});
    load_rows<kP, 2 * kThreads>(sY, kPitchT, static_cast<const T*>(p.dy) + row0 * kP, static_cast<int64_t>(p.h) * kP, rows, One{});
    block_decay(s_dt, s_cum, p.dt + row0, p.h, rows, a);  // and all tiles are there
    const float end = s_cum[kT - 1];

    if (!second) {
      // gradient of the scores, and through their decays of cum
      {
        float v[4][4], col[4] = {0.f, 0.f, 0.f, 0.f};
        zero(v);
        mm<4, 4, true, true>(v, sY, kPitchT, sX, kPitchT, kP, ty, tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = ty + 16 * i;
          float row = 0.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int u = tx + 16 * j;
            const float w = u <= t ? expf(s_cum[t] - s_cum[u]) : 0.f, wg = w * sG[t * kPitchT + u];
            sM[t * kPitchT + u] = wg;
            const float d = v[i][j] * s_dt[u];
            dG[i][j] = fmaf(d, w, dG[i][j]);
            const float q = u < t ? d * wg : 0.f;           // on the diagonal the two ends cancel
            row += q;
            col[j] += q;
          }
          row = half_warp_sum(row);
          if (tx == 0) s_row[t] = row;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          col[j] += __shfl_xor_sync(0xffffffffu, col[j], 16);
          if (lane < 16) s_col[warp * kT + tx + 16 * j] = col[j];
        }
      }
      // C through the starting state
      {
        float v[4][NI];
        zero(v);
        mm<4, NI, true, false>(v, sY, kPitchT, sS, kPitchN, kP, ty, tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = ty + 16 * i;
          const float e = expf(s_cum[t]);
          float row = 0.f;
#pragma unroll
          for (int j = 0; j < NI; ++j) {
            const float w = e * v[i][j];
            acc[i][j] += w;
            row = fmaf(w, sC[t * kPitchN + col4(tx, j)], row);
          }
          row = half_warp_sum(row);
          if (tx == 0) s_row[t] += row;
        }
      }
    } else {
      // the end state's part of dx
      {
        float v[4][4];
        zero(v);
        mm<4, 4, true, true>(v, sB, kPitchN, sR, kPitchN, N, ty, tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float e = expf(end - s_cum[ty + 16 * i]);
#pragma unroll
          for (int j = 0; j < 4; ++j) sQ[(ty + 16 * i) * kPitchT + tx + 16 * j] = e * v[i][j];
        }
      }
      // B through the end state
      {
        float v[4][NI];
        zero(v);
        mm<4, NI, true, false>(v, sX, kPitchT, sR, kPitchN, kP, ty, tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int u = ty + 16 * i;
          const float e = expf(end - s_cum[u]) * s_dt[u];
          float z = 0.f;
#pragma unroll
          for (int j = 0; j < NI; ++j) {
            const float w = e * v[i][j];
            acc[i][j] += w;
            z = fmaf(w, sB[u * kPitchN + col4(tx, j)], z);
          }
          z = half_warp_sum(z);
          if (tx == 0) s_end[u] = z;
        }
      }
      // the end state's gradient times the starting state
      {
        float rs = 0.f;
        for (int i = tid; i < kP * (N / 4); i += kThreads) {
          const int r = i / (N / 4), q = (i % (N / 4)) * 4;
          const float4 s = *reinterpret_cast<const float4*>(sS + r * kPitchN + q), e = *reinterpret_cast<const float4*>(sR + r * kPitchN + q);
          rs += s.x * e.x + s.y * e.y + s.z * e.z + s.w * e.w;
        }
        rs = dev::warp_sum(rs);
        if (lane == 0) s_red[8 + warp] = rs;
      }
    }
    __syncthreads();
    if (second) {
      if (hi + 1 < per) {
        load_rows<N>(sS, kPitchN, p.states + state_at(h + 1), static_cast<int64_t>(N), kP, One{});
        load_rows<N>(sR, kPitchN, p.dstates + state_at(h + 1), static_cast<int64_t>(N), kP, One{});
      }
      continue;
    }
    // dx, dt through x, and D
    float dd = 0.f;
    {
      float v[4][4];
      zero(v);
      mm<4, 4, false, false>(v, sM, kPitchT, sY, kPitchT, kT, ty, tx);
      const float d = p.D[h];
      T* dx = static_cast<T*>(p.dx) + row0 * kP;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int u = ty * 4 + i;
        float dir = 0.f, o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int q = tx * 4 + j;
          const float pre = v[i][j] + sQ[u * kPitchT + q], xv = sX[u * kPitchT + q], yv = sY[u * kPitchT + q];
          dir = fmaf(xv, pre, dir);
          dd = fmaf(xv, yv, dd);
          o[j] = fmaf(s_dt[u], pre, d * yv);
        }
        if (u < rows) st4(dx + static_cast<int64_t>(u) * p.h * kP + tx * 4, make_float4(o[0], o[1], o[2], o[3]));
        dir = half_warp_sum(dir);
        if (tx == 0) s_dir[u] = dir;
      }
      dd = dev::warp_sum(dd);
      if (lane == 0) s_red[warp] = dd;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");                  // the first half alone
    // cum's gradient summed from the block's end, for dt and A
    if (warp == 0) {
      float g0[2], z = 0.f, acc_d = 0.f, acc_r = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        acc_d += s_red[w];
        acc_r += s_red[8 + w];
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        float v = s_row[t] - s_end[t];
        z += s_end[t];
#pragma unroll
        for (int w = 0; w < 8; ++w) v -= s_col[w * kT + t];
        g0[e] = v;
      }
      z = dev::warp_sum(z);
      if (lane == 31) g0[1] += z + expf(end) * acc_r;
      float incl = g0[0] + g0[1];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float v = __shfl_down_sync(0xffffffffu, incl, o);
        if (lane + o < 32) incl += v;
      }
      const float dda0 = incl, dda1 = incl - g0[0];
      const int t = 2 * lane;
      if (t < rows) p.ddt[row0 + static_cast<int64_t>(t) * p.h] = fmaf(a, dda0, s_dir[t]);
      if (t + 1 < rows) p.ddt[row0 + static_cast<int64_t>(t + 1) * p.h] = fmaf(a, dda1, s_dir[t + 1]);
      const float da = dev::warp_sum(s_dt[t] * dda0 + s_dt[t + 1] * dda1);
      if (lane == 0) {
        const int64_t at = (static_cast<int64_t>(b) * p.n_chunks + c) * p.h + h;
        p.dA[at] = da;
        p.dD[at] = acc_d;
      }
    }
  }
  // the scores' gradients into B and C
  __syncthreads();
  if (!second) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sM[(ty + 16 * i) * kPitchT + tx + 16 * j] = dG[i][j];
        sQ[(tx + 16 * j) * kPitchT + ty + 16 * i] = dG[i][j];
      }
  }
  __syncthreads();
  mm<4, NI, true, false>(acc, second ? sQ : sM, kPitchT, second ? sC : sB, kPitchN, kT, ty, tx);
  const int64_t plane = static_cast<int64_t>(p.b) * p.l * p.g * N;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = ty + 16 * i;
    if (t >= rows) continue;
    const int64_t at = ((static_cast<int64_t>(b) * p.l + t0 + t) * p.g + g) * N + tx * 4;
#pragma unroll
    for (int q = 0; q < N / 64; ++q) {
      const float4 v = make_float4(acc[i][q * 4], acc[i][q * 4 + 1], acc[i][q * 4 + 2], acc[i][q * 4 + 3]);
      if (p.n_sub == 1) st4(static_cast<T*>(second ? p.dB : p.dC) + at + q * 64, v);
      else st4(p.partial + (sub * 2 + (second ? 0 : 1)) * plane + at + q * 64, v);
    }
  }
}

// ssd_grad_kernel for bf16, the same two halves.  A warp takes 16 rows and half of the columns of every product, so sums along a row come from
// two warps.  The states and the decayed scores stand in shared memory as three bf16 planes.  Bound by the tensor instructions (about 2700 per
// head and block, 18 cycles each in a scheduler: 90 us of the 191 at 64 heads x 2048 steps) and the phases between them.
template <int N>
__global__ void __launch_bounds__(2 * kThreads, 1) ssd_grad_mma_kernel(const SsdArgs p) {
  extern __shared__ __align__(16) float sm[];
  using H = __nv_bfloat16;
  constexpr int kPitchN = N + 8, kPlaneN = kT * kPitchN, NT = N / 16;    // n tiles of 8 in half of the columns
  H* sC = reinterpret_cast<H*>(sm);            // [t][n]
  H* sB = sC + kPlaneN;                        // [u][n]
  H* sS = sB + kPlaneN;                        // 3 x [p][n] state at the block's start
  H* sR = sS + 3 * kPlaneN;                    // 3 x [p][n] gradient of the state at its end
  H* sX = sR + 3 * kPlaneN;                    // [u][p]
  H* sY = sX + kPlane;                         // [t][p] dy
  H* sM = sY + kPlane;                         // 3 x [t][u] decayed scores, then the group's score gradients
  float* sG = reinterpret_cast<float*>(sM + 3 * kPlane);    // [t][u]
  float* sQ = sG + kT * kPitchT;               // [u][p] the end state's part of dx
  float* s_dt = sQ + kT * kPitchT;
  float *s_cum = s_dt + kT, *s_row = s_cum + kT, *s_end = s_row + 4 * kT, *s_dir = s_end + 2 * kT, *s_col = s_dir + 2 * kT, *s_red = s_col + 4 * kT;
  const int c = blockIdx.x, b = blockIdx.z, t0 = c * kT, rows = min(kT, p.l - t0), hpg = p.h / p.g;
  const int g = blockIdx.y / p.n_sub, sub = blockIdx.y % p.n_sub, per = hpg / p.n_sub;
  const bool second = threadIdx.x >= kThreads;
  const int tid = threadIdx.x & (kThreads - 1), warp = tid >> 5, lane = tid & 31, gr = lane >> 2, tg = lane & 3;
  const int m0 = (warp & 3) * 16, side = warp >> 2;             // this warp's rows, and which half of the columns
  const int h0 = g * hpg + sub * per;
  // operand addresses of this lane, see ldm4: rows x k as stored, k x rows transposed; n x k as stored, k x n transposed
  auto a_at = [&](const H* base, int pitch, int m, int k) { return base + (m + (lane & 15)) * pitch + k + (lane >> 4) * 8; };
  auto at_at = [&](const H* base, int pitch, int m, int k) { return base + (k + (lane & 7) + (lane >> 4) * 8) * pitch + m + ((lane >> 3) & 1) * 8; };
  auto b_at = [&](const H* base, int pitch, int n, int k) { return base + (n + (lane & 7) + (lane >> 4) * 8) * pitch + k + ((lane >> 3) & 1) * 8; };
  auto bt_at = [&](const H* base, int pitch, int n, int k) { return base + (k + (lane & 15)) * pitch + n + (lane >> 4) * 8; };
  auto quad_sum = [](float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
  };
  // the second half fetches a head's states and takes its part of their product on the way
  auto fetch_states = [&](int h) {
    const int64_t at = ((static_cast<int64_t>(b) * p.h + h) * p.n_chunks + c) * (kP * N);
    float rs = 0.f;
#pragma unroll 4
    for (int k = 0; k < kP * (N / 4) / kThreads; ++k) {
      const int i = tid + k * kThreads, r = i / (N / 4), q = (i % (N / 4)) * 4;
      const float4 s = *reinterpret_cast<const float4*>(p.states + at + r * N + q), e = *reinterpret_cast<const float4*>(p.dstates + at + r * N + q);
      rs += s.x * e.x + s.y * e.y + s.z * e.z + s.w * e.w;
      uint32_t lo[3], hi[3];
      split3(s.x, s.y, lo);
      split3(s.z, s.w, hi);
#pragma unroll
      for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(sS + j * kPlaneN + r * kPitchN + q) = make_uint2(lo[j], hi[j]);
      split3(e.x, e.y, lo);
      split3(e.z, e.w, hi);
#pragma unroll
      for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(sR + j * kPlaneN + r * kPitchN + q) = make_uint2(lo[j], hi[j]);
    }
    return dev::warp_sum(rs);
  };
  float rs = 0.f;
  if (second) rs = fetch_states(h0);
  else {
    copy_rows<N>(sC, kPitchN, static_cast<const H*>(p.C) + b * p.c_sb + t0 * p.c_sl + g * N, p.c_sl, rows);
    copy_rows<N>(sB, kPitchN, static_cast<const H*>(p.B) + b * p.b_sb + t0 * p.b_sl + g * N, p.b_sl, rows);
    load_rows<kT>(sG, kPitchT, p.scores + ((static_cast<int64_t>(b) * p.n_chunks + c) * p.g + g) * (kT * kT), static_cast<int64_t>(kT), kT, One{});
  }
  float acc[NT][4], dG[4][4];                  // dC in the first half, dB in the second
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
  zero(dG);
  for (int hi = 0; hi < per; ++hi) {
    const int h = h0 + hi;
    const float a = p.A[h];
    const int64_t row0 = (static_cast<int64_t>(b) * p.l + t0) * p.h + h;
    __syncthreads();                           // the head before is done with its tiles
    if (second) copy_rows<kP>(sX, kPitchH, static_cast<const H*>(p.x) + b * p.x_sb + t0 * p.x_sl + h * kP, p.x_sl, rows);
    else copy_rows<kP>(sY, kPitchH, static_cast<const H*>(p.dy) + row0 * kP, static_cast<int64_t>(p.h) * kP, rows);
    block_decay(s_dt, s_cum, p.dt + row0, p.h, rows, a);  // and all tiles are there
    const float end = s_cum[kT - 1];
    const int r0 = m0 + gr, r1 = r0 + 8;       // this thread's two rows
    const float cum0 = s_cum[r0], cum1 = s_cum[r1];
    uint32_t fx[4][4];                         // the warp's rows of Y (first half) or X
#pragma unroll
    for (int k = 0; k < 4; ++k) ldm4(fx[k], a_at(second ? sX : sY, kPitchH, m0, k * 16));

    if (!second) {
      // gradient of the scores, and through their decays of cum
      {
        float v[4][4];
        zero(v);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            uint32_t fb[4];
            ldm4(fb, b_at(sX, kPitchH, side * 32 + j * 8, k * 16));
            mma16816(v[j], fx[k], fb[0], fb[1]);
            mma16816(v[j + 1], fx[k], fb[2], fb[3]);
          }
        float row[2] = {0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int u = side * 32 + j * 8 + tg * 2;
          float col[2] = {0.f, 0.f}, wg[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int t = e < 2 ? r0 : r1, uu = u + (e & 1);
            const float w = uu <= t ? expf((e < 2 ? cum0 : cum1) - s_cum[uu]) : 0.f;
            wg[e] = w * sG[t * kPitchT + uu];
            const float d = v[j][e] * s_dt[uu];
            dG[j][e] = fmaf(d, w, dG[j][e]);
            const float q = uu < t ? d * wg[e] : 0.f;      // on the diagonal the two ends cancel
            row[e >> 1] += q;
            col[e & 1] += q;
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint32_t part[3];
            split3(wg[2 * e], wg[2 * e + 1], part);
#pragma unroll
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint32_t*>(sM + q * kPlane + (e == 0 ? r0 : r1) * kPitchH + u) = part[q];
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) col[e] += __shfl_xor_sync(0xffffffffu, col[e], o);
          }
          if (gr == 0) {
            s_col[(warp & 3) * kT + u] = col[0];
            s_col[(warp & 3) * kT + u + 1] = col[1];
          }
        }
        row[0] = quad_sum(row[0]);
        row[1] = quad_sum(row[1]);
        if (tg == 0) {
          s_row[side * kT + r0] = row[0];
          s_row[side * kT + r1] = row[1];
        }
      }
    } else {
      // the end state's part of dx
      float v[4][4], low[4][4];
      zero(v);
      zero(low);
#pragma unroll 2
      for (int k = 0; k < N / 16; ++k) {
        uint32_t fa[4];
        ldm4(fa, a_at(sB, kPitchN, m0, k * 16));
#pragma unroll
        for (int j = 0; j < 4; j += 2)
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            uint32_t fb[4];
            ldm4(fb, b_at(sR + q * kPlaneN, kPitchN, side * 32 + j * 8, k * 16));
            mma16816(q == 0 ? v[j] : low[j], fa, fb[0], fb[1]);
            mma16816(q == 0 ? v[j + 1] : low[j + 1], fa, fb[2], fb[3]);
          }
      }
      const float e0 = expf(end - cum0), e1 = expf(end - cum1);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float* o = sQ + r0 * kPitchT + side * 32 + j * 8 + tg * 2;
        *reinterpret_cast<float2*>(o) = make_float2(e0 * (v[j][0] + low[j][0]), e0 * (v[j][1] + low[j][1]));
        *reinterpret_cast<float2*>(o + 8 * kPitchT) = make_float2(e1 * (v[j][2] + low[j][2]), e1 * (v[j][3] + low[j][3]));
      }
    }
    // C through the starting state (first half), B through the end state (second): 32 columns at a time
    {
      const float e0 = second ? expf(end - cum0) * s_dt[r0] : expf(cum0), e1 = second ? expf(end - cum1) * s_dt[r1] : expf(cum1);
      float row[2] = {0.f, 0.f};
#pragma unroll
      for (int n0 = 0; n0 < NT; n0 += 4) {
        float v[4][4], low[4][4];
        zero(v);
        zero(low);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int j = 0; j < 4; j += 2)
#pragma unroll
            for (int q = 0; q < 3; ++q) {
              uint32_t fb[4];
              ldm4_trans(fb, bt_at((second ? sR : sS) + q * kPlaneN, kPitchN, side * (N / 2) + (n0 + j) * 8, k * 16));
              mma16816(q == 0 ? v[j] : low[j], fx[k], fb[0], fb[1]);
              mma16816(q == 0 ? v[j + 1] : low[j + 1], fx[k], fb[2], fb[3]);
            }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const H* other = (second ? sB : sC) + r0 * kPitchN + side * (N / 2) + (n0 + j) * 8 + tg * 2;
          const float2 o0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(other));
          const float2 o1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(other + 8 * kPitchN));
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float w = (e < 2 ? e0 : e1) * (v[j][e] + low[j][e]);
            acc[n0 + j][e] += w;
            row[e >> 1] = fmaf(w, e == 0 ? o0.x : e == 1 ? o0.y : e == 2 ? o1.x : o1.y, row[e >> 1]);
          }
        }
      }
      row[0] = quad_sum(row[0]);
      row[1] = quad_sum(row[1]);
      float* dst = second ? s_end + side * kT : s_row + (2 + side) * kT;
      if (tg == 0) {
        dst[r0] = row[0];
        dst[r1] = row[1];
      }
    }
    if (second && lane == 0) s_red[8 + warp] = rs;
    __syncthreads();
    if (second) {
      if (hi + 1 < per) rs = fetch_states(h + 1);
      continue;
    }
    // dx, dt through x, and D; rows are steps u now
    float dd = 0.f;
    {
      float v[4][4], low[4][4];
      zero(v);
      zero(low);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k * 16 < m0) continue;             // no later step's scores before the diagonal
        uint32_t fa[3][4];
#pragma unroll
        for (int q = 0; q < 3; ++q) ldm4_trans(fa[q], at_at(sM + q * kPlane, kPitchH, m0, k * 16));
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          uint32_t fb[4];
          ldm4_trans(fb, bt_at(sY, kPitchH, side * 32 + j * 8, k * 16));
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            mma16816(q == 0 ? v[j] : low[j], fa[q], fb[0], fb[1]);
            mma16816(q == 0 ? v[j + 1] : low[j + 1], fa[q], fb[2], fb[3]);
          }
        }
      }
      const float d = p.D[h];
      H* dx = static_cast<H*>(p.dx) + row0 * kP;
      float dir[2] = {0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int u = e == 0 ? r0 : r1, q = side * 32 + j * 8 + tg * 2;
          const float2 end_part = *reinterpret_cast<const float2*>(sQ + u * kPitchT + q);
          const float2 xv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sX + u * kPitchH + q));
          const float2 yv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sY + u * kPitchH + q));
          const float pre0 = v[j][2 * e] + low[j][2 * e] + end_part.x, pre1 = v[j][2 * e + 1] + low[j][2 * e + 1] + end_part.y;
          dir[e] = fmaf(xv.x, pre0, fmaf(xv.y, pre1, dir[e]));
          dd = fmaf(xv.x, yv.x, fmaf(xv.y, yv.y, dd));
          if (u < rows)
            *reinterpret_cast<__nv_bfloat162*>(dx + static_cast<int64_t>(u) * p.h * kP + q) =
                __floats2bfloat162_rn(fmaf(s_dt[u], pre0, d * yv.x), fmaf(s_dt[u], pre1, d * yv.y));
        }
      dir[0] = quad_sum(dir[0]);
      dir[1] = quad_sum(dir[1]);
      if (tg == 0) {
        s_dir[side * kT + r0] = dir[0];
        s_dir[side * kT + r1] = dir[1];
      }
      dd = dev::warp_sum(dd);
      if (lane == 0) s_red[warp] = dd;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");                  // the first half alone
    // cum's gradient summed from the block's end, for dt and A
    if (warp == 0) {
      float g0[2], z = 0.f, acc_d = 0.f, acc_r = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        acc_d += s_red[w];
        acc_r += s_red[8 + w];
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        const float to_end = s_end[t] + s_end[kT + t];
        float v = (s_row[t] + s_row[kT + t]) + (s_row[2 * kT + t] + s_row[3 * kT + t]) - to_end;
        z += to_end;
#pragma unroll
        for (int w = 0; w < 4; ++w) v -= s_col[w * kT + t];
        g0[e] = v;
      }
      z = dev::warp_sum(z);
      if (lane == 31) g0[1] += z + expf(end) * acc_r;
      float incl = g0[0] + g0[1];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float v = __shfl_down_sync(0xffffffffu, incl, o);
        if (lane + o < 32) incl += v;
      }
      const float dda0 = incl, dda1 = incl - g0[0];
      const int t = 2 * lane;
      if (t < rows) p.ddt[row0 + static_cast<int64_t>(t) * p.h] = fmaf(a, dda0, s_dir[t] + s_dir[kT + t]);
      if (t + 1 < rows) p.ddt[row0 + static_cast<int64_t>(t + 1) * p.h] = fmaf(a, dda1, s_dir[t + 1] + s_dir[kT + t + 1]);
      const float da = dev::warp_sum(s_dt[t] * dda0 + s_dt[t + 1] * dda1);
      if (lane == 0) {
        const int64_t at = (static_cast<int64_t>(b) * p.n_chunks + c) * p.h + h;
        p.dA[at] = da;
        p.dD[at] = acc_d;
      }
    }
  }
  // the scores' gradients into B and C
  __syncthreads();
  if (!second) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t part[3];
        split3(dG[j][2 * e], dG[j][2 * e + 1], part);
#pragma unroll
        for (int q = 0; q < 3; ++q)
          *reinterpret_cast<uint32_t*>(sM + q * kPlane + (m0 + gr + 8 * e) * kPitchH + side * 32 + j * 8 + tg * 2) = part[q];
      }
  }
  __syncthreads();
  uint32_t fa[4][3][4];                        // rows of the score gradients, or of their transpose
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      if (second) ldm4_trans(fa[k][q], at_at(sM + q * kPlane, kPitchH, m0, k * 16));
      else ldm4(fa[k][q], a_at(sM + q * kPlane, kPitchH, m0, k * 16));
    }
  const int64_t plane = static_cast<int64_t>(p.b) * p.l * p.g * N;
#pragma unroll
  for (int j = 0; j < NT; j += 2) {
    float v[2][4], low[2][4];
    zero(v);
    zero(low);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t fb[4];
      ldm4_trans(fb, bt_at(second ? sC : sB, kPitchN, side * (N / 2) + j * 8, k * 16));
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        mma16816(q == 0 ? v[0] : low[0], fa[k][q], fb[0], fb[1]);
        mma16816(q == 0 ? v[1] : low[1], fa[k][q], fb[2], fb[3]);
      }
    }
#pragma unroll
    for (int jj = 0; jj < 2; ++jj)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = m0 + gr + 8 * e;
        if (t >= rows) continue;
        const float o0 = acc[j + jj][2 * e] + (v[jj][2 * e] + low[jj][2 * e]), o1 = acc[j + jj][2 * e + 1] + (v[jj][2 * e + 1] + low[jj][2 * e + 1]);
        const int64_t at = ((static_cast<int64_t>(b) * p.l + t0 + t) * p.g + g) * N + side * (N / 2) + (j + jj) * 8 + tg * 2;
        if (p.n_sub == 1) *reinterpret_cast<__nv_bfloat162*>(static_cast<H*>(second ? p.dB : p.dC) + at) = __floats2bfloat162_rn(o0, o1);
        else *reinterpret_cast<float2*>(p.partial + (sub * 2 + (second ? 0 : 1)) * plane + at) = make_float2(o0, o1);
      }
  }
}

// dB and dC from the partial sums of n_sub CTAs
template <typename T>
__global__ void __launch_bounds__(kThreads) ssd_merge_kernel(const float4* __restrict__ part, T* __restrict__ dB, T* __restrict__ dC, int64_t plane4, int n_sub) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  if (i >= 2 * plane4) return;
  const int64_t at = i % plane4;
  float4 s = part[i];
  for (int k = 1; k < n_sub; ++k) {
    const float4 v = part[k * 2 * plane4 + i];
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  st4((i < plane4 ? dB : dC) + at * 4, s);
}

template <int N> constexpr int scores_smem() { return 2 * kT * (N + 4) * 4; }
template <int N> constexpr int state_smem() { return (kT * kPitchT + kT * (N + 4) + 2 * kT) * 4; }
template <int N> constexpr int out_smem() { return (2 * kT * kPitchT + 2 * kT * (N + 4) + 2 * kT) * 4; }
template <int N> constexpr int state_mma_smem() { return (3 * kPlane + kT * (N + 8)) * 2 + 2 * kT * 4; }
template <int N> constexpr int out_mma_smem() { return (4 * kPlane + kT * (N + 16)) * 2 + 2 * kT * 4; }
template <int N> constexpr int grad_smem() { return (4 * kT * (N + 4) + 5 * kT * kPitchT + 13 * kT + 16) * 4; }
template <int N> constexpr int grad_mma_smem() { return (8 * kT * (N + 8) + 5 * kPlane) * 2 + (2 * kT * kPitchT + 14 * kT + 16) * 4; }
static_assert(grad_smem<128>() <= 232448 && grad_mma_smem<128>() <= 232448, "one CTA's shared memory");

template <typename K>
bool with_smem(K kern, int bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

template <int N, typename T>
bool forward(const SsdArgs& p, cudaStream_t s) {
  constexpr bool mma = std::is_same<T, __nv_bfloat16>::value;
  const dim3 grid(p.n_chunks, p.h, p.b);
  static const bool ok = [] {
    bool all = with_smem(ssd_scores_kernel<N, T>, scores_smem<N>());
    if constexpr (mma) return all && with_smem(ssd_state_mma_kernel<N, false>, state_mma_smem<N>()) && with_smem(ssd_out_mma_kernel<N>, out_mma_smem<N>());
    else return all && with_smem(ssd_state_kernel<N, T, false>, state_smem<N>()) && with_smem(ssd_out_kernel<N, T>, out_smem<N>());
  }();
  if (!ok) return false;
  ssd_scores_kernel<N, T><<<dim3(p.n_chunks, p.g, p.b), kThreads, scores_smem<N>(), s>>>(p);
  if constexpr (mma) ssd_state_mma_kernel<N, false><<<grid, kThreads, state_mma_smem<N>(), s>>>(p);
  else ssd_state_kernel<N, T, false><<<grid, kThreads, state_smem<N>(), s>>>(p);
  constexpr int per = kP * N / 4;
  ssd_pass_kernel<false><<<dim3(per / kThreads, p.b * p.h), kThreads, 0, s>>>(reinterpret_cast<float4*>(p.states), p.decay,
                                                                              reinterpret_cast<const float4*>(p.first), reinterpret_cast<float4*>(p.last),
                                                                              p.n_chunks, per);
  if constexpr (mma) ssd_out_mma_kernel<N><<<grid, kThreads, out_mma_smem<N>(), s>>>(p);
  else ssd_out_kernel<N, T><<<grid, kThreads, out_smem<N>(), s>>>(p);
  return true;
}

template <int N, typename T>
bool backward(const SsdArgs& p, cudaStream_t s) {
  constexpr bool mma = std::is_same<T, __nv_bfloat16>::value;
  const dim3 grid(p.n_chunks, p.h, p.b);
  static const bool ok = [] {
    if constexpr (mma) return with_smem(ssd_state_mma_kernel<N, true>, state_mma_smem<N>()) && with_smem(ssd_grad_mma_kernel<N>, grad_mma_smem<N>());
    else return with_smem(ssd_state_kernel<N, T, true>, state_smem<N>()) && with_smem(ssd_grad_kernel<N, T>, grad_smem<N>());
  }();
  if (!ok) return false;
  if constexpr (mma) ssd_state_mma_kernel<N, true><<<grid, kThreads, state_mma_smem<N>(), s>>>(p);
  else ssd_state_kernel<N, T, true><<<grid, kThreads, state_smem<N>(), s>>>(p);
  constexpr int per = kP * N / 4;
  ssd_pass_kernel<true><<<dim3(per / kThreads, p.b * p.h), kThreads, 0, s>>>(reinterpret_cast<float4*>(p.dstates), p.decay,
                                                                             reinterpret_cast<const float4*>(p.dlast), reinterpret_cast<float4*>(p.dfirst),
                                                                             p.n_chunks, per);
  const dim3 grad_grid(p.n_chunks, p.g * p.n_sub, p.b);
  if constexpr (mma) ssd_grad_mma_kernel<N><<<grad_grid, 2 * kThreads, grad_mma_smem<N>(), s>>>(p);
  else ssd_grad_kernel<N, T><<<grad_grid, 2 * kThreads, grad_smem<N>(), s>>>(p);
  if (p.n_sub > 1) {
    const int64_t plane4 = static_cast<int64_t>(p.b) * p.l * p.g * N / 4;
    ssd_merge_kernel<T><<<static_cast<unsigned>((2 * plane4 + kThreads - 1) / kThreads), kThreads, 0, s>>>(
        reinterpret_cast<const float4*>(p.partial), static_cast<T*>(p.dB), static_cast<T*>(p.dC), plane4, p.n_sub);
  }
  return true;
}

}  // namespace

int ssd_block() { return kT; }

// a group's heads are shared among so many CTAs (a divisor of their number) that the grid fills the SMs three times over
int ssd_subgroups(int n_chunks, int groups, int batch, int heads_per_group) {
  int n = 1;
  while (n < heads_per_group && static_cast<int64_t>(n_chunks) * groups * batch * n < 3 * 148) {
    ++n;
    while (heads_per_group % n != 0) ++n;
  }
  return n;
}

bool ssd_supported(int head_dim, int state_dim) { return head_dim == kP && (state_dim == 64 || state_dim == 128); }

bool ssd_forward(const SsdArgs& p, int state_dim, bool bf16, cudaStream_t s) {
  if (state_dim == 128) return bf16 ? forward<128, __nv_bfloat16>(p, s) : forward<128, float>(p, s);
  return bf16 ? forward<64, __nv_bfloat16>(p, s) : forward<64, float>(p, s);
}
bool ssd_backward(const SsdArgs& p, int state_dim, bool bf16, cudaStream_t s) {
  if (state_dim == 128) return bf16 ? backward<128, __nv_bfloat16>(p, s) : backward<128, float>(p, s);
  return bf16 ? backward<64, __nv_bfloat16>(p, s) : backward<64, float>(p, s);
}

}  // namespace b200seq
