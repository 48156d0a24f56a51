// Paged-KV attention for the dynamic (continuous-batching) inference engine.
//
// One step of the engine carries a ragged mix of queries: single decode tokens of running requests and chunks of prompt
// tokens of requests being prefilled.  Every query token t belongs to request r = tok_req[t] and sees the first
// tok_len[t] keys of that request; keys live in fixed-size pages of a shared pool, found through the request's block
// table.
//
// A tile is up to 16, 64 or 128 rows, a row being one (token, query head) of one request and one KV head: all query heads of a group share
// every key/value row that is read, and so do the tokens of a chunk.  Keys come in stages of 64, gathered page by page into a ring of
// shared-memory buffers, for 16 and 64 rows by 16-byte asynchronous copies (32 KB each at d = 128) and
// multiplied by m16n8k16 tensor instructions from there, for 128 by TMA and multiplied on tcgen05.  The weights are fp32: each enters the value product as three 16-bit
// parts that add up to it (fp16: to 2^-40 of the largest weight where it is below 2^-16 of that).
//   rows = 16 (decode, short chunks): the four warps take 16 keys of a stage each, bound by HBM.  The stages of all (request, KV head)
//     pairs stand in one line that is cut evenly over three CTAs per SM, whatever the contexts' lengths; an item that a cut falls into
//     leaves partial (max, sum, accumulator) triples, and the CTA that counts the last of them puts them together.  What a CTA needs to know before its
//     first key (a request per thread) is read while the new keys are still being written.  64 contexts of 1k to 4k, 32 / 8 heads of 128:
//     128 us with the write, 134 with a kernel of its own for the parts; one of 12000: 24 and 29, of 500: 17 and 22 (138 for the former's
//     decode alone with three stages and two CTAs per SM; 456 with a key per 16 lanes and no load in flight behind it).  Many short contexts with few heads a group go by rows instead, see paged_rows_kernel.
//   rows = 64 (chunks of short contexts, or in pages that a TMA box does not fit): a warp takes 16 rows and all keys of a stage, longest tiles first, bound by the
//     tensor instructions.  Where the tiles are few and the context is long, the CTAs of a cluster take key ranges and merge through distributed shared memory.  Two
//     chunks of 500 tokens beside 24 decoding requests, a step: 865 us when every token read all its keys, 110 by these tiles.
//   rows = 128 (chunks otherwise, the plan says which): see paged_wide_kernel, 87 us for the same step.
//
// Replaces the reference's dynamic-context attention (core/inference/contexts/dynamic_context.py + flash_attn_with_kvcache
// in attention.py:590-603) and this repo's earlier gather + einsum path (inference/dynamic.py).
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>
#include <cmath>
#include <string>

#include "b200_api.h"
#include "common.cuh"

namespace cg = cooperative_groups;

namespace b200 {
namespace {

thread_local std::string g_paged_err;

constexpr int kStageKeys = 64;
constexpr int kDecodeCtas = 3 * 148;

template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (kBf16) return pack_bf16x2(lo, hi);
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <bool kBf16>
__device__ __forceinline__ float2 unpack2(uint32_t v) {
  if constexpr (kBf16) return unpack_bf16x2(v);
  return __half22float2(*reinterpret_cast<const __half2*>(&v));
}
// c[16 x 8] += a[16 x 16] b[16 x 8]
template <bool kBf16>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBf16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// 16 bytes, zeros when !valid (the source is not read then)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
// Launches of a step overlap: every kernel lets the next one start once all its own CTAs run, and waits for the one before where it reads
// what that wrote: the write kernel's rows and zeroed counters (the first of the others).  The decode kernel beside chunks reads
// nothing of theirs, and what both read was complete before the first began: its first CTA waits before its end, so that the launch ends after theirs, which
// keeps the stream's order for what follows (pdl_allow_next, pdl_await_previous).  When all CTAs waited, those behind the first on an SM did not start before the
// chunks' end: 51 requests and two portions of 99 tokens x 8 heads of 128 took 38.7 us for 27.3, 150 drawn steps with portions 1.03 times as long.

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int D>
struct Smem {
  static constexpr int kPitch = D * 2 + 16;                          // bytes of a padded row: conflict-free ldmatrix
  static constexpr int kStage = 2 * kStageKeys * kPitch;             // K rows, then V rows
  static constexpr int kStages = D == 128 ? 2 : 3;
  static constexpr int kStatOff = kStages * kStage;                  // max and sum of [4 warps][16] or 64 rows
  static constexpr int kTotal = kStatOff + 2 * 64 * 4;
  static_assert(64 * D * 4 <= kStatOff, "after the last stage, partial accumulators reuse the ring");
};

struct PagedParams {
  PagedAttnArgs a;
  int group_shift, bs_shift;   // log2 of the group; of the block size, or -1
  int n_tiles;                 // chunks: tiles of this launch (its grid is n_tiles * ng * splits); decode: requests
  int splits;                  // chunks: key ranges of a tile; decode: CTAs, or 0 for one per (request, KV head)
  bool beside_chunks;          // decode: the launch before is the chunks'
  float row_scale;             // rows kernel: the scale as it was given
  uint32_t q_keep, q_sign;     // tiles: the kernels' running maxima want a positive scale: queries are negated for a negative one, zeros for zero
  bool behind_write;           // the launch before is the write of this call's keys, before which all else that is read was complete
  float* ws;                   // decode: two partials of 16 rows x (d + 2) per CTA
  int* arrived;                // decode: parts of each (request, KV head) that are in ws, zero at the start
};

// One tile's keys k0 .. k1 - 1 (stages aligned to k0): running maximum, sum and accumulator of this warp's rows g and g + 8.  RW row
// tiles of 16 share the CTA's four warps, the others split the keys of a stage.
template <int D, bool kBf16, int RW>
struct Tile {
  static constexpr int kWarpKeys = kStageKeys / (4 / RW), kNT = kWarpKeys / 8, kChunks = D / 8;
  // weights are at most one.  fp16 parts end at 2^-24, so there they and their sums are carried 2^15 times as large
  static constexpr float kUnit = kBf16 ? 1.f : 32768.f;
  using L = Smem<D>;
  float m[2], l[2], o[D / 8][4];

  // one stage's scores become weights; running maxima and sums follow, and where `plain` the product with V is added
  template <bool kHalf>
  __device__ __forceinline__ void weigh_and_add(float (&s)[kNT][4], uint32_t v_at, float sc, bool plain) {
#pragma unroll
    for (int i = 0; i < (kHalf ? 1 : 2); ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < kNT; ++j) mx = fmaxf(mx, fmaxf(s[j][2 * i], s[j][2 * i + 1]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float mn = fmaxf(m[i], mx);                              // unscaled: the largest score's weight is one whatever its size
      const float use = mn == -INFINITY ? 0.f : mn;                  // nothing visible yet: keep the arithmetic finite
      const float corr = m[i] == mn ? 1.f : exp2f((m[i] - use) * sc);     // also of a row without a key so far: its sums are zero
      m[i] = mn;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < kNT; ++j) {
        s[j][2 * i] = exp2f((s[j][2 * i] - use) * sc) * kUnit;
        s[j][2 * i + 1] = exp2f((s[j][2 * i + 1] - use) * sc) * kUnit;
        sum += s[j][2 * i] + s[j][2 * i + 1];
      }
      l[i] = l[i] * corr + sum;                                      // this thread's columns; the quad's are added at the end
      if (__any_sync(0xffffffffu, corr != 1.f)) {                    // seldom after the first stages
#pragma unroll
        for (int j = 0; j < D / 8; ++j) {
          o[j][2 * i] *= corr;
          o[j][2 * i + 1] *= corr;
          if (kHalf) {
            o[j][2] *= corr;
            o[j][3] *= corr;
          }
        }
      }
    }
    if (!plain) return;
#pragma unroll
    for (int k = 0; k < kWarpKeys / 16; ++k) {
      uint32_t part[3][4];
#pragma unroll
      for (int e = 0; e < 4; e += kHalf ? 2 : 1) {
        float x = s[2 * k + (e >> 1)][(e & 1) * 2], y = s[2 * k + (e >> 1)][(e & 1) * 2 + 1];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          part[q][e] = pack2<kBf16>(x, y);
          const float2 h = unpack2<kBf16>(part[q][e]);
          x -= h.x;
          y -= h.y;
        }
      }
      if (kHalf) {                                                   // the second parts ride in the rows that stand empty
        part[0][1] = part[1][0];
        part[0][3] = part[1][2];
        part[2][1] = part[2][3] = 0u;
      }
#pragma unroll
      for (int j = 0; j < D / 8; j += 2) {
        uint32_t b[4];
        ldsm4_t(v_at + k * 16 * L::kPitch + j * 16, b);
#pragma unroll
        for (int q = 0; q < 3; q += kHalf ? 2 : 1) {
          mma16816<kBf16>(o[j], part[q], b[0], b[1]);
          mma16816<kBf16>(o[j + 1], part[q], b[2], b[3]);
        }
      }
    }
  }

  __device__ __forceinline__ void run(const PagedParams& p, uint8_t* smem, const int32_t* bt, int hk, int t0, int n, int min_vis, int k0, int k1) {
    const PagedAttnArgs& a = p.a;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tg = lane & 3;
    const int G = 1 << p.group_shift, np = a.ng << p.group_shift, n_rows = n << p.group_shift;
    const bool half = RW == 1 && n_rows <= 8;                        // rows 8 to 15 of the tile stand empty
    const int n_stages = k1 > k0 ? (k1 - k0 + kStageKeys - 1) / kStageKeys : 0;
    // ---- gather of one stage into its ring buffer
    const uint32_t ring = smem_u32(smem);
    auto load = [&](int st) {
      const uint32_t dst = ring + (st % L::kStages) * L::kStage + (tid % kChunks) * 16;
#pragma unroll
      for (int i = 0; i < kStageKeys * kChunks / 128; ++i) {
        const int row = i * (128 / kChunks) + tid / kChunks, key = k0 + st * kStageKeys + row;
        const bool valid = key < k1;
        const int kk = valid ? key : k0;
        const int blk = p.bs_shift >= 0 ? kk >> p.bs_shift : kk / a.block_size;
        const int64_t slot = static_cast<int64_t>(bt[blk]) * a.block_size + (kk - blk * a.block_size);
        const int64_t off = (slot * a.ng + hk) * D + (tid % kChunks) * 8;
        cp_async16(dst + row * L::kPitch, static_cast<const uint16_t*>(a.k_cache) + off, valid);
        cp_async16(dst + (kStageKeys + row) * L::kPitch, static_cast<const uint16_t*>(a.v_cache) + off, valid);
      }
    };
#pragma unroll
    for (int st = 0; st < L::kStages - 1; ++st) {
      if (st < n_stages) load(st);
      cp_async_commit();
    }

    // ---- queries of this warp's rows g and g + 8, as A fragments
    const int wrow = RW == 1 ? 0 : warp * 16, wkey = RW == 1 ? warp * kWarpKeys : 0;
    uint32_t qf[D / 16][4];
    int vis[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = wrow + g + i * 8;
      const bool valid = row < n_rows;
      const int t = t0 + (valid ? row >> p.group_shift : 0);
      vis[i] = valid ? a.tok_len[t] : 0;
      const uint32_t* qp = reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(a.q) +
                                                             (static_cast<int64_t>(t) * np + hk * G + (valid ? row & (G - 1) : 0)) * D) + tg;
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        qf[k][i] = valid ? (qp[k * 8] & p.q_keep) ^ p.q_sign : 0u;
        qf[k][i + 2] = valid ? (qp[k * 8 + 4] & p.q_keep) ^ p.q_sign : 0u;
      }
    }
    m[0] = m[1] = -INFINITY;
    l[0] = l[1] = 0.f;
#pragma unroll
    for (int j = 0; j < D / 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
    const float sc = a.scale_log2;
    // ldmatrix row addresses: K in pairs of 8-key groups and 8-column groups, V in pairs of 8-column groups (transposed)
    const uint32_t k_off = (wkey + (lane & 7) + ((lane >> 4) << 3)) * L::kPitch + ((lane >> 3) & 1) * 16;
    const uint32_t v_off = (kStageKeys + wkey + (lane & 15)) * L::kPitch + (lane >> 4) * 16;

    for (int st = 0; st < n_stages; ++st) {
      cp_async_wait<L::kStages - 2>();
      __syncthreads();                                               // stage st has landed; the buffer of st - 1 is free
      if (st + L::kStages - 1 < n_stages) load(st + L::kStages - 1);
      cp_async_commit();
      const uint32_t buf = ring + (st % L::kStages) * L::kStage;
      const int kb = k0 + st * kStageKeys;
      const bool masked = kb + kStageKeys > min_vis || kb + kStageKeys > k1;
      bool plain = true;
      if (masked && n > 1) {
        // a value that only some rows see must not reach the others, not even as zero times infinity
        bool odd = false;
        const int from = max(0, min_vis - kb);
        for (int c = from * kChunks + tid; c < kStageKeys * kChunks; c += 128) {
          const uint4 w = *reinterpret_cast<const uint4*>(smem + (st % L::kStages) * L::kStage + (kStageKeys + c / kChunks) * L::kPitch + (c % kChunks) * 16);
          const uint32_t e = kBf16 ? 0x7f80u : 0x7c00u, ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) odd |= (ws[j] & e) == e || ((ws[j] >> 16) & e) == e;
        }
        plain = !__syncthreads_or(odd);
      }

      float s[kNT][4];
#pragma unroll
      for (int j = 0; j < kNT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[j][e] = 0.f;
#pragma unroll
      for (int k = 0; k < D / 16; ++k)
#pragma unroll
        for (int j = 0; j < kNT; j += 2) {
          uint32_t b[4];
          ldsm4(buf + k_off + j * 8 * L::kPitch + k * 32, b);
          mma16816<kBf16>(s[j], qf[k], b[0], b[1]);
          mma16816<kBf16>(s[j + 1], qf[k], b[2], b[3]);
        }
      if (masked) {
#pragma unroll
        for (int j = 0; j < kNT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (kb + wkey + j * 8 + tg * 2 + (e & 1) >= min(vis[e >> 1], k1)) s[j][e] = -INFINITY;
      }
      if (RW == 1 && half) weigh_and_add<true>(s, buf + v_off, sc, plain);
      else weigh_and_add<false>(s, buf + v_off, sc, plain);
      if (!plain) {
        const uint8_t* vrow = smem + (st % L::kStages) * L::kStage + (kStageKeys + wkey) * L::kPitch + tg * 4;
#pragma unroll
        for (int j = 0; j < kNT; ++j)
          for (int c = 0; c < 8; ++c) {                              // key kb + wkey + 8 j + c, whose weights lane c / 2 of the quad holds
            const float mine0 = (c & 1) ? s[j][1] : s[j][0], mine1 = (c & 1) ? s[j][3] : s[j][2];
            const float p0 = __shfl_sync(0xffffffffu, mine0, (lane & ~3) | (c >> 1)), p1 = __shfl_sync(0xffffffffu, mine1, (lane & ~3) | (c >> 1));
            const int key = kb + wkey + j * 8 + c;
            const bool see0 = key < vis[0], see1 = key < vis[1];
#pragma unroll
            for (int d = 0; d < D / 8; ++d) {
              const float2 v = unpack2<kBf16>(*reinterpret_cast<const uint32_t*>(vrow + (j * 8 + c) * L::kPitch + d * 16));
              if (see0) { o[d][0] = fmaf(p0, v.x, o[d][0]); o[d][1] = fmaf(p0, v.y, o[d][1]); }
              if (see1) { o[d][2] = fmaf(p1, v.x, o[d][2]); o[d][3] = fmaf(p1, v.y, o[d][3]); }
            }
          }
      }
    }
    cp_async_wait<0>();
    if (half) {
#pragma unroll
      for (int j = 0; j < D / 8; ++j) {
        o[j][0] += o[j][2];
        o[j][1] += o[j][3];
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
      l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    }
  }

  // this warp's accumulator as rows of a [64][D] fp32 buffer, with their maxima and sums
  __device__ __forceinline__ void spill(float* part, float* s_m, float* s_l) const {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = warp * 16 + g + i * 8;
#pragma unroll
      for (int j = 0; j < D / 8; ++j) *reinterpret_cast<float2*>(part + row * D + j * 8 + tg * 2) = make_float2(o[j][2 * i], o[j][2 * i + 1]);
      if (tg == 0) {
        s_m[row] = m[i];
        s_l[row] = l[i];
      }
    }
  }
};

// running sum of weighted partials; no keys: zeros
struct Merge {
  float sc, M = -INFINITY, L = 0.f;
  float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
  __device__ __forceinline__ explicit Merge(float scale_log2) : sc(scale_log2) {}
  __device__ __forceinline__ void add(float m, float l, const float4& v) {
    const float f = exp2f((m - M) * sc);
    L = fmaf(l, f, L);
    if (l > 0.f) {
      O.x = fmaf(v.x, f, O.x); O.y = fmaf(v.y, f, O.y); O.z = fmaf(v.z, f, O.z); O.w = fmaf(v.w, f, O.w);
    }
  }
  template <bool kBf16> __device__ __forceinline__ uint2 result() const {
    const float inv = L > 0.f ? 1.f / L : L;                         // 0 without keys; NaN stays NaN
    return make_uint2(pack2<kBf16>(O.x * inv, O.y * inv), pack2<kBf16>(O.z * inv, O.w * inv));
  }
};

// ---- decode: the stages of every (request, KV head), in one line
// request r (or token, without cu) as this launch sees it: its tokens and its stages, 0 for requests that are chunks
struct Item { int t0, n, stages, max_vis, min_vis; };
__device__ __forceinline__ Item decode_item(const PagedParams& p, int r) {
  Item it{0, 0, 0, 0, 0x7fffffff};
  if (r >= p.n_tiles) return it;
  it.t0 = p.a.cu == nullptr ? r : p.a.cu[r];
  it.n = p.a.cu == nullptr ? 1 : p.a.cu[r + 1] - it.t0;
  if ((it.n << p.group_shift) > 16) it.n = 0;
  for (int i = 0; i < it.n; ++i) {
    const int v = p.a.tok_len[it.t0 + i];
    it.max_vis = max(it.max_vis, v);
    it.min_vis = min(it.min_vis, v);
  }
  it.stages = it.n > 0 ? max(1, (it.max_vis + kStageKeys - 1) / kStageKeys) : 0;      // a request without keys still gets its zeros written
  return it;
}
// where the line is cut: its first `rem` parts have q + 1 stages, the others q
struct Cuts {
  int q, rem;
  __device__ __forceinline__ Cuts(int line, int parts) : q(line / parts), rem(line % parts) {}
  __device__ __forceinline__ int at(int i) const { return q * i + min(i, rem); }
  __device__ __forceinline__ int part_of(int x) const { return x < rem * (q + 1) ? x / (q + 1) : rem + (x - rem * (q + 1)) / max(q, 1); }
};

// An item that cuts fell into: parts i0 .. i1 of it are in ws, the CTA that came last puts them together.  slot(i): part i
template <int D, bool kBf16, typename Slot, typename Out>
__device__ __forceinline__ void merge_parts(float scale_log2, uint8_t* smem, int rows, int i0, int i1, Slot slot, Out out_row) {
  float* s_inv = reinterpret_cast<float*>(smem);                     // [16]
  float4* s_o = reinterpret_cast<float4*>(smem + 64);                // [128]
  float* s_f = reinterpret_cast<float*>(smem + 64 + 2048);           // [16][parts]: the parts' weights
  static_assert(64 + 2048 + 16 * kDecodeCtas * 4 <= Smem<D>::kStatOff, "over the ring");
  const int parts = i1 - i0 + 1, lane = threadIdx.x & 31;
  for (int row = threadIdx.x >> 5; row < rows; row += 4) {
    float M = -INFINITY, L = 0.f;
    float* f_row = s_f + row * parts;
    for (int i = lane; i < parts; i += 32) {
      f_row[i] = __ldcg(slot(i0 + i) + 16 * D + row);
      M = fmaxf(M, f_row[i]);
    }
    M = warp_max(M);
    const float use = M == -INFINITY ? 0.f : M;
    for (int i = lane; i < parts; i += 32) {
      const float f = exp2f((f_row[i] - use) * scale_log2), l = __ldcg(slot(i0 + i) + 16 * D + 16 + row);
      f_row[i] = l > 0.f ? f : 0.f;
      L = fmaf(l, f, L);
    }
    L = warp_sum(L);
    if (lane == 0) s_inv[row] = L > 0.f ? 1.f / L : L;               // 0 without keys; NaN stays NaN
  }
  __syncthreads();
  // where the rows leave threads over, these take every second or fourth part
  const int quads = rows * (D / 4), share = quads <= 32 ? 4 : (quads <= 64 ? 2 : 1), step = 128 / share;
  const int mine = static_cast<int>(threadIdx.x) / step, thread = static_cast<int>(threadIdx.x) % step;
  for (int idx0 = 0; idx0 < quads; idx0 += step) {
    const int idx = idx0 + thread, row = idx / (D / 4), col = (idx % (D / 4)) * 4;
    const bool valid = idx < quads;
    float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid) {
#pragma unroll 8
      for (int i = mine; i < parts; i += share) {
        const float f = s_f[row * parts + i];
        const float4 v = __ldcg(reinterpret_cast<const float4*>(slot(i0 + i) + row * D + col));
        O.x = fmaf(v.x, f, O.x); O.y = fmaf(v.y, f, O.y); O.z = fmaf(v.z, f, O.z); O.w = fmaf(v.w, f, O.w);
      }
    }
    if (share > 1) {                                                 // then idx0 is 0: one trip
      s_o[threadIdx.x] = O;
      __syncthreads();
      if (mine == 0) {
        for (int k = 1; k < share; ++k) {
          const float4 v = s_o[k * step + thread];
          O.x += v.x; O.y += v.y; O.z += v.z; O.w += v.w;
        }
      }
    }
    if (mine == 0 && valid) {
      const float inv = s_inv[row];
      *reinterpret_cast<uint2*>(out_row(row) + col) = make_uint2(pack2<kBf16>(O.x * inv, O.y * inv), pack2<kBf16>(O.z * inv, O.w * inv));
    }
  }
}

// kCut: a part of the line per CTA, else one item
template <int D, bool kBf16, bool kCut>
__global__ void __launch_bounds__(128, 3) paged_decode_kernel(const PagedParams p) {
  using L = Smem<D>;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ int s_inside, s_r, s_last, s_sum[2][4];
  __shared__ Item s_item;
  const PagedAttnArgs& a = p.a;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = 1 << p.group_shift, np = a.ng << p.group_shift;
  pdl_allow_next();
  if (!p.beside_chunks && !p.behind_write) pdl_await_previous();
  int at, end, parts_of_line = 0, line = 0, r = 0, inside = 0;
  Item it;
  if constexpr (!kCut) {
    r = blockIdx.x / a.ng;
    it = decode_item(p, r);
    at = 0;
    end = it.stages;
    inside = static_cast<int>(blockIdx.x % a.ng) * it.stages;
  } else {
    // a request per thread; the first 128 stay in registers for the search
    Item mine = decode_item(p, tid);
    int total = mine.stages;
    for (int r0 = tid + 128; r0 < p.n_tiles; r0 += 128) total += decode_item(p, r0).stages;
    total = __reduce_add_sync(0xffffffffu, total);
    if (lane == 0) s_sum[1][warp] = total;
    __syncthreads();
    total = s_sum[1][0] + s_sum[1][1] + s_sum[1][2] + s_sum[1][3];
    line = total * a.ng;
    parts_of_line = p.splits;
    const Cuts cuts(line, p.splits);
    at = cuts.at(blockIdx.x);
    end = cuts.at(blockIdx.x + 1);
    // the request that this CTA's part of the line starts in
    int seen = 0;
    for (int r0 = 0, turn = 0; r0 < p.n_tiles && at < end; r0 += 128, turn ^= 1) {
      if (r0 > 0) mine = decode_item(p, r0 + tid);
      int incl = mine.stages;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) s_sum[turn][warp] = incl;
      __syncthreads();
      int before = seen;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        if (w < warp) before += s_sum[turn][w];
        seen += s_sum[turn][w];
      }
      const int first = (before + incl - mine.stages) * a.ng;
      if (mine.stages > 0 && at >= first && at < first + mine.stages * a.ng) {
        s_r = r0 + tid;
        s_item = mine;
        s_inside = at - first;
      }
      if (seen * a.ng > at) break;
    }
  }
  if (at >= end) {
    if ((p.beside_chunks && blockIdx.x == 0) || p.behind_write) pdl_await_previous();
    return;
  }
  if constexpr (kCut) {
    __syncthreads();
    r = s_r;
    inside = s_inside;
    it = s_item;
  }
  float* part = reinterpret_cast<float*>(smem);                      // [4 warps][16][D] over the ring
  float* s_m = reinterpret_cast<float*>(smem + L::kStatOff);
  float* s_l = s_m + 64;
  Tile<D, kBf16, 1> tile;
  const Cuts cuts(kCut ? line : 0, kCut ? parts_of_line : 1);
  if (p.behind_write) pdl_await_previous();                          // the new keys are in their pages, the counters zero
  while (true) {
    const int hk = inside / it.stages, st0 = inside % it.stages;
    const int n_st = min(it.stages - st0, end - at);
    tile.run(p, smem, a.block_table + static_cast<int64_t>(a.tok_req[it.t0]) * a.max_blocks, hk, it.t0, it.n, it.min_vis, st0 * kStageKeys,
             min(it.max_vis, (st0 + n_st) * kStageKeys));
    __syncthreads();                                                 // the ring is not read any more
    tile.spill(part, s_m, s_l);
    __syncthreads();
    const bool whole = n_st == it.stages;
    auto out_row = [&](int row) {
      return static_cast<uint16_t*>(a.out) + (static_cast<int64_t>(it.t0 + (row >> p.group_shift)) * np + hk * G + (row & (G - 1))) * D;
    };
    // slot 0: a part that starts inside its item; slot 1: one that starts with it
    float* ws = p.ws + (static_cast<int64_t>(blockIdx.x) * 2 + (st0 == 0 ? 1 : 0)) * (16 * (D + 2));
    for (int idx = tid; idx < (it.n << p.group_shift) * (D / 4); idx += 128) {
      const int row = idx / (D / 4), col = (idx % (D / 4)) * 4;
      Merge x(a.scale_log2);
#pragma unroll
      for (int w = 0; w < 4; ++w) x.M = fmaxf(x.M, s_m[w * 16 + row]);
      if (x.M > -INFINITY) {
#pragma unroll
        for (int w = 0; w < 4; ++w) x.add(s_m[w * 16 + row], s_l[w * 16 + row], *reinterpret_cast<const float4*>(part + (w * 16 + row) * D + col));
      }
      if (whole) {
        *reinterpret_cast<uint2*>(out_row(row) + col) = x.result<kBf16>();
      } else {
        *reinterpret_cast<float4*>(ws + row * D + col) = x.O;
        if (col == 0) {
          ws[16 * D + row] = x.M;
          ws[16 * D + 16 + row] = x.L;
        }
      }
    }
    if (kCut && !whole) {
      const int first = at - st0, i0 = cuts.part_of(first), i1 = cuts.part_of(first + it.stages - 1);
      __threadfence();
      __syncthreads();                                               // this part is in ws for whoever counts it
      if (tid == 0) s_last = atomicAdd(p.arrived + r * a.ng + hk, 1) == i1 - i0;
      __syncthreads();
      if (s_last) {
        __threadfence();
        merge_parts<D, kBf16>(a.scale_log2, smem, it.n << p.group_shift, i0, i1,
                              [&](int i) { return p.ws + (static_cast<int64_t>(i) * 2 + (i > i0 || cuts.at(i) > first ? 0 : 1)) * (16 * (D + 2)); }, out_row);
      }
    }
    at += n_st;
    inside += n_st;
    if (at >= end) break;
    if (inside == it.stages * a.ng) {                                // on to the next request that is not a chunk
      inside = 0;
      do it = decode_item(p, ++r); while (it.stages == 0 && r < p.n_tiles);
      if (it.stages == 0) break;
    }
    __syncthreads();                                                 // the partials have been read; the ring fills again
  }
  if (p.beside_chunks && blockIdx.x == 0) pdl_await_previous();
}

// ---- decode with few rows per key and many short contexts: a tile of the kernels above is mostly empty and its start and end cost more than
// its keys.  D / 8 lanes share a key (16 bytes each), the CTA's key groups walk a token's keys side by side in fp32 multiply-adds and merge at the
// end; small CTAs, many per SM, hide the latency that the tiles' rings hide there.
template <bool kBf16>
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = unpack2<kBf16>(w[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}
template <int D, int G, bool kBf16>
__global__ void __launch_bounds__(128, G == 1 ? 12 : G == 2 ? 7 : 4) paged_rows_kernel(const PagedParams p) {
  constexpr int kLanes = D / 8, kWarpKeys = 32 / kLanes, kGroups = 4 * kWarpKeys;
  __shared__ float s_m[kGroups][G], s_l[kGroups][G];
  __shared__ float s_acc[kGroups][G][D];
  const PagedAttnArgs& a = p.a;
  pdl_allow_next();
  if (!p.beside_chunks) pdl_await_previous();
  const int r = blockIdx.x / a.ng, hk = blockIdx.x % a.ng, np = a.ng * G;
  const Item it = decode_item(p, r);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lk = lane % kLanes, grp = warp * kWarpKeys + lane / kLanes;
  // the key groups of a warp run different trip counts at the end of a context: shuffles name only the group's lanes
  const unsigned gmask = ((1u << kLanes) - 1u) << (lane / kLanes * kLanes);
  for (int t = it.t0; t < it.t0 + it.n; ++t) {
    const int len = a.tok_len[t];
    float q[G][8], m[G], l[G], acc[G][8];
    const uint16_t* qp = static_cast<const uint16_t*>(a.q) + (static_cast<int64_t>(t) * np + hk * G) * D + lk * 8;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      unpack8<kBf16>(*reinterpret_cast<const uint4*>(qp + g * D), q[g]);
      m[g] = -INFINITY;
      l[g] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        q[g][j] *= p.row_scale;
        acc[g][j] = 0.f;
      }
    }
    const int32_t* bt = a.block_table + static_cast<int64_t>(a.tok_req[t]) * a.max_blocks;
    for (int k = grp; k < len; k += kGroups) {
      const int blk = p.bs_shift >= 0 ? k >> p.bs_shift : k / a.block_size;
      const int64_t slot = static_cast<int64_t>(bt[blk]) * a.block_size + (k - blk * a.block_size);
      const int64_t off = (slot * a.ng + hk) * D + lk * 8;
      const uint4 kraw = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(a.k_cache) + off);
      const uint4 vraw = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(a.v_cache) + off);
      float kf[8], vf[8];
      unpack8<kBf16>(kraw, kf);
      unpack8<kBf16>(vraw, vf);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) s = fmaf(q[g][j], kf[j], s);
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(gmask, s, o, kLanes);
        const float mn = fmaxf(m[g], s);
        const float corr = exp2f(m[g] - mn), w = exp2f(s - mn);
        l[g] = l[g] * corr + w;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[g][j] = fmaf(acc[g][j], corr, w * vf[j]);
        m[g] = mn;
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (lk == 0) {
        s_m[grp][g] = m[g];
        s_l[grp][g] = l[g];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s_acc[grp][g][lk * 8 + j] = acc[g][j];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < G * D; idx += 128) {
      const int g = idx / D, d = idx % D;
      float M = -INFINITY, L = 0.f, O = 0.f;
#pragma unroll
      for (int c = 0; c < kGroups; ++c) M = fmaxf(M, s_m[c][g]);
      if (M > -INFINITY) {
#pragma unroll
        for (int c = 0; c < kGroups; ++c) {
          const float w = exp2f(s_m[c][g] - M);
          L = fmaf(s_l[c][g], w, L);
          O = fmaf(s_acc[c][g][d], w, O);
        }
      }
      const uint32_t o16 = pack2<kBf16>(L > 0.f ? O / L : 0.f, 0.f);
      static_cast<uint16_t*>(a.out)[(static_cast<int64_t>(t) * np + hk * G + g) * D + d] = static_cast<uint16_t>(o16);
    }
    __syncthreads();                                                 // the groups' shares have been read
  }
  if (p.beside_chunks && blockIdx.x == 0) pdl_await_previous();
}

// ---- chunks
// one warp: that run of `per_tile` tokens among the requests with more than 16 rows: its first token, and how many it has
__device__ __forceinline__ void find_tile(const PagedParams& p, int per_tile, int tile_at, int* s_tile) {
  const PagedAttnArgs& a = p.a;
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int r0 = 0; r0 < a.n_seqs; r0 += 32) {
    const int r = r0 + lane;
    const int c0 = r < a.n_seqs ? a.cu[r] : 0, c1 = r < a.n_seqs ? a.cu[r + 1] : 0, len = c1 - c0;
    const int tiles = (len << p.group_shift) > 16 ? (len + per_tile - 1) / per_tile : 0;
    int incl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int first = before + incl - tiles;
    if (tiles > 0 && tile_at >= first && tile_at < first + tiles) {
      const int off = (tile_at - first) * per_tile;
      s_tile[0] = c0 + off;
      s_tile[1] = min(per_tile, len - off);
    }
    before += __shfl_sync(0xffffffffu, incl, 31);
    if (before > tile_at) break;
  }
  if (lane == 0 && before <= tile_at) s_tile[1] = 0;                 // more tiles launched than there are
}
// the partials of a cluster's CTAs, behind its barrier: thread `first` of all of them
template <int D, bool kBf16, typename Out>
__device__ __forceinline__ void merge_cluster(const PagedParams& p, int first, int threads, int n_rows, const float* part, const float* s_m, const float* s_l, Out out_row) {
  cg::cluster_group cluster = cg::this_cluster();
  for (int idx = first; idx < n_rows * (D / 4); idx += p.splits * threads) {
    const int row = idx / (D / 4), col = (idx % (D / 4)) * 4;
    Merge x(p.a.scale_log2);
    for (int c = 0; c < p.splits; ++c) x.M = fmaxf(x.M, *cluster.map_shared_rank(s_m + row, c));
    if (x.M > -INFINITY) {
      for (int c = 0; c < p.splits; ++c)
        x.add(*cluster.map_shared_rank(s_m + row, c), *cluster.map_shared_rank(s_l + row, c),
              *cluster.map_shared_rank(reinterpret_cast<const float4*>(part + row * D + col), c));
    }
    *reinterpret_cast<uint2*>(out_row(row) + col) = x.result<kBf16>();
  }
}

template <int D, bool kBf16>
__global__ void __launch_bounds__(128, 2) paged_chunk_kernel(const PagedParams p) {
  using L = Smem<D>;
  constexpr int kRows = 64;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ int s_tile[2];
  const PagedAttnArgs& a = p.a;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tg = lane & 3;
  const int rank = static_cast<int>(blockIdx.x) % p.splits, item = static_cast<int>(blockIdx.x) / p.splits;
  const int hk = item % a.ng, tile_at = p.n_tiles - 1 - item / a.ng; // later tiles of a chunk see more keys: they go first
  const int G = 1 << p.group_shift, np = a.ng << p.group_shift;
  pdl_await_previous();
  pdl_allow_next();
  if (warp == 0) find_tile(p, kRows >> p.group_shift, tile_at, s_tile);
  __syncthreads();
  const int t0 = s_tile[0], n = s_tile[1];
  if (n == 0) return;
  const int n_rows = n << p.group_shift;
  // keys that the tile's tokens see: all of them below min_vis, some up to max_vis
  int max_vis = 0, min_vis = 0x7fffffff;
  for (int i = lane; i < n; i += 32) {
    const int v = a.tok_len[t0 + i];
    max_vis = max(max_vis, v);
    min_vis = min(min_vis, v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    max_vis = max(max_vis, __shfl_xor_sync(0xffffffffu, max_vis, o));
    min_vis = min(min_vis, __shfl_xor_sync(0xffffffffu, min_vis, o));
  }
  const int per = ((max_vis + p.splits - 1) / p.splits + kStageKeys - 1) / kStageKeys * kStageKeys;
  const int k0 = rank * per, k1 = min(max_vis, k0 + per);
  Tile<D, kBf16, 4> tile;
  tile.run(p, smem, a.block_table + static_cast<int64_t>(a.tok_req[t0]) * a.max_blocks, hk, t0, n, min_vis, k0, k1);
  auto out_row = [&](int row) {
    return static_cast<uint16_t*>(a.out) + (static_cast<int64_t>(t0 + (row >> p.group_shift)) * np + hk * G + (row & (G - 1))) * D;
  };
  if (p.splits == 1) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = warp * 16 + g + i * 8;
      if (row >= n_rows) continue;
      const float inv = tile.l[i] > 0.f ? 1.f / tile.l[i] : tile.l[i];
      uint32_t* dst = reinterpret_cast<uint32_t*>(out_row(row)) + tg;
#pragma unroll
      for (int j = 0; j < D / 8; ++j) dst[j * 4] = pack2<kBf16>(tile.o[j][2 * i] * inv, tile.o[j][2 * i + 1] * inv);
    }
    return;
  }
  // ---- the cluster's partials
  __syncthreads();                                                   // the ring is not read any more
  float* part = reinterpret_cast<float*>(smem);                      // [64][D]
  float* s_m = reinterpret_cast<float*>(smem + L::kStatOff);
  float* s_l = s_m + 64;
  tile.spill(part, s_m, s_l);
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  merge_cluster<D, kBf16>(p, rank * 128 + tid, 128, n_rows, part, s_m, s_l, out_row);
  cluster.sync();                                                    // no CTA leaves while another reads its partials
}

// ---- chunks on tcgen05: pages of 8 to 64 slots, or whole multiples of 64, which a TMA box can fetch.  A tile is 128 rows.  Its stages of 64
// keys go through a ring of three; scores and weights have two TMEM buffers each, so that a stage's scores are made under the one before's
// exponentials.  The weights' three parts (see weigh_and_add) lie side by side in TMEM as A operands of three products with the same V.  Two threads
// share a row, 32 keys each.  Where only some rows see a stage's keys, its V is looked at in shared memory first: keys that nobody sees
// become zeros, and values that are not finite are taken out and added by hand to the rows that see them.
// Bound by the chain of a stage and by the products (8 + 24 MMAs a stage at d = 128).  Two portions of 500 tokens x 32 / 8 heads of 128 beside 24 decoding
// requests: 87 us the step, 110 with the 64-row tiles; four of 512 and one request 83 and 160.  Registers and ring are kept so small that a decode CTA
// fits beside one of these.
template <int D>
struct WideSmem {
  static constexpr int kDC = D / 64, kRows = 128, kStages = 3;
  static constexpr int kQ = kRows * 128 * kDC, kKV = kStageKeys * 128 * kDC;
  static constexpr int kKOff = kQ, kVOff = kKOff + kStages * kKV;
  static constexpr int kExOff = kVOff + kStages * kKV;               // [parity][half][row]: partial maxima, then sums
  static constexpr int kStatOff = kExOff + 2 * 2 * kRows * 4;        // max and sum of a row, for the cluster
  static constexpr int kBarOff = kStatOff + 2 * kRows * 4;
  static constexpr int kTotal = kBarOff + 256 + 1024;                // + alignment slack
  static_assert(kRows * D * 4 <= 2 * kStages * kKV, "after the last stage, partial accumulators reuse the ring");
};
constexpr int kWideThreads = 384, kWideTries = 1 << 20;
__device__ int g_paged_error = 0;

// bounded: a wait that runs out is noted, and every later one ends at once.  At its end the CTA then leaves g_paged_error for paged_status, fills its rows with
// NaN and waits (always within kWideTries) for its own copies and MMAs in flight.
__device__ __forceinline__ void wide_wait(uint64_t* bar, uint32_t parity, volatile int* failed, int limit = kWideTries) {
  for (int left = limit; left > 0; --left) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return;
    if ((left & 255) == 0 && __any_sync(0xffffffffu, *failed != 0)) return;
  }
  *failed = 1;
}
__device__ __forceinline__ void wide_arrive(uint64_t* bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
// whether any of the 256 softmax threads says so; they meet here
__device__ __forceinline__ bool wide_any(bool mine) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred P, Q;\n\t"
      "setp.ne.u32 P, %1, 0;\n\t"
      "barrier.cta.red.or.pred Q, 2, 256, P;\n\t"
      "selp.u32 %0, 1, 0, Q;\n\t}\n"
      : "=r"(r) : "r"(mine ? 1u : 0u) : "memory");
  return r != 0;
}

// at most 96 registers (a bound of 576 threads): with 384 threads, room for a decode CTA's
template <int D, bool kBf16>
__global__ void __launch_bounds__(576, 1)
paged_wide_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const PagedParams p) {
  using L = WideSmem<D>;
  constexpr int kS = L::kStages;
  constexpr float kUnit = kBf16 ? 1.f : 32768.f;                     // see Tile
  constexpr float kSlack = kBf16 ? 8.f : 0.f;                        // accumulators are rescaled when a maximum has grown by 2^8; fp16 weights stay below one
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ int s_tile[2];
  float* s_ex = reinterpret_cast<float*>(smem + L::kExOff);
  uint64_t* k_full = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* k_empty = k_full + kS;
  uint64_t* v_full = k_empty + kS;
  uint64_t* v_empty = v_full + kS;
  uint64_t* s_full = v_empty + kS;     // 2
  uint64_t* s_read = s_full + 2;       // 2: scores are in registers
  uint64_t* p_ready = s_read + 2;      // 2
  uint64_t* pv_done = p_ready + 2;     // 2: the weights' columns are free, the accumulator is up to date
  uint64_t* drained = pv_done + 2;     // 1, after a wait that ran out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
  volatile int* failed = reinterpret_cast<volatile int*>(drained + 2);
  const PagedAttnArgs& a = p.a;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(blockIdx.x) % p.splits, item = static_cast<int>(blockIdx.x) / p.splits;
  const int hk = item % a.ng, tile_at = p.n_tiles - 1 - item / a.ng;
  const int G = 1 << p.group_shift, np = a.ng << p.group_shift, per_tile = L::kRows >> p.group_shift;
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < kS; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_read[i], 8); mbar_init(&p_ready[i], 8); mbar_init(&pv_done[i], 1); }
    mbar_init(drained, 2);
    *failed = 0;
    mbar_fence_init();
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  if (warp == 2) tmem_alloc<512>(tmem_slot);
  pdl_await_previous();
  pdl_allow_next();
  if (warp == 0) find_tile(p, per_tile, tile_at, s_tile);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_O = tmem, tmem_S = tmem + 128, tmem_P = tmem + 256;      // S: 2 x 64 columns; P: 2 x 3 x 32
  const int t0 = s_tile[0], n = s_tile[1];
  if (n == 0) {
    if (warp == 2) tmem_dealloc<512>(tmem);
    return;
  }
  const int n_rows = n << p.group_shift;
  int max_vis = 0, min_vis = 0x7fffffff;
  for (int i = lane; i < n; i += 32) {
    const int v = a.tok_len[t0 + i];
    max_vis = max(max_vis, v);
    min_vis = min(min_vis, v);
  }
  max_vis = __reduce_max_sync(0xffffffffu, max_vis);
  min_vis = __reduce_min_sync(0xffffffffu, min_vis);
  const int per = ((max_vis + p.splits - 1) / p.splits + kStageKeys - 1) / kStageKeys * kStageKeys;
  const int k0 = rank * per, k1 = min(max_vis, k0 + per), n_st = k1 > k0 ? (k1 - k0 + kStageKeys - 1) / kStageKeys : 0;
  const int32_t* bt = a.block_table + static_cast<int64_t>(a.tok_req[t0]) * a.max_blocks;
  uint8_t *sQ = smem, *sK = smem + L::kKOff, *sV = smem + L::kVOff;
  int n_loaded = 0;                                                  // warp 0: stages whose copies it has started
  auto out_row = [&](int row) {
    return static_cast<uint16_t*>(a.out) + (static_cast<int64_t>(t0 + (row >> p.group_shift)) * np + hk * G + (row & (G - 1))) * D;
  };
  float m = -INFINITY, l = 0.f;                                      // softmax threads: the row's

  if (warp == 0) {
    // ---- copies: a lane per page
    const int box = min(a.block_size, kStageKeys);
    fence_proxy_async_all();                                         // the new keys were written by plain stores
    for (; n_loaded < n_st; ++n_loaded) {
      const int st = n_loaded % kS, key = k0 + n_loaded * kStageKeys + lane * box;
      const bool mine = lane * box < kStageKeys && key < k1;
      const int pages = __popc(__ballot_sync(0xffffffffu, mine));
      int slot = 0;
      if (mine) {
        const int blk = p.bs_shift >= 0 ? key >> p.bs_shift : key / a.block_size;
        slot = bt[blk] * a.block_size + (key - blk * a.block_size);
      }
      wide_wait(&k_empty[st], ((n_loaded / kS) & 1) ^ 1, failed, a.wait_limit);
      wide_wait(&v_empty[st], ((n_loaded / kS) & 1) ^ 1, failed, a.wait_limit);
      if (__any_sync(0xffffffffu, *failed != 0)) break;
      for (int kv = 0; kv < 2; ++kv) {
        uint64_t* full = kv == 0 ? &k_full[st] : &v_full[st];
        if (lane == 0) mbar_arrive_expect_tx(full, pages * box * D * 2);
        __syncwarp();
        if (mine) {
          uint8_t* dst = (kv == 0 ? sK : sV) + st * L::kKV + lane * box * 128;
          for (int c = 0; c < L::kDC; ++c) tma_load_3d(kv == 0 ? &map_k : &map_v, full, dst + c * (kStageKeys * 128), c * 64, hk, slot);
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    // ---- S = Q K^T
    constexpr uint32_t idesc = make_idesc_f16(kBf16, L::kRows, kStageKeys, false, false);
    const uint64_t q_desc = make_smem_desc_sw128(smem_u32(sQ), 1024, 0), k_desc = make_smem_desc_sw128(smem_u32(sK), 1024, 0);
    named_bar_sync(3, 288);                                          // the queries are in place
    for (int j = 0; j < n_st; ++j) {
      const int st = j % kS, b = j & 1;
      wide_wait(&k_full[st], (j / kS) & 1, failed, a.wait_limit);
      if (j >= 2) wide_wait(&s_read[b], ((j >> 1) - 1) & 1, failed, a.wait_limit);
      if (__any_sync(0xffffffffu, *failed != 0)) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_f16_ss(tmem_S + b * kStageKeys, q_desc + (((k >> 2) * (L::kRows * 128) + (k & 3) * 32) >> 4),
                      k_desc + ((st * L::kKV + (k >> 2) * (kStageKeys * 128) + (k & 3) * 32) >> 4), idesc, k != 0 ? 1u : 0u);
        umma_commit(&s_full[b]);
        umma_commit(&k_empty[st]);
      }
      __syncwarp();
    }
  } else if (warp == 2) {
    // ---- O += P V, part by part
    constexpr uint32_t idesc = make_idesc_f16(kBf16, L::kRows, D, false, true);
    const uint64_t v_desc = make_smem_desc_sw128(smem_u32(sV), 1024, kStageKeys * 128);
    for (int j = 0; j < n_st; ++j) {
      const int st = j % kS, b = j & 1;
      wide_wait(&v_full[st], (j / kS) & 1, failed, a.wait_limit);
      wide_wait(&p_ready[b], (j >> 1) & 1, failed, a.wait_limit);
      if (__any_sync(0xffffffffu, *failed != 0)) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < kStageKeys / 16; ++k)
#pragma unroll
          for (int q = 0; q < 3; ++q)
            umma_f16_ts(tmem_O, tmem_P + b * 96 + q * 32 + k * 8, v_desc + ((st * L::kKV + k * 16 * 128) >> 4), idesc, j != 0 || k != 0 || q != 0 ? 1u : 0u);
        umma_commit(&pv_done[b]);
        umma_commit(&v_empty[st]);
      }
      __syncwarp();
    }
  } else if (warp >= 4) {
    // ---- softmax: half of a stage's keys of a row
    const int tid = threadIdx.x - 128, half = tid >> 7, quad = warp & 3, r = quad * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(quad * 32) << 16;
    for (int i = tid; i < L::kRows * (D / 8); i += 256) {            // queries, 16 bytes at a time, 128B-swizzled
      const int row = i / (D / 8), ch = i % (D / 8);
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (row < n_rows) {
        w = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(a.q) +
                                            (static_cast<int64_t>(t0 + (row >> p.group_shift)) * np + hk * G + (row & (G - 1))) * D + ch * 8);
        w.x = (w.x & p.q_keep) ^ p.q_sign; w.y = (w.y & p.q_keep) ^ p.q_sign; w.z = (w.z & p.q_keep) ^ p.q_sign; w.w = (w.w & p.q_keep) ^ p.q_sign;
      }
      st_shared_v4(smem_u32(sQ) + (ch >> 3) * (L::kRows * 128) + row * 128 + (((ch & 7) ^ (row & 7)) << 4), w.x, w.y, w.z, w.w);
    }
    fence_proxy_async_smem();
    named_bar_sync(3, 288);
    const int vis = r < n_rows ? a.tok_len[t0 + (r >> p.group_shift)] : 0;
    const float sc = a.scale_log2;
    const uint32_t tO = tmem_O + half * (D / 2) + lanes;
    for (int j = 0; j < n_st; ++j) {
      const int b = j & 1, kb = k0 + j * kStageKeys;
      uint32_t v[32];
      float s[32];
      wide_wait(&s_full[b], (j >> 1) & 1, failed, a.wait_limit);
      tc_fence_after();
      tmem_ld_32x32(tmem_S + b * kStageKeys + half * 32 + lanes, v);
      tmem_ld_wait();
      tc_fence_before();
      wide_arrive(&s_read[b]);
#pragma unroll
      for (int i = 0; i < 32; ++i) s[i] = __uint_as_float(v[i]);
      bool odd = false;
      if (kb + kStageKeys > min_vis || kb + kStageKeys > k1) {
        const int lim = min(vis, k1) - kb - half * 32;
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i >= lim) s[i] = -INFINITY;
        // V of keys that nobody sees, and values that only some rows see and that are not finite: not as zero times infinity
        wide_wait(&v_full[j % kS], (j / kS) & 1, failed, a.wait_limit);
        const int from = max(0, min(min_vis, k1) - kb), none = k1 - kb;
        uint8_t* tile = sV + (j % kS) * L::kKV;
        bool found = false;
        for (int i = tid; i < (kStageKeys - from) * (D / 8); i += 256) {
          const int row = from + i / (D / 8), ch = i % (D / 8);
          uint4* at = reinterpret_cast<uint4*>(tile + (ch >> 3) * (kStageKeys * 128) + row * 128 + (((ch & 7) ^ (row & 7)) << 4));
          if (row >= none) {
            *at = make_uint4(0u, 0u, 0u, 0u);
          } else if (n > 1) {
            const uint32_t e = kBf16 ? 0x7f80u : 0x7c00u;
            uint4 w4 = *at;
            uint32_t ws[4] = {w4.x, w4.y, w4.z, w4.w};
            bool here = false;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if ((ws[q] & e) == e) { ws[q] &= 0xffff0000u; here = true; }
              if (((ws[q] >> 16) & e) == e) { ws[q] &= 0x0000ffffu; here = true; }
            }
            if (here) {
              *at = make_uint4(ws[0], ws[1], ws[2], ws[3]);
              found = true;
            }
          }
        }
        fence_proxy_async_smem();
        odd = wide_any(found);
      }
      float mx = -INFINITY;
#pragma unroll
      for (int i = 0; i < 32; ++i) mx = fmaxf(mx, s[i]);
      float* slot = s_ex + (j & 1) * (2 * L::kRows);
      slot[half * L::kRows + r] = mx;
      named_bar_sync(4 + quad, 64);                                  // the two warps of these rows
      const float mn = fmaxf(m, fmaxf(mx, slot[(half ^ 1) * L::kRows + r]));
      const bool grow = mn > m && !((mn - m) * sc <= kSlack);        // from nothing at the first visible key: the difference is infinite
      if (__any_sync(0xffffffffu, grow)) {
        const float corr = grow ? exp2f((m - mn) * sc) : 1.f;        // also of a row without a key so far: its sums are zero
        if (grow) m = mn;
        l *= corr;
        if (j > 0) {
          wide_wait(&pv_done[(j - 1) & 1], ((j - 1) >> 1) & 1, failed, a.wait_limit);
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            uint32_t o[16];
            tmem_ld_32x16(tO + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
            tmem_st_32x16(tO + c * 16, o);
          }
        }
      }
      const float use = m == -INFINITY ? 0.f : m;                    // nothing visible yet: keep the arithmetic finite
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        s[i] = exp2f((s[i] - use) * sc) * kUnit;
        sum += s[i];
      }
      l += sum;
      if (j >= 2) {
        wide_wait(&pv_done[b], ((j >> 1) - 1) & 1, failed, a.wait_limit);
        tc_fence_after();
      }
      const uint32_t tP = tmem_P + b * 96 + half * 16 + lanes;
      {
        float x[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = s[i];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          uint32_t part[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            part[i] = pack2<kBf16>(x[2 * i], x[2 * i + 1]);
            const float2 h = unpack2<kBf16>(part[i]);
            x[2 * i] -= h.x;
            x[2 * i + 1] -= h.y;
          }
          tmem_st_32x16(tP + q * 32, part);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      wide_arrive(&p_ready[b]);
      if (odd) {                                                     // what was taken out of V, by hand: one half's keys, then the other's
        wide_wait(&pv_done[b], (j >> 1) & 1, failed, a.wait_limit);
        tc_fence_after();
        for (int turn = 0; turn < 2; ++turn) {
          if (turn == half) {
            for (int c = 0; c < D / 16; ++c) {
              uint32_t o[16];
              tmem_ld_32x16(tmem_O + c * 16 + lanes, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const int key = kb + half * 32 + i;
                if (key >= min(vis, k1) || key < min_vis) continue;
                const int blk = key / a.block_size;
                const uint16_t* src = static_cast<const uint16_t*>(a.v_cache) +
                                      ((static_cast<int64_t>(bt[blk]) * a.block_size + (key - blk * a.block_size)) * a.ng + hk) * D + c * 16;
#pragma unroll
                for (int d = 0; d < 16; ++d) {
                  const uint16_t raw = src[d], e = kBf16 ? 0x7f80 : 0x7c00;
                  if ((raw & e) == e) o[d] = __float_as_uint(fmaf(s[i], unpack2<kBf16>(raw).x, __uint_as_float(o[d])));
                }
              }
              __syncwarp();
              tmem_st_32x16(tmem_O + c * 16 + lanes, o);
            }
            tmem_st_wait();
            tc_fence_before();
          }
          named_bar_sync(2, 256);
          tc_fence_after();
        }
      }
    }
    if (n_st > 0) {
      wide_wait(&pv_done[(n_st - 1) & 1], ((n_st - 1) >> 1) & 1, failed, a.wait_limit);
      tc_fence_after();
    }
    float* slot = s_ex + (n_st & 1) * (2 * L::kRows);
    slot[half * L::kRows + r] = l;
    named_bar_sync(4 + quad, 64);
    l = slot[r] + slot[L::kRows + r];
    if (p.splits == 1) {
      const float inv = l > 0.f ? 1.f / l : l;                       // 0 without keys; NaN stays NaN
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        uint32_t o[32];
        if (n_st > 0) {
          tmem_ld_32x32(tO + c * 32, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0u;
        }
        if (r < n_rows) {
          uint4* dst = reinterpret_cast<uint4*>(out_row(r) + half * (D / 2) + c * 32);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              w[i] = pack2<kBf16>(__uint_as_float(o[u * 8 + 2 * i]) * inv, __uint_as_float(o[u * 8 + 2 * i + 1]) * inv);
            dst[u] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    } else {
      // the cluster's partials, over the ring: every product has been made
      named_bar_sync(2, 256);
      float* part = reinterpret_cast<float*>(smem + L::kKOff) + r * D + half * (D / 2);
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        uint32_t o[32];
        if (n_st > 0) {
          tmem_ld_32x32(tO + c * 32, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) reinterpret_cast<uint4*>(part + c * 32)[i] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
      }
      if (half == 0) {
        reinterpret_cast<float*>(smem + L::kStatOff)[r] = m;
        reinterpret_cast<float*>(smem + L::kStatOff)[L::kRows + r] = l;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*failed) {                                                     // every wait is over, so all threads read the same
    volatile int never = 0;
    if (threadIdx.x == 0) atomicExch(&g_paged_error, 1);
    if (warp == 0) {
      for (int i = max(0, n_loaded - kS); i < n_loaded; ++i) {
        wide_wait(&k_full[i % kS], (i / kS) & 1, &never);
        wide_wait(&v_full[i % kS], (i / kS) & 1, &never);
      }
    } else if (warp == 1 || warp == 2) {
      if (elect_one()) umma_commit(drained);
      wide_wait(drained, 0, &never);
    } else if (warp >= 4) {
      const float nan = __int_as_float(0x7fffffff);
      for (int i = threadIdx.x - 128; i < n_rows * (D / 8); i += 256)
        *reinterpret_cast<uint4*>(out_row(i / (D / 8)) + i % (D / 8) * 8) = make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
      if (threadIdx.x - 128 < L::kRows) {                            // for the cluster: a sum that is not a number
        reinterpret_cast<float*>(smem + L::kStatOff)[threadIdx.x - 128] = 0.f;
        reinterpret_cast<float*>(smem + L::kStatOff)[L::kRows + threadIdx.x - 128] = nan;
      }
    }
    __syncthreads();
  }
  if (warp == 2) tmem_dealloc<512>(tmem);
  if (p.splits == 1) return;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const float* part = reinterpret_cast<const float*>(smem + L::kKOff);
  const float* s_m = reinterpret_cast<const float*>(smem + L::kStatOff);
  const float* s_l = s_m + L::kRows;
  merge_cluster<D, kBf16>(p, rank * kWideThreads + threadIdx.x, kWideThreads, n_rows, part, s_m, s_l, out_row);
  cluster.sync();                                                    // no CTA leaves while another reads its partials
}

// new keys and values [T, ng, d] (any token and head strides) into their cache rows, 16 bytes per thread
// kCount: counters of the decode kernel are set to zero too.  Kernels of their own: with the few instructions more, steps that need no counters took 1.2 to
// 1.8 us longer (81 requests of up to 182 keys x 12 heads of 128: 21.7 -> 23.5)
template <bool kCount>
__global__ void __launch_bounds__(256) paged_write_kernel(const uint4* __restrict__ k, const uint4* __restrict__ v, uint4* __restrict__ kc,
                                                          uint4* __restrict__ vc, const int64_t* __restrict__ slots, int n_tok, int ng, int chunks,
                                                          int64_t k_st, int64_t k_sh, int64_t v_st, int64_t v_sh, int* __restrict__ arrived,
                                                          int64_t n_arrived) {
  pdl_allow_next();
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x, row = static_cast<int64_t>(ng) * chunks;
  if (kCount && idx < n_arrived) arrived[idx] = 0;
  if (idx >= n_tok * row) return;
  const int64_t t = idx / row;
  const int c = static_cast<int>(idx % row), h = c / chunks, u = c % chunks;
  const int64_t dst = slots[t] * row + c;
  kc[dst] = k[t * k_st + h * k_sh + u];
  vc[dst] = v[t * v_st + h * v_sh + u];
}

// in the stream's order, but for what the kernels' own waits leave open (pdl_await_previous)
struct Launch {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2]{};
  Launch(unsigned ctas, int threads, int smem, int cluster, cudaStream_t s) {
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
  }
  Launch(const Launch&) = delete;
};
template <typename K, typename... Args>
int launch(K kern, unsigned ctas, int threads, int smem, int cluster, cudaStream_t s, const Args&... args) {
  const Launch l(ctas, threads, smem, cluster, s);
  const cudaError_t e = cudaLaunchKernelEx(&l.cfg, kern, args...);
  if (e != cudaSuccess) { g_paged_err = std::string("paged attention launch: ") + cudaGetErrorString(e); return -11; }
  return 0;
}

template <int D, bool kBf16>
int launch_chunks(const PagedParams& p, cudaStream_t s) {
  auto kern = paged_chunk_kernel<D, kBf16>;
  static const cudaError_t ready = [&] {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<D>::kTotal);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  }();
  if (ready != cudaSuccess) { g_paged_err = std::string("paged attention: ") + cudaGetErrorString(ready); return -10; }
  const int64_t ctas = static_cast<int64_t>(p.n_tiles) * p.a.ng * p.splits;
  if (ctas > 0x7fffffff) { g_paged_err = "paged attention: too many tiles"; return -12; }
  return launch(kern, static_cast<unsigned>(ctas), 128, Smem<D>::kTotal, p.splits, s, p);
}

// the pages of a cache as boxes of up to 64 slots x 64 values of one head
bool page_map(CUtensorMap* map, const void* cache, const PagedAttnArgs& a) {
  typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const EncodeFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess;
    return ok ? reinterpret_cast<EncodeFn>(ptr) : nullptr;
  }();
  if (fn == nullptr) return false;
  ensure_cuda_context();
  const cuuint64_t d = a.head_dim, ng = a.ng;
  const cuuint64_t dims[3] = {d, ng, static_cast<cuuint64_t>(a.n_slots)}, strides[2] = {d * 2, d * ng * 2};
  const cuuint32_t box[3] = {64, 1, static_cast<cuuint32_t>(a.block_size < kStageKeys ? a.block_size : kStageKeys)}, step[3] = {1, 1, 1};
  return fn(map, a.is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(cache), dims, strides, box, step,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D, bool kBf16>
cudaError_t wide_ready() {
  static const cudaError_t ready = [] {
    auto kern = paged_wide_kernel<D, kBf16>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WideSmem<D>::kTotal);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  }();
  return ready;
}

// how many clusters of 2^log CTAs of this kernel the device has room for at once (0: none, or it cannot say); asked once a device
template <int D, bool kBf16>
int wide_clusters(int log) {
  constexpr int kDevices = 16;
  static std::atomic<int> known[kDevices][5];                        // + 1
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 0;
  if (const int v = known[dev][log].load(std::memory_order_relaxed); v > 0) return v - 1;
  if (wide_ready<D, kBf16>() != cudaSuccess) return 0;
  const Launch l(1u << log, kWideThreads, WideSmem<D>::kTotal, 1 << log, nullptr);
  if (cudaOccupancyMaxActiveClusters(&n, paged_wide_kernel<D, kBf16>, &l.cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  known[dev][log].store(n + 1, std::memory_order_relaxed);
  return n;
}
int wide_clusters(const PagedAttnArgs& a, int log) {
  return a.head_dim == 128 ? (a.is_bf16 ? wide_clusters<128, true>(log) : wide_clusters<128, false>(log))
                           : (a.is_bf16 ? wide_clusters<64, true>(log) : wide_clusters<64, false>(log));
}

// A tile's key ranges are the CTAs of a cluster, which start together or not at all.  One CTA takes an SM, and a cluster's SMs lie side by side: of the 148, ones of 16
// find room for fewer than nine.  So there are only as many ranges as let all clusters run at once.
int wide_ranges(const PagedAttnArgs& a) {
  const int64_t clusters = static_cast<int64_t>(a.wide_tiles) * a.ng;
  int log = 0;
  while (log < 4 && (2 << log) <= a.wide_splits) ++log;
  while (log > 0 && wide_clusters(a, log) < clusters) --log;
  return 1 << log;
}

template <int D, bool kBf16>
int launch_wide(const PagedParams& p, const CUtensorMap& mk, const CUtensorMap& mv, cudaStream_t s) {
  if (const cudaError_t e = wide_ready<D, kBf16>(); e != cudaSuccess) { g_paged_err = std::string("paged attention: ") + cudaGetErrorString(e); return -10; }
  const int64_t ctas = static_cast<int64_t>(p.n_tiles) * p.a.ng * p.splits;
  if (ctas > 0x7fffffff) { g_paged_err = "paged attention: too many tiles"; return -12; }
  return launch(paged_wide_kernel<D, kBf16>, static_cast<unsigned>(ctas), kWideThreads, WideSmem<D>::kTotal, p.splits, s, mk, mv, p);
}

template <int D, bool kBf16>
int launch_decode(const PagedParams& p, cudaStream_t s) {
  auto cut = paged_decode_kernel<D, kBf16, true>, whole = paged_decode_kernel<D, kBf16, false>;
  static const cudaError_t ready = [&] {
    const cudaError_t e = cudaFuncSetAttribute(cut, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<D>::kTotal);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(whole, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<D>::kTotal);
  }();
  if (ready != cudaSuccess) { g_paged_err = std::string("paged attention: ") + cudaGetErrorString(ready); return -10; }
  // the line of stages is counted in 32 bits
  if (static_cast<int64_t>(p.n_tiles) * p.a.ng * ((static_cast<int64_t>(p.a.max_blocks) * p.a.block_size + kStageKeys - 1) / kStageKeys + 1) > 0x7fffffff) {
    g_paged_err = "paged attention: too many requests";
    return -12;
  }
  const unsigned items = static_cast<unsigned>(p.n_tiles * p.a.ng);
  return launch(p.splits > 0 ? cut : whole, p.splits > 0 ? p.splits : items, 128, Smem<D>::kTotal, 1, s, p);
}

template <int D, bool kBf16>
int launch_rows(const PagedParams& p, cudaStream_t s) {
  const unsigned items = static_cast<unsigned>(p.n_tiles * p.a.ng);
  if (p.a.group == 1) return launch(paged_rows_kernel<D, 1, kBf16>, items, 128, 0, 1, s, p);
  if (p.a.group == 2) return launch(paged_rows_kernel<D, 2, kBf16>, items, 128, 0, 1, s, p);
  return launch(paged_rows_kernel<D, 4, kBf16>, items, 128, 0, 1, s, p);
}

int log2_exact(int v) {
  for (int i = 0; i < 31; ++i)
    if (v == 1 << i) return i;
  return -1;
}

int64_t decode_items(const PagedAttnArgs& a) { return static_cast<int64_t>(a.cu != nullptr ? a.n_seqs : a.n_tokens) * a.ng; }
// keys of the longest context, as far as the caller knows
int64_t decode_keys(const PagedAttnArgs& a) {
  const int64_t all = static_cast<int64_t>(a.max_blocks) * a.block_size;
  return a.decode_len > 0 && a.decode_len < all ? a.decode_len : all;
}

// the line of decode stages is cut for three CTAs per SM, but for no more than there can be pairs of stages.  Where that gains little the items stay whole (0):
// putting parts together costs as much as the imbalance that it removes.  A stage of heads of 64 takes half as long: us, whole / cut, 10 requests of up to 824 keys x 12
// beside chunks 21.9 / 29.3, 1 of 522 x 8 10.3 / 12.4.  Heads of 128, geometric means of cut / whole over 513 drawn steps: alone, up to 24 (request, head) pairs of 5
// stages 1.20, of 8 0.87, of 10 0.74; 100 to 300 of 9 1.00, of 12 0.92, of 14 0.85; above 444 of 9 to 13 1.06, of 16 0.93: what counts is by how much the longest
// exceeds a CTA's share.  Beside chunks, behind whose CTAs the many short parts start: up to 96 of 9 0.92, of 12 0.79; 100 to 300 of 9 1.13, of 13 1.06, of 14 0.97 (up to 1.24), of 15 0.88
int decode_ctas(const PagedAttnArgs& a) {
  const int64_t items = decode_items(a), longest = (decode_keys(a) + kStageKeys - 1) / kStageKeys;
  const int64_t n = items * longest / 2, ctas = n < 1 ? 1 : (n > kDecodeCtas ? kDecodeCtas : n);
  bool whole;
  if (a.head_dim == 64) whole = longest <= (items <= kDecodeCtas ? 16 : 8);
  else if (a.beside_chunks) whole = longest <= (items <= 96 ? 8 : 14);
  else {
    const double mean = a.decode_mean > 0 ? a.decode_mean / static_cast<double>(kStageKeys) : static_cast<double>(longest), share = items * mean / ctas;
    whole = (longest <= 8 && items > 16) || longest - (share > 1. ? share : 1.) < 6.;
  }
  return whole ? 0 : static_cast<int>(ctas);
}

// a workspace holds the CTAs' partials and, behind them, a counter for each (request, KV head)
int64_t decode_parts(const PagedAttnArgs& a) { return static_cast<int64_t>(decode_ctas(a)) * 2 * 16 * (a.head_dim + 2); }
int* arrived_in(const PagedAttnArgs& a, float* ws) { return reinterpret_cast<int*>(ws + decode_parts(a)); }

}  // namespace

const char* paged_attention_last_error() { return g_paged_err.c_str(); }

// Rows of a tile that stand empty (all but `group` of 16) against keys to share: from how many (request, KV head) pairs on, and up to which
// context, a CTA per pair is the better one.  us, tiles / rows: 256 requests of 100 keys x 32 heads of 128, group 1 165 / 88, group 2 167 / 133;
// of 600 keys 581 / 422 and 596 / 703; 512 of 600 x 32 heads of 64 947 / 519 and 949 / 676; 512 of 16 keys x 8 heads of 128, group 4 60 / 41,
// of 63 keys 70 / 76; 64 of 300 x 8 heads of 128, group 1 35 / 45: there all pairs run at once.  Lengths that differ leave the rows' CTAs
// uneven, which the tiles' line is not: 96 requests of 64 to 1000 keys x 12 heads of 128 96 / 111, of 64 70 / 61.
bool paged_decode_by_rows(const PagedAttnArgs& a) {
  if (a.cu != nullptr && !a.decode_single) return false;             // tokens of one request would each read all its keys
  const int64_t items = decode_items(a), keys = decode_keys(a);
  if (items <= kDecodeCtas) return false;
  const bool many = items > 2 * kDecodeCtas, narrow = a.head_dim == 64;
  if (a.group == 1) {
    if (a.decode_mean > 0 && 2 * keys > 3 * a.decode_mean && keys > (narrow ? 1024 : 256)) return false;
    return keys <= (items >= 4096 ? 2048 : many ? 1024 : narrow ? 640 : 160);
  }
  if (a.group == 2) return keys <= (many ? (narrow ? 640 : 160) : 32);
  return a.group == 4 && many && keys <= 32;
}

// Whether chunks go by tiles of 128 rows on tcgen05: where a stage of 64 keys is whole pages, or a piece of one, on 8-row boundaries of the swizzle
bool paged_wide_tiles(const PagedAttnArgs& a) {
  return a.wide_tiles > 0 && a.n_slots > 0 && a.n_slots <= 0x7fffffff && a.block_size % 8 == 0 &&
         (kStageKeys % a.block_size == 0 || a.block_size % kStageKeys == 0);
}

namespace {
bool wide_maps(const PagedAttnArgs& a, CUtensorMap* mk, CUtensorMap* mv) { return paged_wide_tiles(a) && page_map(mk, a.k_cache, a) && page_map(mv, a.v_cache, a); }
}  // namespace

int paged_chunk_rows(const PagedAttnArgs& a) {
  CUtensorMap mk, mv;
  return wide_maps(a, &mk, &mv) ? 128 : 64;
}

int paged_wide_ranges(const PagedAttnArgs& a, int* resident) {
  const int ranges = wide_ranges(a);
  int log = 0;
  while ((1 << log) < ranges) ++log;
  *resident = wide_clusters(a, log);
  return ranges;
}

int paged_status(bool clear) {
  int v = 0;
  const int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_paged_error, sizeof(int)) != cudaSuccess) return -1;
  if (clear && v != 0 && cudaMemcpyToSymbol(g_paged_error, &zero, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

bool paged_attention_supported(int head_dim, int group) {
  return (head_dim == 64 || head_dim == 128) && (group == 1 || group == 2 || group == 4 || group == 8);
}

int paged_decode_cut(const PagedAttnArgs& a) { return paged_decode_by_rows(a) ? 0 : decode_ctas(a); }

int64_t paged_decode_workspace(const PagedAttnArgs& a) {
  if (paged_decode_by_rows(a)) return 0;
  const int64_t parts = decode_parts(a);
  return parts > 0 ? parts + decode_items(a) : 0;
}

// zeroes the decode kernel's counters (`ws`, where that call will have a workspace) too
void paged_write(const PagedWriteArgs& w, const PagedAttnArgs& a, float* ws, cudaStream_t s) {
  const int chunks = w.head_dim / 8;
  const int64_t n = static_cast<int64_t>(w.n_tokens) * w.ng * chunks;
  if (n == 0) return;
  const int64_t n_arrived = ws != nullptr ? decode_items(a) : 0;
  auto kern = n_arrived > 0 ? paged_write_kernel<true> : paged_write_kernel<false>;
  kern<<<static_cast<unsigned>(((n > n_arrived ? n : n_arrived) + 255) / 256), 256, 0, s>>>(
      static_cast<const uint4*>(w.k), static_cast<const uint4*>(w.v), static_cast<uint4*>(w.k_cache), static_cast<uint4*>(w.v_cache), w.slots,
      w.n_tokens, w.ng, chunks, w.k_st / 8, w.k_sh / 8, w.v_st / 8, w.v_sh / 8, n_arrived > 0 ? arrived_in(a, ws) : nullptr, n_arrived);
}

// with cu: chunk_tiles tiles of 64 rows over the requests with more than 16, in chunk_splits key ranges; decode: whether there are others
// `written`: paged_write went before it with the same workspace
int paged_attention(const PagedAttnArgs& a, bool decode, int chunk_tiles, int chunk_splits, float* ws, bool written, cudaStream_t s) {
  PagedParams p{};
  p.a = a;
  p.a.wait_limit = a.wait_limit < 0 ? kWideTries : a.wait_limit;
  p.row_scale = a.scale_log2;
  p.a.scale_log2 = a.scale_log2 == 0.f ? 1.f : fabsf(a.scale_log2);
  p.q_keep = a.scale_log2 == 0.f ? 0u : 0xffffffffu;
  p.q_sign = a.scale_log2 < 0.f ? 0x80008000u : 0u;
  p.group_shift = log2_exact(a.group);
  p.bs_shift = log2_exact(a.block_size);
  // Counters that no write kernel of this call has zeroed are zeroed in front of all launches: the first one waits for that, and the decode kernel
  // beside chunks, which counts without a wait of its own, starts when all of theirs have
  const int decode_cut = decode && !paged_decode_by_rows(a) ? decode_ctas(a) : 0;
  if (decode_cut > 0 && !written) {
    const cudaError_t e = cudaMemsetAsync(arrived_in(a, ws), 0, sizeof(int) * static_cast<size_t>(decode_items(a)), s);
    if (e != cudaSuccess) { g_paged_err = std::string("paged attention: ") + cudaGetErrorString(e); return -13; }
  }
  CUtensorMap mk, mv;
  if (a.cu != nullptr && chunk_tiles > 0 && wide_maps(a, &mk, &mv)) {
    p.n_tiles = a.wide_tiles;
    p.splits = wide_ranges(a);
    const int rc = a.head_dim == 128 ? (a.is_bf16 ? launch_wide<128, true>(p, mk, mv, s) : launch_wide<128, false>(p, mk, mv, s))
                                     : (a.is_bf16 ? launch_wide<64, true>(p, mk, mv, s) : launch_wide<64, false>(p, mk, mv, s));
    if (rc != 0) return rc;
  } else if (a.cu != nullptr && chunk_tiles > 0) {
    p.n_tiles = chunk_tiles;
    p.splits = 1;
    while (2 * p.splits <= chunk_splits && p.splits < 16) p.splits *= 2;
    const int rc = a.head_dim == 128 ? (a.is_bf16 ? launch_chunks<128, true>(p, s) : launch_chunks<128, false>(p, s))
                                     : (a.is_bf16 ? launch_chunks<64, true>(p, s) : launch_chunks<64, false>(p, s));
    if (rc != 0) return rc;
  }
  if (a.cu != nullptr && !decode) return 0;                          // every request is a chunk
  p.n_tiles = a.cu != nullptr ? a.n_seqs : a.n_tokens;
  p.beside_chunks = a.beside_chunks;
  if (paged_decode_by_rows(a)) {
    if (decode_items(a) > 0x7fffffff) { g_paged_err = "paged attention: too many requests"; return -12; }
    return a.head_dim == 128 ? (a.is_bf16 ? launch_rows<128, true>(p, s) : launch_rows<128, false>(p, s))
                             : (a.is_bf16 ? launch_rows<64, true>(p, s) : launch_rows<64, false>(p, s));
  }
  p.splits = decode_cut;
  p.behind_write = written && !p.beside_chunks;
  p.ws = ws;
  if (p.splits > 0) p.arrived = arrived_in(a, ws);
  return a.head_dim == 128 ? (a.is_bf16 ? launch_decode<128, true>(p, s) : launch_decode<128, false>(p, s))
                           : (a.is_bf16 ? launch_decode<64, true>(p, s) : launch_decode<64, false>(p, s));
}

}  // namespace b200
