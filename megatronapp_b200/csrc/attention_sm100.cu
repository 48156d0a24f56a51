// Flash attention for sm_100a: tcgen05 MMAs with S / O accumulators in TMEM, TMA-fed K/V ring,
// two 128-row query tiles per CTA processed ping-pong by two softmax warpgroups.
//
// Forward  (attn_fwd_kernel):  S = Q K^T -> online softmax (exp2 domain, lazy rescale) ->
//                              P (16-bit, TMEM columns of its own) -> O += P V (O stays in TMEM).
// Backward (one launch of two parts, deterministic, no atomics):
//   bwd_part<dK, dV> : CTA per 128-key block, loops over 64-query blocks
//                             S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q
//   bwd_part<dQ>     : CTA per 128-query block, loops over 64-key blocks
//                             S = Q K^T, dP = dO V^T, dQ += dS K
// Operands are strided [b, h, s, d] views (last dim contiguous) so the Megatron [s, b, h, d]
// activations are consumed in place (4-D tensor maps); outputs are written in [s, b, h, d].
//
// Replaces reference dot_product_attention.py:106-208 (baddbmm -> fused softmax -> bmm) and the
// TE/cuDNN path extensions/transformer_engine.py:609-.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <mutex>
#include <string>
#include <type_traits>

#include "b200_api.h"
#include "common.cuh"

namespace b200 {
namespace {

constexpr int kBlockQ = 128;    // query rows per tile
constexpr int kBlockKV = 128;   // keys per block (forward)
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.0f;  // lazy O rescale: only when the row max grows by > 2^8

__device__ __forceinline__ void tma_load_4d(const void* tmap, uint64_t* bar, void* smem_dst, int32_t c0,
                                            int32_t c1, int32_t c2, int32_t c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <bool kBf16>
__device__ __forceinline__ uint32_t pack16(float lo, float hi) {
  if constexpr (kBf16) return pack_bf16x2(lo, hi);
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
// two fp32 lanes of one 64-bit register: the packed forms round like the scalar ones at half the issue slots
__device__ __forceinline__ uint64_t f2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void un2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// tcgen05.mma takes its descriptors from uniform registers.  A loop run by one lane of a diverged warp moves each of them over before
// every instruction (70 cycles an MMA measured, more than the 32 to 64 that these tiles take to execute); the issuing warp therefore runs
// its loop converged, on descriptors that advance by constants, and one elected lane issues.
__device__ __forceinline__ uint64_t desc_at(uint64_t base, uint32_t bytes) { return base + (bytes >> 4); }

// A wait that runs out is noted in `failed`.  At its end the CTA then leaves g_attn_error for attn_status, fills the rows that it owns with NaN
// and waits (always within kWaitLimit) for its own copies and MMAs in flight.
constexpr int kWaitLimit = 1 << 20;
__device__ int g_attn_error = 0;
// false: the wait ran out here, or another thread of the CTA gave up
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, volatile int* failed, int limit = kWaitLimit) {
  for (int i = 0; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255) == 255 && *failed) return false;
  }
  *failed = 1;
  return false;
}
// the same for a whole warp, which votes after every try and so stays converged: 65 cycles for a barrier that is ready (123 where the lanes
// loop on their own and vote at the end)
__device__ __forceinline__ bool wait_bar_warp(uint64_t* bar, uint32_t parity, volatile int* failed, int limit = kWaitLimit) {
  for (int i = 0; i < limit; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((i & 255) == 255 && __any_sync(0xffffffffu, *failed != 0)) return false;
  }
  *failed = 1;
  return false;
}

// A look ahead at a barrier, whose answer is wanted some instructions later
__device__ __forceinline__ uint32_t mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// One arrival for a warp: 32 of them on one word are carried out one after another
__device__ __forceinline__ void warp_arrive(uint64_t* bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

// One warpgroup copies and issues, four do the softmax arithmetic.  A CTA of 640 threads starts with 96 registers each; the math
// warpgroups take 104 and leave 64 to the first.
constexpr int kThreads = 640, kMathRegs = 104, kIssueRegs = 64;
static_assert(512 * kMathRegs + 128 * kIssueRegs <= kThreads * 96, "the shares come out of what the CTA was launched with");
// The forward's two math warpgroups have a thread to a row of scores: 384 threads start with 168 registers each.
constexpr int kFwdThreads = 384, kFwdMathRegs = 208, kFwdIssueRegs = 80;
static_assert(256 * kFwdMathRegs + 128 * kFwdIssueRegs <= kFwdThreads * 168, "the shares come out of what the CTA was launched with");
template <int N> __device__ __forceinline__ void regs_take() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_give() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// 32 accumulator columns of this thread's row, scaled, as 64 bytes of 16-bit results
template <bool kBf16>
__device__ __forceinline__ void store_row32(uint8_t* dst, const uint32_t (&v)[32], float mul) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    uint4 w;
    w.x = pack16<kBf16>(__uint_as_float(v[u * 8 + 0]) * mul, __uint_as_float(v[u * 8 + 1]) * mul);
    w.y = pack16<kBf16>(__uint_as_float(v[u * 8 + 2]) * mul, __uint_as_float(v[u * 8 + 3]) * mul);
    w.z = pack16<kBf16>(__uint_as_float(v[u * 8 + 4]) * mul, __uint_as_float(v[u * 8 + 5]) * mul);
    w.w = pack16<kBf16>(__uint_as_float(v[u * 8 + 6]) * mul, __uint_as_float(v[u * 8 + 7]) * mul);
    *reinterpret_cast<uint4*>(dst + u * 16) = w;
  }
}
// after a wait that ran out, by the math warps: NaN (in either type) in `rows` rows of D columns
template <int D, int kN = kThreads>
__device__ __forceinline__ void fill_nan(void* out, int64_t base, int64_t stride, int rows) {
  constexpr int kChunks = D / 8;
  for (int i = threadIdx.x - 128; i < rows * kChunks; i += kN - 128)
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(out) + base + i / kChunks * stride + i % kChunks * 8) =
        make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
}
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

struct FwdParams {
  float* lse;            // [b, h, sq]
  void* o;               // [sq, b, h, d] strides below
  int64_t o_sb, o_sh, o_ss;
  int b, hq, hkv, sq, sk;
  float scale_log2;      // softmax scale * log2(e)
  int causal;
  int wait_limit;        // tries of a wait before it gives up
};

template <int D>
struct FwdSmem {
  static constexpr int kDC = D / 64;                    // 64-element (128 B) chunks along d
  static constexpr int kTile = kBlockQ * 128 * kDC;     // bytes of a [128 x D] 16-bit tile
  static constexpr int kStages = 2;
  static constexpr int kQOff = 0;
  static constexpr int kKOff = kQOff + 2 * kTile;
  static constexpr int kVOff = kKOff + kStages * kTile;
  static constexpr int kBarOff = kVOff + kStages * kTile;
  static constexpr int kTotal = kBarOff + 256 + 1024;   // + barriers + alignment slack
};

// ------------------------------------------------------------------------------------ forward
// P (16-bit) goes to TMEM columns of its own and feeds the PV product as the TMEM A operand.  Two query tiles alternate between the tensor
// core (1024 cycles a key block at D = 128) and the softmax (1024 cycles of exponentials at one block's rate).  A thread has a row of 128 scores, read once
// into registers: with 208 of them its exponentials follow one another at the unit's rate for two warps, where two threads to a row with 104 each took twice as long
// for theirs and had maxima and sums to exchange (cycles from scores to weights, 2900 there and 2300 here).  S's columns are free again as soon as they are in
// registers, so the next S (the other tile's where there is one buffer, this tile's where there are two) is made under this one's exponentials.
// A look at a barrier takes 130 cycles with the steps around it even if it is open, so the answer is fetched ahead of its use where it is most likely yes
// (D = 64: the next S, the product that frees P's columns; at D = 128 there the scores of the other tile come first, and it cost 1 to 10 %).
// Two warps issue: a wait that is already over costs 65 to 120 cycles, the tensor core's queue holds four
// MMAs (256 cycles), and one warp that goes through all waits in turn leaves it empty (174 us where two take 139).
// us, two threads to a row / one: 32 heads x 8192 x 64 causal 404 / 367, 32 x 3 x 1337 x 64 65 / 61, 32 / 8 x 4096 x 128 130 / 126, x 512 16.5 / 14.5.
// CTAs that go on to further blocks of the grid (clusterlaunchcontrol), and tiles that take turns at the exponentials, gave nothing or cost time.
template <int D, bool kBf16>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const FwdParams p) {
  using L = FwdSmem<D>;
  constexpr int kS = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + L::kQOff;
  uint8_t* sK = smem + L::kKOff;
  uint8_t* sV = smem + L::kVOff;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* q_full = bars;            // 1
  uint64_t* k_full = bars + 1;        // 2
  uint64_t* k_empty = bars + 3;       // 2
  uint64_t* v_full = bars + 5;        // 2
  uint64_t* v_empty = bars + 7;       // 2
  uint64_t* s_full = bars + 9;        // 2 (per q tile)
  uint64_t* s_read = bars + 11;       // 2 (per q tile): S is in registers
  uint64_t* p_ready = bars + 13;      // 2 (per q tile)
  uint64_t* pv_done = bars + 15;      // 2 (per q tile): P's columns are free and O is up to date
  uint64_t* drained = bars + 17;      // 1, after a wait that ran out
  uint64_t* s_issued = bars + 18;     // 4: the CTA's S number i (of both tiles) is in the tensor core's queue, at i % 4
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 22);
  volatile int* failed = reinterpret_cast<volatile int*>(bars + 23);

  const int warp_idx = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // known to be uniform: see desc_at
  const int lane = threadIdx.x & 31;
  // (query block, head, batch) from one grid dimension, the longest rows of every head before any shorter ones
  const int n_hb = p.hq * p.b, hb = static_cast<int>(blockIdx.x) % n_hb;
  const int qblk2 = static_cast<int>(gridDim.x) / n_hb - 1 - static_cast<int>(blockIdx.x) / n_hb;
  const int h = hb % p.hq, bi = hb / p.hq;
  const int hk = h / (p.hq / p.hkv);
  const int q0_0 = qblk2 * 2 * kBlockQ, q0_1 = q0_0 + kBlockQ;
  const int nkv_all = (p.sk + kBlockKV - 1) / kBlockKV;
  auto blocks_for = [&](int q0) {
    if (q0 >= p.sq) return 0;
    return p.causal ? min(nkv_all, q0 / kBlockKV + 1) : nkv_all;
  };
  const int nkv_0 = blocks_for(q0_0), nkv_1 = blocks_for(q0_1);
  const int nmax = max(nkv_0, nkv_1);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&s_read[i], 4);
      mbar_init(&p_ready[i], 4); mbar_init(&pv_done[i], 1);
    }
    mbar_init(drained, 2);
    for (int i = 0; i < 4; ++i) mbar_init(&s_issued[i], 1);
    *failed = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v);
  }
  if (warp_idx == 2) tmem_alloc<512>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  int n_loaded = 0;                           // blocks whose copies this thread (lane 0 of warps 0 and 3) has started
  const uint32_t tmem_O = tmem_base;                                 // O[t] at col t*D
  const uint32_t tmem_P = tmem_base + 2 * D;                         // P[t] at col 2*D + t*64
  const uint32_t tmem_S = tmem_base + 2 * D + 128;                   // S[t] at t*128 of the remaining 256, or one S for both in 128
  constexpr int kSBufs = D == 64 ? 2 : 1;
  static_assert(2 * D + 128 + kSBufs * 128 <= 512, "TMEM columns");

  if (warp_idx < 4) {
    regs_give<kFwdIssueRegs>();
    if (warp_idx == 0 && lane == 0) {
      // ============================================================ TMA producer
      const int ntiles = (nkv_1 > 0) ? 2 : 1;
      mbar_arrive_expect_tx(q_full, ntiles * L::kTile);
      for (int t = 0; t < ntiles; ++t)
        for (int c = 0; c < L::kDC; ++c)
          tma_load_4d(&tmap_q, q_full, sQ + t * L::kTile + c * (kBlockQ * 128), c * 64, h, bi, t == 0 ? q0_0 : q0_1);
      for (; n_loaded < nmax; ++n_loaded) {
        const int st = n_loaded % kS;
        if (!wait_bar(&k_empty[st], ((n_loaded / kS) & 1) ^ 1, failed, p.wait_limit)) break;
        mbar_arrive_expect_tx(&k_full[st], L::kTile);
        for (int c = 0; c < L::kDC; ++c)
          tma_load_4d(&tmap_k, &k_full[st], sK + st * L::kTile + c * (kBlockKV * 128), c * 64, hk, bi, n_loaded * kBlockKV);
      }
    } else if (warp_idx == 3 && lane == 0) {
      // K runs up to two blocks ahead of V: a producer each
      for (; n_loaded < nmax; ++n_loaded) {
        const int st = n_loaded % kS;
        if (!wait_bar(&v_empty[st], ((n_loaded / kS) & 1) ^ 1, failed, p.wait_limit)) break;
        mbar_arrive_expect_tx(&v_full[st], L::kTile);
        for (int c = 0; c < L::kDC; ++c)
          tma_load_4d(&tmap_v, &v_full[st], sV + st * L::kTile + c * (kBlockKV * 128), c * 64, hk, bi, n_loaded * kBlockKV);
      }
    } else if (warp_idx == 1) {
      // ============================================================ issuer of S = Q K^T
      constexpr uint32_t idesc_s = make_idesc_f16(kBf16, kBlockQ, kBlockKV, false, false);
      const uint64_t q_desc = make_smem_desc_sw128(smem_u32(sQ), 1024, 0), k_desc = make_smem_desc_sw128(smem_u32(sK), 1024, 0);
      bool ok = nmax > 0 && wait_bar_warp(q_full, 0, failed, p.wait_limit);
      int item = 0;
      for (int j = 0; j < nmax && ok; ++j) {
        const int st = j % kS;
        ok = wait_bar_warp(&k_full[st], (j / kS) & 1, failed, p.wait_limit);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (j >= (t == 0 ? nkv_0 : nkv_1) || !ok) continue;
          // the S before it in its buffer is in registers: this tile's where each has its own, else the other's, if that has such a block
          const bool other = kSBufs == 1 && (t == 1 ? j < nkv_0 : j <= nkv_1);
          const int rt = other ? 1 - t : t, rj = other && t == 1 ? j : j - 1;
          ok = rj < 0 || wait_bar_warp(&s_read[rt], rj & 1, failed, p.wait_limit);
          if (!ok) continue;
          tc_fence_after();
          const uint64_t a0 = desc_at(q_desc, t * L::kTile), b0 = desc_at(k_desc, st * L::kTile);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < D / 16; ++k) {
              const uint32_t off = (k >> 2) * (kBlockQ * 128) + (k & 3) * 32;
              umma_f16_ss(tmem_S + (kSBufs == 2 ? t * 128 : 0), desc_at(a0, off), desc_at(b0, off), idesc_s, k != 0 ? 1u : 0u);
            }
            umma_commit(&s_full[t]);
            if (t == 1 || j >= nkv_1) umma_commit(&k_empty[st]);
            if (kSBufs == 1) mbar_arrive(&s_issued[item & 3]);
          }
          ++item;
        }
      }
    } else if (warp_idx == 2) {
      // ============================================================ issuer of O += P V
      // a warp of its own: a wait and the steps around it take a few hundred cycles beside the math, and the tensor core's queue is short
      constexpr uint32_t idesc_o = make_idesc_f16(kBf16, kBlockQ, D, false, true);
      // V is MN-major for its product (N = d contiguous): 16 key rows per k-step, LBO = next 64-wide d chunk
      const uint64_t v_desc = make_smem_desc_sw128(smem_u32(sV), 1024, kBlockKV * 128);
      bool ok = true;
      // With one S buffer its next S is what everything waits for: 512 cycles of MMAs, and as long again for the steps from S to registers to
      // the next S.  A product goes into that gap, behind the S two blocks on, and never beside one.
      const int n_items = nkv_0 + nkv_1;
      int item = 2;
      for (int j = 0; j < nmax && ok; ++j) {
        const int st = j % kS;
        ok = wait_bar_warp(&v_full[st], (j / kS) & 1, failed, p.wait_limit);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (j >= (t == 0 ? nkv_0 : nkv_1)) continue;
          if (kSBufs == 1 && item < n_items) ok = ok && wait_bar_warp(&s_issued[item & 3], (item >> 2) & 1, failed, p.wait_limit);
          ++item;
          ok = ok && wait_bar_warp(&p_ready[t], j & 1, failed, p.wait_limit);
          if (!ok) continue;
          tc_fence_after();
          const uint64_t b0 = desc_at(v_desc, st * L::kTile);
          if (elect_one()) {
#pragma unroll
            for (int i = 0; i < kBlockKV / 16; ++i) {
              // A = P from TMEM: row = lane, 16 keys = 8 packed 32-bit columns per k-step.  The first 32 keys of both halves go before the other 32: fp32
              // sums depend on the order, and results stay what they are only while it does
              const int k = (i >> 2) * 2 + ((i >> 1) & 1) * 4 + (i & 1);
              umma_f16_ts(tmem_O + t * D, tmem_P + t * 64 + k * 8, desc_at(b0, k * 16 * 128), idesc_o, i != 0 || j != 0 ? 1u : 0u);
            }
            umma_commit(&pv_done[t]);
            if (t == 1 || j >= nkv_1) umma_commit(&v_empty[st]);
          }
        }
      }
    }
  } else {
    // ============================================================ softmax / correction / epilogue
    regs_take<kFwdMathRegs>();
    const int t = (warp_idx - 4) >> 2;            // q tile of this warpgroup
    const int quad = warp_idx & 3;                // TMEM lane quadrant
    const int r = quad * 32 + lane;               // row inside the tile
    const int q0 = t == 0 ? q0_0 : q0_1;
    const int qrow = q0 + r;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t tS = tmem_S + (kSBufs == 2 ? t * 128 : 0) + lane_addr;
    const uint32_t tP = tmem_P + t * 64 + lane_addr;
    const uint32_t tO = tmem_O + t * D + lane_addr;
    float m = -INFINITY;                          // running max (exp2 domain, already scaled)
    uint64_t l2[2] = {0, 0};                      // running sums of the even and odd columns of both halves
    const int n = t == 0 ? nkv_0 : nkv_1;
    const float sc = p.scale_log2;
    const uint64_t sc2 = f2(sc, sc);

    uint32_t next_there = 0;                      // the next block's scores have been made
    auto block = [&](int j, auto masked_tag) {
      constexpr bool kMasked = decltype(masked_tag)::value;
      const int limit = (kMasked ? min(p.sk, p.causal ? qrow + 1 : p.sk) : 0) - j * kBlockKV;   // valid: col < limit
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(tS + c * 32, v[c]);
      tmem_ld_wait();
      tc_fence_before();
      warp_arrive(&s_read[t]);
      float mx[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) mx[i] = -INFINITY;
      // the product before, after which P's columns are free: most likely over by now
      const uint32_t free_now = j == 0 ? 1u : kSBufs == 1 ? 0u : mbar_test(&pv_done[t], (j - 1) & 1);
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          if (kMasked && c * 32 + i >= limit) v[c][i] = 0xff800000u;   // -inf
          if (kMasked && c * 32 + i + 1 >= limit) v[c][i + 1] = 0xff800000u;
          mx[(i >> 1) & 7] = max3(mx[(i >> 1) & 7], __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
        }
      const float mine = max3(max3(mx[0], mx[1], mx[2]), max3(mx[3], mx[4], mx[5]), fmaxf(mx[6], mx[7]));
      float m_new = fmaxf(m, mine * sc);           // softmax scale is positive
      if (m_new == -INFINITY) m_new = 0.f;         // fully masked so far: keep everything finite
      const bool grow = (m_new - m) > kRescaleThreshold;   // also true on the first block (m = -inf)
      if (__any_sync(0xffffffffu, grow)) {
        const float m_cur = grow ? m_new : m;
        const float alpha = grow ? fast_exp2(m - m_cur) : 1.f;
        m = m_cur;
        l2[0] = mul2(l2[0], f2(alpha, alpha));
        l2[1] = mul2(l2[1], f2(alpha, alpha));
        if (j > 0) {
          wait_bar_warp(&pv_done[t], (j - 1) & 1, failed, p.wait_limit);
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < D / 16; ++c) {     // in small pieces: the scores are in registers
            uint32_t o[16];
            tmem_ld_32x16(tO + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x16(tO + c * 16, o);
          }
        }
      }
      const uint64_t nm2 = f2(-m, -m);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float p0, p1;
          un2(fma2(f2(__uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1])), sc2, nm2), p0, p1);
          p0 = fast_exp2(p0);
          p1 = fast_exp2(p1);
          l2[c >> 1] = add2(l2[c >> 1], f2(p0, p1));
          pk[i >> 1] = pack16<kBf16>(p0, p1);
        }
        if (c == 0 && j > 0) {                     // P's columns are free, after the product before
          if (!__all_sync(0xffffffffu, free_now)) wait_bar_warp(&pv_done[t], (j - 1) & 1, failed, p.wait_limit);
          tc_fence_after();
        }
        tmem_st_32x16(tP + c * 16, pk);
      }
      if (kSBufs == 2) next_there = mbar_test(&s_full[t], (j + 1) & 1);
      tmem_st_wait();
      tc_fence_before();
      warp_arrive(&p_ready[t]);
    };

    // a wait that runs out is noted, not acted on: every later wait ends at once
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      if (!__all_sync(0xffffffffu, next_there)) wait_bar_warp(&s_full[t], j & 1, failed, p.wait_limit);
      tc_fence_after();
      const int kbase = j * kBlockKV;
      // diagonal block of a causal tile, or the ragged tail of the key sequence
      const bool need_mask = (p.causal && kbase + kBlockKV - 1 > q0) || (kbase + kBlockKV > p.sk);
      if (need_mask) block(j, std::true_type{});
      else block(j, std::false_type{});
    }
    if (n > 0) {
      ok = wait_bar_warp(&pv_done[t], (n - 1) & 1, failed, p.wait_limit);
      tc_fence_after();
      float la, lb, lc, ld;
      un2(l2[0], la, lb);
      un2(l2[1], lc, ld);
      const float l = (la + lb) + (lc + ld);
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      const bool valid = qrow < p.sq && ok;
      uint8_t* orow = reinterpret_cast<uint8_t*>(p.o) +
                      (static_cast<int64_t>(qrow) * p.o_ss + static_cast<int64_t>(bi) * p.o_sb +
                       static_cast<int64_t>(h) * p.o_sh) * 2;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(tO + c * 32, v);
        tmem_ld_wait();
        if (valid) store_row32<kBf16>(orow + c * 64, v, inv_l);
      }
      if (valid)
        p.lse[(static_cast<int64_t>(bi) * p.hq + h) * p.sq + qrow] = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*failed) {                                  // every wait is over, so all threads read the same
    volatile int never = 0;
    if (threadIdx.x == 0) {
      atomicExch(&g_attn_error, 1);
      wait_bar(q_full, 0, &never);
      for (int i = max(0, n_loaded - kS); i < n_loaded; ++i) wait_bar(&k_full[i % kS], (i / kS) & 1, &never);
    } else if (warp_idx == 3 && lane == 0) {
      for (int i = max(0, n_loaded - kS); i < n_loaded; ++i) wait_bar(&v_full[i % kS], (i / kS) & 1, &never);
    } else if (warp_idx == 1 || warp_idx == 2) {
      if (elect_one()) umma_commit(drained);
      wait_bar_warp(drained, 0, &never);
    } else if (warp_idx >= 4) {
      const int rows = min(2 * kBlockQ, p.sq - q0_0);
      fill_nan<D, kFwdThreads>(p.o, static_cast<int64_t>(q0_0) * p.o_ss + static_cast<int64_t>(bi) * p.o_sb + static_cast<int64_t>(h) * p.o_sh, p.o_ss, rows);
      for (int i = threadIdx.x - 128; i < rows; i += kFwdThreads - 128)
        p.lse[(static_cast<int64_t>(bi) * p.hq + h) * p.sq + q0_0 + i] = __int_as_float(0x7fffffff);
    }
    __syncthreads();
  }
  if (warp_idx == 2) tmem_dealloc<512>(tmem_base);
}


// ------------------------------------------------------------------------------------ backward
// -delta[b, h, s] = -sum_d O * dO and -lse * log2e, the addends of the backward kernels' packed multiply-adds, in rows of whole blocks of 64: behind the last query
// stand zeros and -infinity, of which come weights of zero.  D / 8 lanes share a row
// (16 bytes each), a warp takes four groups of rows with all its loads in flight: 12.5 us for 32 heads x 4096 x 128 (a warp per row and
// 4 bytes a lane took 35).
template <int D>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const uint16_t* __restrict__ o, const uint16_t* __restrict__ d_o, float* __restrict__ ndelta, const float* __restrict__ lse,
                  float* __restrict__ nlse2, int h, int s, int pitch, int64_t o_sb, int64_t o_sh, int64_t o_ss, int64_t do_sb, int64_t do_sh, int64_t do_ss,
                  int is_bf16) {
  constexpr int kLanes = D / 8, kRows = 32 / kLanes, kSteps = 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, col = (lane % kLanes) * 8;
  const int hi = blockIdx.y, bi = blockIdx.z;
  const int s0 = (blockIdx.x * 8 + warp) * (kRows * kSteps) + lane / kLanes;
  pdl_allow_next();
  const uint16_t* po = o + bi * o_sb + hi * o_sh + col;
  const uint16_t* pd = d_o + bi * do_sb + hi * do_sh + col;
  uint4 a[kSteps], c[kSteps];
#pragma unroll
  for (int i = 0; i < kSteps; ++i) {
    const int si = s0 + i * kRows;
    a[i] = c[i] = make_uint4(0u, 0u, 0u, 0u);
    if (si < s) {
      a[i] = *reinterpret_cast<const uint4*>(po + si * o_ss);
      c[i] = *reinterpret_cast<const uint4*>(pd + si * do_ss);
    }
  }
#pragma unroll
  for (int i = 0; i < kSteps; ++i) {
    const int si = s0 + i * kRows;
    const uint32_t wa[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, wc[4] = {c[i].x, c[i].y, c[i].z, c[i].w};
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float2 fa, fc;
      if (is_bf16) { fa = unpack_bf16x2(wa[k]); fc = unpack_bf16x2(wc[k]); }
      else { fa = __half22float2(*reinterpret_cast<const __half2*>(&wa[k])); fc = __half22float2(*reinterpret_cast<const __half2*>(&wc[k])); }
      acc += fa.x * fc.x + fa.y * fc.y;
    }
#pragma unroll
    for (int k = kLanes / 2; k > 0; k >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
    if (si < pitch && lane % kLanes == 0) {
      const int64_t head = static_cast<int64_t>(bi) * h + hi, row = head * pitch + si;
      const float lv = si < s ? lse[head * s + si] : -INFINITY;
      ndelta[row] = -acc;
      nlse2[row] = lv == -INFINITY ? -INFINITY : -lv * kLog2e;   // fully masked rows give P = 0
    }
  }
}

struct BwdParams {
  const float* nlse;    // [b, hq, pitch] -LSE in the exp2 domain (-lse * log2e)
  const float* ndelta;  // [b, hq, pitch] -delta
  int pitch;            // sq in whole blocks of 64
  void *dq, *dk, *dv;
  int64_t dq_sb, dq_sh, dq_ss, dk_sb, dk_sh, dk_ss, dv_sb, dv_sh, dv_ss;
  int b, hq, hkv, sq, sk;
  float scale_log2, scale;
  int causal;
  int wait_limit;       // tries of a wait before it gives up
  int n_kv;             // CTAs for dK and dV; those behind them are for dQ
};

constexpr int kBwdRows = 128;   // resident rows per CTA (keys for dK/dV, queries for dQ)
constexpr int kBwdCols = 64;    // streamed rows per iteration (queries for dK/dV, keys for dQ)

template <int D>
struct BwdSmem {
  static constexpr int kDC = D / 64;
  static constexpr int kStages = 4;                     // streamed-tile ring depth (hides TMA latency)
  static constexpr int kX = kBwdRows * 128 * kDC;       // resident tile bytes
  static constexpr int kY = kBwdCols * 128 * kDC;       // streamed tile bytes
  static constexpr int kX1Off = 0;
  static constexpr int kX2Off = kX;
  static constexpr int kStageOff = 2 * kX;              // stage s: Y1 at s*2*kY, Y2 at s*2*kY + kY
  static constexpr int kStatOff = kStageOff + kStages * 2 * kY;   // stage s: lse2[64], delta[64] floats
  static constexpr int kBarOff = kStatOff + kStages * 512;
  static constexpr int kTotal = kBarOff + 256 + 1024;
};

// kDQ = false: rows are keys   (X1 = K, X2 = V, Y1 = Q_i, Y2 = dO_i): acc1 = dV, acc2 = dK
// kDQ = true : rows are queries (X1 = Q, X2 = dO, Y1 = K_j, Y2 = V_j): acc1 = dQ
// P / dS (16-bit) go to TMEM columns of their own and feed the accumulate MMAs as the TMEM A operand, so the only shared-memory
// traffic is the operand tiles themselves.
// A block's MMAs take about 1300 cycles (T at N = 64 is bound by its shared-memory reads), its exponentials and products about 2500
// in one warpgroup: a warp per scheduler that waits on its own results.  So the blocks alternate between two T buffers, the
// tensor core working on one while the other's P / dS are made, and two warpgroups share a buffer, 32 columns each.  T is in registers
// 150 cycles after it is complete; its columns then take the next T, so that the math finds it made.  One warp issues T, one the products
// with P / dS: the waits of either take long enough to empty the tensor core's queue.
// CTAs start with the longest rows of a causal problem.  32 / 8 heads x 4096 x 128, both parts: 513 us with P / dS over T, 441 so.
// The maps' boxes are 64 rows high.  bid: this CTA's place among those of its part.
template <int D, bool kDQ, bool kBf16>
__device__ __forceinline__ void bwd_part(const CUtensorMap& tmap_x1, const CUtensorMap& tmap_x2, const CUtensorMap& tmap_y1, const CUtensorMap& tmap_y2,
                                         const BwdParams& p, int bid) {
  using L = BwdSmem<D>;
  constexpr int kS = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sX1 = smem + L::kX1Off;
  uint8_t* sX2 = smem + L::kX2Off;
  uint8_t* sY = smem + L::kStageOff;
  float* sStat = reinterpret_cast<float*>(smem + L::kStatOff);   // stage s: -lse2 at s*128, -delta at s*128+64
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* x_full = bars;               // 1
  uint64_t* y_full = bars + 1;           // kS
  uint64_t* y_empty = bars + 1 + kS;     // kS
  uint64_t* t_full = bars + 1 + 2 * kS;  // 2
  uint64_t* t_read = t_full + 2;         // 2: T1 and T2 are in registers
  uint64_t* pds_ready = t_read + 2;      // 2
  uint64_t* acc_done = pds_ready + 2;    // 2: the P / dS columns are free, the accumulators up to date
  uint64_t* drained = acc_done + 2;      // 1, after a wait that ran out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);
  volatile int* failed = reinterpret_cast<volatile int*>(bars + 25);

  const int warp_idx = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // known to be uniform: see desc_at
  const int lane = threadIdx.x & 31;
  const int G = p.hq / p.hkv;
  // (row block, head, batch) from one grid dimension: every head's longest row block comes before any shorter one
  const int n_out = kDQ ? p.hq : p.hkv;
  const int blk = bid / (n_out * p.b), hb = bid % (n_out * p.b);
  const int out_head = hb % n_out, bi = hb / n_out;
  const int n_blk = ((kDQ ? p.sq : p.sk) + kBwdRows - 1) / kBwdRows;
  const int r0 = (kDQ ? n_blk - 1 - blk : blk) * kBwdRows;
  // iteration space
  int col_blk0, n_col, n_heads, head0;
  if (kDQ) {
    head0 = out_head; n_heads = 1;
    col_blk0 = 0;
    const int kmax = p.causal ? min(p.sk, r0 + kBwdRows) : p.sk;
    n_col = (kmax + kBwdCols - 1) / kBwdCols;
  } else {
    head0 = out_head * G; n_heads = G;
    col_blk0 = p.causal ? r0 / kBwdCols : 0;
    n_col = (p.sq + kBwdCols - 1) / kBwdCols - col_blk0;
    if (n_col < 0) n_col = 0;
  }
  const int n_iter = n_col * n_heads;

  if (threadIdx.x == 0) {
    mbar_init(x_full, 1);
    for (int i = 0; i < kS; ++i) { mbar_init(&y_full[i], 1); mbar_init(&y_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&t_full[i], 1); mbar_init(&t_read[i], 8); mbar_init(&pds_ready[i], 8); mbar_init(&acc_done[i], 1); }
    mbar_init(drained, 2);
    *failed = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_x1); tma_prefetch_desc(&tmap_x2); tma_prefetch_desc(&tmap_y1); tma_prefetch_desc(&tmap_y2);
  }
  if (warp_idx == 2) tmem_alloc<512>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_await_previous();                        // the statistics of the launch before
  volatile int* s_loaded = failed + 2;         // blocks whose copies were started, for the end of a CTA in which a wait ran out
  constexpr int kTBufs = kDQ || D == 64 ? 2 : 1;   // T1 and T2 of dK / dV at D = 128 have room for one block
  const uint32_t tmem_A1 = tmem_base;              // dV or dQ
  const uint32_t tmem_A2 = tmem_base + D;          // dK
  const uint32_t tmem_P = tmem_base + (kDQ ? D : 2 * D);   // [buf] at buf*64: 32 columns of P, 32 of dS
  const uint32_t tmem_T = tmem_P + 128;            // [buf] at buf*128: T1 in 64 columns, T2 in 64
  static_assert((kDQ ? D : 2 * D) + 128 + kTBufs * 128 <= 512, "TMEM columns");

  if (warp_idx < 4) {
    regs_give<kIssueRegs>();
    if (warp_idx == 0 && lane == 0 && n_iter > 0) {
      // ============================================================ TMA producer
      mbar_arrive_expect_tx(x_full, 2 * L::kX);
      for (int c = 0; c < 2 * L::kDC; ++c) {
        const int off = (c >> 1) * (kBwdRows * 128) + (c & 1) * (64 * 128), row = r0 + (c & 1) * 64;
        tma_load_4d(&tmap_x1, x_full, sX1 + off, (c >> 1) * 64, out_head, bi, row);
        tma_load_4d(&tmap_x2, x_full, sX2 + off, (c >> 1) * 64, out_head, bi, row);
      }
      int n_loaded = 0;
      for (; n_loaded < n_iter; ++n_loaded) {
        const int it = n_loaded, ys = it % kS;
        const int head = kDQ ? out_head / G : head0 + it / n_col;   // head of the streamed tiles
        const int c0 = (col_blk0 + it % n_col) * kBwdCols;
        if (!wait_bar(&y_empty[ys], ((it / kS) & 1) ^ 1, failed, p.wait_limit)) break;
        mbar_arrive_expect_tx(&y_full[ys], 2 * L::kY + (kDQ ? 0 : 512));
        uint8_t* y1 = sY + ys * 2 * L::kY;
        uint8_t* y2 = y1 + L::kY;
        for (int c = 0; c < L::kDC; ++c) {
          tma_load_4d(&tmap_y1, &y_full[ys], y1 + c * (kBwdCols * 128), c * 64, head, bi, c0);
          tma_load_4d(&tmap_y2, &y_full[ys], y2 + c * (kBwdCols * 128), c * 64, head, bi, c0);
        }
        if (!kDQ) {
          const int64_t base = (static_cast<int64_t>(bi) * p.hq + head) * p.pitch + c0;
          bulk_load_1d(sStat + ys * 128, p.nlse + base, 256, &y_full[ys]);
          bulk_load_1d(sStat + ys * 128 + 64, p.ndelta + base, 256, &y_full[ys]);
        }
      }
      *s_loaded = n_loaded;
    } else if (warp_idx == 1 && n_iter > 0) {
      // ============================================================ issuer of T1 and T2
      constexpr uint32_t idesc_t = make_idesc_f16(kBf16, kBwdRows, kBwdCols, false, false);
      const uint64_t x_desc = make_smem_desc_sw128(smem_u32(sX1), 1024, 0), y_desc = make_smem_desc_sw128(smem_u32(sY), 1024, 0);
      bool ok = wait_bar_warp(x_full, 0, failed, p.wait_limit);
      for (int it = 0; it < n_iter && ok; ++it) {
        const int ys = it % kS, before = it - kTBufs;          // the block before it in its buffer is in registers
        ok = wait_bar_warp(&y_full[ys], (it / kS) & 1, failed, p.wait_limit) &&
             (before < 0 || wait_bar_warp(&t_read[before & 1], (before >> 1) & 1, failed, p.wait_limit));
        if (!ok) break;
        tc_fence_after();
        const uint32_t tT = tmem_T + (kTBufs == 2 ? (it & 1) * 128 : 0);
        const uint64_t y1 = desc_at(y_desc, ys * 2 * L::kY);
        if (elect_one()) {
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int k = 0; k < D / 16; ++k) {
              const uint32_t xo = x * (L::kX2Off - L::kX1Off) + (k >> 2) * (kBwdRows * 128) + (k & 3) * 32;
              const uint32_t yo = x * L::kY + (k >> 2) * (kBwdCols * 128) + (k & 3) * 32;
              umma_f16_ss(tT + x * 64, desc_at(x_desc, xo), desc_at(y1, yo), idesc_t, k != 0 ? 1u : 0u);
            }
          umma_commit(&t_full[it & 1]);
        }
      }
    } else if (warp_idx == 2) {
      // ============================================================ issuer of the products with P and dS
      constexpr uint32_t idesc_a = make_idesc_f16(kBf16, kBwdRows, D, false, true);
      // streamed tile as MN-major B (N = d contiguous, K = its 64 rows)
      const uint64_t yn_desc = make_smem_desc_sw128(smem_u32(sY), 1024, kBwdCols * 128);
      for (int it = 0; it < n_iter; ++it) {
        const int ys = it % kS, tb = it & 1;
        if (!wait_bar_warp(&y_full[ys], (it / kS) & 1, failed, p.wait_limit) ||
            !wait_bar_warp(&pds_ready[tb], (it >> 1) & 1, failed, p.wait_limit)) break;
        tc_fence_after();
        const uint64_t y1 = desc_at(yn_desc, ys * 2 * L::kY);
        const uint32_t first = it != 0 ? 1u : 0u;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kBwdCols / 16; ++k) {
            // A = P / dS from TMEM (row = lane, 16 k-values = 8 packed 32-bit columns per step)
            const uint32_t tP = tmem_P + tb * 64 + k * 8, acc = k != 0 ? 1u : first;
            if (kDQ) {
              umma_f16_ts(tmem_A1, tP + 32, desc_at(y1, k * 16 * 128), idesc_a, acc);
            } else {
              umma_f16_ts(tmem_A1, tP, desc_at(y1, L::kY + k * 16 * 128), idesc_a, acc);
              umma_f16_ts(tmem_A2, tP + 32, desc_at(y1, k * 16 * 128), idesc_a, acc);
            }
          }
          umma_commit(&acc_done[tb]);
          umma_commit(&y_empty[ys]);
        }
      }
    }
  } else {
    // ============================================================ P / dS math + epilogue
    regs_take<kMathRegs>();
    const int wg = (warp_idx - 4) >> 2;
    const int tb = wg >> 1, half = wg & 1;         // this warpgroup's blocks: it = tb, tb + 2, ...; its columns: 32 half .. 32 half + 31
    const int quad = warp_idx & 3;
    const int r = quad * 32 + lane;
    const int grow = r0 + r;                       // global row (key for dK/dV, query for dQ)
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint64_t sc2 = f2(p.scale_log2, p.scale_log2);
    uint64_t row_nlse = 0, row_ndelta = 0;         // dQ mode: statistics of this thread's query row
    if (kDQ) {
      const int64_t idx = (static_cast<int64_t>(bi) * p.hq + out_head) * p.pitch + min(grow, p.sq - 1);
      row_nlse = f2(p.nlse[idx], p.nlse[idx]);     // already in the exp2 domain (-inf for fully masked rows)
      row_ndelta = f2(p.ndelta[idx], p.ndelta[idx]);
    }
    const uint32_t a1 = tmem_T + (kTBufs == 2 ? tb * 128 : 0) + half * 32 + lane_addr, a2 = a1 + 64;
    const uint32_t tP = tmem_P + tb * 64 + half * 16 + lane_addr;
    // one streamed block: P = exp2(T1 * scale - lse2), dS = P * (T2 - delta), written back to TMEM
    auto block = [&](int it, int c0, auto masked_tag) {
      constexpr bool kMasked = decltype(masked_tag)::value;
      const ulonglong2* s_nlse = reinterpret_cast<const ulonglong2*>(sStat + (it % kS) * 128 + half * 32);
      const ulonglong2* s_ndelta = s_nlse + 16;
      uint32_t t1[2][16], t2[2][16];
      tmem_ld_32x16(a1, t1[0]);
      tmem_ld_32x16(a2, t2[0]);
      tmem_ld_32x16(a1 + 16, t1[1]);
      tmem_ld_32x16(a2 + 16, t2[1]);
      tmem_ld_wait();
      tc_fence_before();
      warp_arrive(&t_read[tb]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pk[8], dk[8];
#pragma unroll
        for (int i4 = 0; i4 < 4; ++i4) {
          ulonglong2 nl = make_ulonglong2(row_nlse, row_nlse), nd = make_ulonglong2(row_ndelta, row_ndelta);
          if (!kDQ) { nl = s_nlse[c * 4 + i4]; nd = s_ndelta[c * 4 + i4]; }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int i = i4 * 4 + e * 2;
            float p0, p1, d0, d1;
            un2(fma2(f2(__uint_as_float(t1[c][i]), __uint_as_float(t1[c][i + 1])), sc2, e == 0 ? nl.x : nl.y), p0, p1);
            p0 = fast_exp2(p0);
            p1 = fast_exp2(p1);
            if (kMasked) {
              const int col = c0 + half * 32 + c * 16 + i;     // global column (query for dK/dV, key for dQ)
              auto hidden = [&](int cc) {
                const int key = kDQ ? cc : grow, qry = kDQ ? grow : cc;
                return (p.causal && key > qry) || key >= p.sk || qry >= p.sq;
              };
              if (hidden(col)) p0 = 0.f;
              if (hidden(col + 1)) p1 = 0.f;
            }
            un2(mul2(f2(p0, p1), add2(f2(__uint_as_float(t2[c][i]), __uint_as_float(t2[c][i + 1])), e == 0 ? nd.x : nd.y)), d0, d1);
            if (!kDQ) pk[i >> 1] = pack16<kBf16>(p0, p1);
            dk[i >> 1] = pack16<kBf16>(d0, d1);
          }
        }
        if (c == 0 && it >= 2) {                           // this buffer's P / dS have been multiplied
          wait_bar_warp(&acc_done[tb], ((it >> 1) - 1) & 1, failed, p.wait_limit);
          tc_fence_after();
        }
        tmem_st_32x8(tP + 32 + c * 8, dk);
        if (!kDQ) tmem_st_32x8(tP + c * 8, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      warp_arrive(&pds_ready[tb]);
    };
    bool ok = true;
    for (int it = tb; it < n_iter; it += 2) {
      const int c0 = (col_blk0 + it % n_col) * kBwdCols;
      ok = wait_bar_warp(&t_full[tb], (it >> 1) & 1, failed, p.wait_limit);
      if (!ok) break;
      tc_fence_after();
      // masking: key index > query index is masked (causal); also ragged tails
      bool need_mask;
      if (kDQ) need_mask = (p.causal && c0 + kBwdCols - 1 > r0) || (c0 + kBwdCols > p.sk) || (r0 + kBwdRows > p.sq);
      else need_mask = (p.causal && c0 < r0 + kBwdRows - 1) || (c0 + kBwdCols > p.sq) || (r0 + kBwdRows > p.sk);
      if (need_mask) block(it, c0, std::true_type{});
      else block(it, c0, std::false_type{});
    }
    // the products of this buffer's last block, then of the last one: a barrier is never more than one phase ahead of a wait
    for (int it = max(0, n_iter - 2); it < n_iter; ++it)
      if (ok && (it == n_iter - 1 || (it & 1) == tb)) ok = wait_bar_warp(&acc_done[it & 1], (it >> 1) & 1, failed, p.wait_limit);
    if (ok) {
      tc_fence_after();
      const int limit = kDQ ? p.sq : p.sk;
      const bool valid = grow < limit;
      auto store_acc = [&](uint32_t tacc, void* out, int64_t sb, int64_t sh, int64_t ss, float mul, int ch0, int ch1) {
        uint8_t* orow = reinterpret_cast<uint8_t*>(out) +
                        (static_cast<int64_t>(grow) * ss + static_cast<int64_t>(bi) * sb + static_cast<int64_t>(out_head) * sh) * 2;
        for (int c = ch0; c < ch1; ++c) {
          uint32_t v[32];
          if (n_iter > 0) {
            tmem_ld_32x32(tacc + c * 32 + lane_addr, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
          if (valid) store_row32<kBf16>(orow + c * 64, v, mul);
        }
      };
      // the warpgroups share the epilogue: 32 columns of dQ each, or half of dV's or dK's
      if (kDQ) store_acc(tmem_A1, p.dq, p.dq_sb, p.dq_sh, p.dq_ss, p.scale, min(wg, D / 32), min(wg + 1, D / 32));
      else if (tb == 0) store_acc(tmem_A1, p.dv, p.dv_sb, p.dv_sh, p.dv_ss, 1.f, half * (D / 64), (half + 1) * (D / 64));
      else store_acc(tmem_A2, p.dk, p.dk_sb, p.dk_sh, p.dk_ss, p.scale, half * (D / 64), (half + 1) * (D / 64));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*failed) {                                  // every wait is over, so all threads read the same
    volatile int never = 0;
    if (threadIdx.x == 0) {
      atomicExch(&g_attn_error, 1);
      wait_bar(x_full, 0, &never);
      const int n_loaded = *s_loaded;
      for (int i = max(0, n_loaded - kS); i < n_loaded; ++i) wait_bar(&y_full[i % kS], (i / kS) & 1, &never);
    } else if (warp_idx == 1 || warp_idx == 2) {
      if (elect_one()) umma_commit(drained);
      wait_bar_warp(drained, 0, &never);
    } else if (warp_idx >= 4) {
      const int rows = min(kBwdRows, (kDQ ? p.sq : p.sk) - r0);
      auto fill = [&](void* out, int64_t sb, int64_t sh, int64_t ss) {
        fill_nan<D>(out, static_cast<int64_t>(r0) * ss + static_cast<int64_t>(bi) * sb + static_cast<int64_t>(out_head) * sh, ss, rows);
      };
      if (kDQ) {
        fill(p.dq, p.dq_sb, p.dq_sh, p.dq_ss);
      } else {
        fill(p.dv, p.dv_sb, p.dv_sh, p.dv_ss);
        fill(p.dk, p.dk_sb, p.dk_sh, p.dk_ss);
      }
    }
    __syncthreads();
  }
  if (warp_idx == 2) tmem_dealloc<512>(tmem_base);
}

// dK and dV first, then dQ, each with its longest rows first: neither waits for the other, and the short rows of the former end under the long ones of
// the latter.  us of a backward call, a launch each / one: 1 x 32 / 8 heads x 4096 x 128 457 / 439, x 512 54 / 41; 4 x 12 x 1024 x 64 73 / 64, 2 x 16 x 256
// x 64 23 / 12.5 (neither part fills the SMs).
template <int D, bool kBf16>
__global__ void __launch_bounds__(kThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                const __grid_constant__ CUtensorMap tmap_do, const BwdParams p) {
  const int bid = static_cast<int>(blockIdx.x);
  if (bid < p.n_kv) bwd_part<D, false, kBf16>(tmap_k, tmap_v, tmap_q, tmap_do, p, bid);
  else bwd_part<D, true, kBf16>(tmap_q, tmap_do, tmap_k, tmap_v, p, bid - p.n_kv);
}

// ------------------------------------------------------------------------------------ host side
typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(ptr);
  });
  return fn;
}
thread_local std::string g_attn_err;

// 4-D map over a strided [b, h, s, d] view: dims (d, h, b, s); box (64, 1, 1, rows)
bool make_tmap_bhsd(CUtensorMap* map, const void* base, bool is_bf16, int d, int h, int b, int s, int64_t sh,
                    int64_t sb, int64_t ss, int rows) {
  ensure_cuda_context();
  EncodeFn fn = encode_fn();
  if (!fn) { g_attn_err = "cuTensorMapEncodeTiled unavailable"; return false; }
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(d), static_cast<cuuint64_t>(h), static_cast<cuuint64_t>(b),
                        static_cast<cuuint64_t>(s)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(sh) * 2, static_cast<cuuint64_t>(sb) * 2,
                           static_cast<cuuint64_t>(ss) * 2};
  cuuint32_t box[4] = {64, 1, 1, static_cast<cuuint32_t>(rows)};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                  const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    g_attn_err = "cuTensorMapEncodeTiled(4d) failed: code " + std::to_string(static_cast<int>(r));
    return false;
  }
  return true;
}

// once per kernel: its shared memory, and that its register shares (regs_take / regs_give) fit what it is launched with
template <typename K>
bool prepare_kernel(K kern, int smem, const char* name, int threads, int shares) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) { g_attn_err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e); return false; }
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess || fa.numRegs * threads < shares) {
    g_attn_err = std::string(name) + ": built with too few registers for its warpgroups' shares";
    return false;
  }
  return true;
}

bool strides_ok(int64_t sb, int64_t sh, int64_t ss, const void* ptr) {
  return (sb % 8 == 0) && (sh % 8 == 0) && (ss % 8 == 0) && (reinterpret_cast<uintptr_t>(ptr) % 16 == 0);
}

template <int D, bool kBf16>
int launch_fwd(const AttnArgs& a, cudaStream_t s) {
  using L = FwdSmem<D>;
  CUtensorMap tq{}, tk{}, tv{};
  if (!make_tmap_bhsd(&tq, a.q, a.is_bf16, D, a.hq, a.b, a.sq, a.q_sh, a.q_sb, a.q_ss, kBlockQ)) return -5;
  if (!make_tmap_bhsd(&tk, a.k, a.is_bf16, D, a.hkv, a.b, a.sk, a.k_sh, a.k_sb, a.k_ss, kBlockKV)) return -5;
  if (!make_tmap_bhsd(&tv, a.v, a.is_bf16, D, a.hkv, a.b, a.sk, a.v_sh, a.v_sb, a.v_ss, kBlockKV)) return -5;
  auto kern = attn_fwd_kernel<D, kBf16>;
  static const bool ready = prepare_kernel(kern, L::kTotal, "attn_fwd", kFwdThreads, 256 * kFwdMathRegs + 128 * kFwdIssueRegs);
  if (!ready) return -10;
  FwdParams p{};
  p.lse = a.lse; p.o = a.o; p.o_sb = a.o_sb; p.o_sh = a.o_sh; p.o_ss = a.o_ss;
  p.b = a.b; p.hq = a.hq; p.hkv = a.hkv; p.sq = a.sq; p.sk = a.sk;
  p.scale_log2 = a.scale * kLog2e; p.causal = a.causal ? 1 : 0; p.wait_limit = a.wait_limit < 0 ? kWaitLimit : a.wait_limit;
  const int64_t ctas = static_cast<int64_t>((a.sq + 2 * kBlockQ - 1) / (2 * kBlockQ)) * a.hq * a.b;
  if (ctas > 0x7fffffff) { g_attn_err = "too many query blocks"; return -12; }
  kern<<<static_cast<unsigned>(ctas), kFwdThreads, L::kTotal, s>>>(tq, tk, tv, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { g_attn_err = std::string("attn_fwd launch: ") + cudaGetErrorString(e); return -11; }
  return 0;
}


template <int D, bool kBf16>
int launch_bwd_parts(const AttnArgs& a, cudaStream_t s) {
  using L = BwdSmem<D>;
  CUtensorMap tq{}, tk{}, tv{}, tdo{};
  if (!make_tmap_bhsd(&tq, a.q, a.is_bf16, D, a.hq, a.b, a.sq, a.q_sh, a.q_sb, a.q_ss, kBwdCols) ||
      !make_tmap_bhsd(&tk, a.k, a.is_bf16, D, a.hkv, a.b, a.sk, a.k_sh, a.k_sb, a.k_ss, kBwdCols) ||
      !make_tmap_bhsd(&tv, a.v, a.is_bf16, D, a.hkv, a.b, a.sk, a.v_sh, a.v_sb, a.v_ss, kBwdCols) ||
      !make_tmap_bhsd(&tdo, a.d_o, a.is_bf16, D, a.hq, a.b, a.sq, a.do_sh, a.do_sb, a.do_ss, kBwdCols))
    return -5;
  auto kern = attn_bwd_kernel<D, kBf16>;
  static const bool ready = prepare_kernel(kern, L::kTotal, "attn_bwd", kThreads, 512 * kMathRegs + 128 * kIssueRegs);
  if (!ready) return -10;
  BwdParams p{};
  p.pitch = attn_stat_pitch(a.sq);
  p.nlse = a.delta + static_cast<int64_t>(a.b) * a.hq * p.pitch;   // written by attn_delta_kernel
  p.ndelta = a.delta;
  p.dq = a.dq; p.dq_sb = a.dq_sb; p.dq_sh = a.dq_sh; p.dq_ss = a.dq_ss;
  p.dk = a.dk; p.dk_sb = a.dk_sb; p.dk_sh = a.dk_sh; p.dk_ss = a.dk_ss;
  p.dv = a.dv; p.dv_sb = a.dv_sb; p.dv_sh = a.dv_sh; p.dv_ss = a.dv_ss;
  p.b = a.b; p.hq = a.hq; p.hkv = a.hkv; p.sq = a.sq; p.sk = a.sk;
  p.scale_log2 = a.scale * kLog2e; p.scale = a.scale; p.causal = a.causal ? 1 : 0; p.wait_limit = a.wait_limit < 0 ? kWaitLimit : a.wait_limit;
  const int64_t n_kv = static_cast<int64_t>((a.sk + kBwdRows - 1) / kBwdRows) * a.hkv * a.b, n_q = static_cast<int64_t>((a.sq + kBwdRows - 1) / kBwdRows) * a.hq * a.b;
  if (n_kv + n_q > 0x7fffffff) { g_attn_err = "too many row blocks"; return -12; }
  p.n_kv = static_cast<int>(n_kv);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(n_kv + n_q));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = L::kTotal;
  cfg.stream = s;
  cudaLaunchAttribute attr{};                    // CTAs may start under the statistics' kernel, and wait for its end
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tq, tk, tv, tdo, p);
  if (e != cudaSuccess) { g_attn_err = std::string("attn_bwd launch: ") + cudaGetErrorString(e); return -11; }
  return 0;
}

template <int D>
int launch_bwd(const AttnArgs& a, cudaStream_t s) {
  const int pitch = attn_stat_pitch(a.sq);
  const int64_t rows = static_cast<int64_t>(a.b) * a.hq * pitch;
  constexpr int kPerBlock = 8 * 4 * (256 / D);   // warps x row groups x rows
  if (a.hq > 65535 || a.b > 65535) { g_attn_err = "too many heads or sequences"; return -12; }
  attn_delta_kernel<D><<<dim3((pitch + kPerBlock - 1) / kPerBlock, a.hq, a.b), 256, 0, s>>>(
      static_cast<const uint16_t*>(a.o), static_cast<const uint16_t*>(a.d_o), a.delta, a.lse, a.delta + rows, a.hq, a.sq, pitch, a.o_sb, a.o_sh, a.o_ss,
      a.do_sb, a.do_sh, a.do_ss, a.is_bf16 ? 1 : 0);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { g_attn_err = std::string("attn_delta launch: ") + cudaGetErrorString(e); return -11; }
  return a.is_bf16 ? launch_bwd_parts<D, true>(a, s) : launch_bwd_parts<D, false>(a, s);
}

}  // namespace

const char* attn_last_error() { return g_attn_err.c_str(); }

int attn_stat_pitch(int sq) { return (sq + kBwdCols - 1) / kBwdCols * kBwdCols; }

int attn_status(bool clear) {
  int v = 0;
  const int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_attn_error, sizeof(int)) != cudaSuccess) return -1;
  if (clear && v != 0 && cudaMemcpyToSymbol(g_attn_error, &zero, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

int attn_fwd(const AttnArgs& a, cudaStream_t s) {
  if (a.d != 64 && a.d != 128) { g_attn_err = "head dim must be 64 or 128"; return -1; }
  if (a.hq % a.hkv != 0) { g_attn_err = "hq must be a multiple of hkv"; return -1; }
  if (a.causal && a.sq != a.sk) { g_attn_err = "causal attention needs sq == sk"; return -2; }
  if (a.probs_out) { g_attn_err = "probability export uses the materialising path"; return -3; }
  if (!strides_ok(a.q_sb, a.q_sh, a.q_ss, a.q) || !strides_ok(a.k_sb, a.k_sh, a.k_ss, a.k) ||
      !strides_ok(a.v_sb, a.v_sh, a.v_ss, a.v) || !strides_ok(a.o_sb, a.o_sh, a.o_ss, a.o)) {
    g_attn_err = "q/k/v/o need 16-byte aligned base and strides";
    return -4;
  }
  if (a.is_bf16) return a.d == 128 ? launch_fwd<128, true>(a, s) : launch_fwd<64, true>(a, s);
  return a.d == 128 ? launch_fwd<128, false>(a, s) : launch_fwd<64, false>(a, s);
}

int attn_bwd(const AttnArgs& a, cudaStream_t s) {
  if (a.d != 64 && a.d != 128) { g_attn_err = "head dim must be 64 or 128"; return -1; }
  if (a.hq % a.hkv != 0) { g_attn_err = "hq must be a multiple of hkv"; return -1; }
  if (a.causal && a.sq != a.sk) { g_attn_err = "causal attention needs sq == sk"; return -2; }
  if (!a.causal && (a.sq % kBwdCols != 0 || a.sk % kBwdCols != 0)) { g_attn_err = "backward that is not causal needs sq, sk multiples of 64"; return -3; }
  if (!strides_ok(a.q_sb, a.q_sh, a.q_ss, a.q) || !strides_ok(a.k_sb, a.k_sh, a.k_ss, a.k) ||
      !strides_ok(a.v_sb, a.v_sh, a.v_ss, a.v) || !strides_ok(a.o_sb, a.o_sh, a.o_ss, a.o) ||
      !strides_ok(a.do_sb, a.do_sh, a.do_ss, a.d_o) || !strides_ok(a.dq_sb, a.dq_sh, a.dq_ss, a.dq) ||
      !strides_ok(a.dk_sb, a.dk_sh, a.dk_ss, a.dk) || !strides_ok(a.dv_sb, a.dv_sh, a.dv_ss, a.dv)) {
    g_attn_err = "attention operands need 16-byte aligned base and strides";
    return -4;
  }
  return a.d == 128 ? launch_bwd<128>(a, s) : launch_bwd<64>(a, s);
}

}  // namespace b200
