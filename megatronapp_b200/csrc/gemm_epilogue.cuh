// Epilogue of the tcgen05 GEMMs: accumulators -> registers -> shared memory -> TMA store.
//
// A warp drains its own 32 rows, 64 columns of 16 bits or 32 of fp32 at a time, through two 4 KB slabs of its own: no warp waits for another, the bias comes
// as one load a slab, and what the problem asks for (type, activation, bias) is decided once per slab and not per element.  In cycles, of
// one 256 x 256 tile of a CTA pair, beside 6400 of 12 k-blocks of MMAs: 3700, with a bias 5900; slabs of 128 rows between barriers of the four
// warps, every element's form chosen by selects, 7800, with a bias (a 4-byte load in front of every pair) 20300.
#pragma once
#include "common.cuh"

#include <type_traits>

namespace b200 {
namespace {

constexpr uint32_t kSlabRows = 32, kSlabBytes = kSlabRows * 128;

__device__ __forceinline__ float gelu_tanh(float x) {
  return 0.5f * x * (1.f + tanhf(0.79788456f * x * (1.f + 0.044715f * x * x)));
}

// 64 accumulator columns of one row (a lane's), + bias, GELU, row scale, as 16 bits into the row's 128 swizzled bytes of a staging slab.
// `bias2`: the lane's two of the 64 columns' bias values; the others come by shuffles, whatever the pointer's alignment.
template <bool kBf16, bool kGelu, bool kBias, bool kScale>
__device__ __forceinline__ void stage_row16(uint32_t row, int swz, const uint32_t (&v0)[32], const uint32_t (&v1)[32], uint32_t bias2, float scale) {
  uint32_t bb[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) bb[i] = kBias ? __shfl_sync(0xffffffffu, bias2, i) : 0u;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint32_t pk[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = j * 8 + 2 * q;
      uint32_t ua = i < 32 ? v0[i] : v1[i - 32], ub = i < 32 ? v0[i + 1] : v1[i - 31];
      // values of this branch's own: the compiler would otherwise make every form (both types, the tanh of all elements) before it looks which one
      // is wanted, 1200 cycles a slab
      asm volatile("" : "+r"(ua), "+r"(ub));
      float a = __uint_as_float(ua), b = __uint_as_float(ub);
      if constexpr (kBias) {
        const float2 bf = kBf16 ? unpack_bf16x2(bb[j * 4 + q]) : __half22float2(*reinterpret_cast<const __half2*>(&bb[j * 4 + q]));
        a += bf.x;
        b += bf.y;
      }
      if constexpr (kGelu) { a = gelu_tanh(a); b = gelu_tanh(b); }
      if constexpr (kScale) { a *= scale; b *= scale; }
      if constexpr (kBf16) pk[q] = pack_bf16x2(a, b);
      else {
        const __half2 h = __floats2half2_rn(a, b);
        pk[q] = *reinterpret_cast<const uint32_t*>(&h);
      }
    }
    st_shared_v4(row + ((j ^ swz) << 4), pk[0], pk[1], pk[2], pk[3]);
  }
}
// the bias of columns col + 2 lane and col + 2 lane + 1, of any alignment
__device__ __forceinline__ uint32_t bias_pair(const uint16_t* bias, int col, int n, int lane) {
  col += 2 * lane;
  if (bias == nullptr || col >= n) return 0u;
  return ld_awaited(bias + col) | (col + 1 < n ? ld_awaited(bias + col + 1) << 16 : 0u);
}

// one warp's two slabs and where they go: rows `row0` on of a matrix, nothing where these lie below it
struct Slabs {
  int lane, buf = 0, row0 = 0;
  bool inside = false;
  uint8_t* base = nullptr;
  __device__ __forceinline__ explicit Slabs(int lane_) : lane(lane_) {}
  __device__ __forceinline__ void at(uint8_t* smem, int row, bool in) {
    base = smem;
    row0 = row;
    inside = in;
  }
  // this lane's row of the next slab, whose last store has been read
  __device__ __forceinline__ uint32_t next() {
    if (lane == 0) tma_store_wait_read<1>();
    __syncwarp();
    return smem_u32(base) + buf * kSlabBytes + lane * 128;
  }
  template <bool kAdd>
  __device__ __forceinline__ void send(const CUtensorMap* map, int col) {
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      if (inside) {
        if constexpr (kAdd) tma_reduce_add_2d(map, base + buf * kSlabBytes, col, row0);
        else tma_store_2d(map, base + buf * kSlabBytes, col, row0);
      }
      tma_store_commit();
    }
    buf ^= 1;
  }
  template <bool kScale>
  __device__ __forceinline__ void store16(const CUtensorMap* map, int col, bool bf16, bool gelu, bool bias, const uint32_t (&v0)[32],
                                          const uint32_t (&v1)[32], uint32_t bias2, float scale) {
    const uint32_t row = next();
    auto go = [&](auto b, auto g, auto w) { stage_row16<b.value, g.value, w.value, kScale>(row, lane & 7, v0, v1, bias2, scale); };
    using T = std::true_type;
    using F = std::false_type;
    if (bf16) {
      if (gelu) bias ? go(T{}, T{}, T{}) : go(T{}, T{}, F{});
      else bias ? go(T{}, F{}, T{}) : go(T{}, F{}, F{});
    } else {
      if (gelu) bias ? go(F{}, T{}, T{}) : go(F{}, T{}, F{});
      else bias ? go(F{}, F{}, T{}) : go(F{}, F{}, F{});
    }
    send<false>(map, col);
  }
  template <bool kAdd>
  __device__ __forceinline__ void store32(const CUtensorMap* map, int col, const uint32_t (&v)[32]) {
    const uint32_t row = next();
#pragma unroll
    for (int j = 0; j < 8; ++j) st_shared_v4(row + ((j ^ (lane & 7)) << 4), v[j * 4], v[j * 4 + 1], v[j * 4 + 2], v[j * 4 + 3]);
    send<kAdd>(map, col);
  }
};

}  // namespace
}  // namespace b200
