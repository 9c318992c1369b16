// Attention forward, what its two kernels (fa_fwd.cu, fa_split.cu) share: the tile shapes, and the softmax of
// one tile of scores by the thread that owns the row.
#pragma once
#include "tcgen05.cuh"

namespace ixb {
namespace fa {

constexpr int BM = 128;          // rows of one query tile
constexpr int NQ = 2;            // tiles of scores in tensor memory
constexpr int BN = 128;          // keys per tile
constexpr int HD = 128;          // head dimension
constexpr int kTileBytes = BN * HD * 2;     // one operand tile, 16-bit elements
constexpr int kHalfBytes = kTileBytes / 2;  // one 64-column TMA box of the tile
constexpr int kThreads = 128 + NQ * 128;  // a warpgroup for producer and issuer, one per tile of scores
constexpr int kSplit = 96;  // keys of P handed to the tensor core ahead of the rest of the tile
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColS = 0, kColO = 256;  // + 128 * tile
constexpr float kRescaleThreshold = 8.f;    // log2 units

__device__ __forceinline__ uint32_t pack_pair(float lo, float hi, bool is_bf16) {
  if (is_bf16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Scores of this thread's row (tensor memory at s_addr) to probabilities relative to the running reference
// maximum m_used, written over them as 16-bit pairs and handed over in two parts (p_full after kSplit keys,
// p_rest); l grows by their sum.  `edge`: keys behind `lim` (relative to the tile) are hidden from this
// row.  `first`: the row's accumulator at o_addr holds nothing yet.
template <bool IS_BF16>
__device__ __forceinline__ void softmax_tile(uint32_t s_addr, uint32_t o_addr, bool edge, int lim, bool first, float scale_log2,
                                             float& m_used, float& l, uint64_t* p_full, uint64_t* p_rest) {
  // the row of scores stays in registers: one trip through tensor memory per tile
  uint32_t raw[BN];
#pragma unroll
  for (int c = 0; c < BN / 32; ++c)
    tc::tmem_ld32(s_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&raw[c * 32]));
  tc::tmem_wait_ld();
  if (edge) {
#pragma unroll
    for (int c = 0; c < BN / 32; ++c) {
      if (__all_sync(kFull, lim >= c * 32 + 31)) continue;  // (what every row of the warp sees stays)
#pragma unroll
      for (int e = c * 32; e < c * 32 + 32; ++e)
        if (e > lim) raw[e] = 0xff800000u;  // -inf
    }
  }
  // four independent chains: one chain of 64 dependent max3 would cost its latency 64 times
  float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int e = 0; e < BN; e += 2)
    mx4[(e >> 1) & 3] = max3(mx4[(e >> 1) & 3], __uint_as_float(raw[e]), __uint_as_float(raw[e + 1]));
  float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
  mx *= scale_log2;  // scale > 0: scaling commutes with the maximum
  // lazy rescale: move the reference maximum only when it would grow by > 2^8
  const bool grow = mx > m_used + kRescaleThreshold;  // also true for the first tile
  if (__any_sync(kFull, grow)) {
    const float m_new = grow ? mx : m_used;
    const float f = !grow ? 1.f : ((m_used == -INFINITY) ? 0.f : fast_exp2(m_used - m_new));
    l *= f;
    if (!first) {
      // O may only be touched once O += P(j-1) V(j-1) has completed: it has - S(j),
      // which this warp has waited for, was committed behind it
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tc::tmem_ld32(o_addr + c * 32, o);
        tc::tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
        tc::tmem_st32(o_addr + c * 32, o);
      }
      tc::tmem_wait_st();
    }
    m_used = m_new;
  }
  // ---- P = exp2(s * scale - m_used), written over the scores as 16-bit pairs
  const float mref = (m_used == -INFINITY) ? 0.f : m_used;
  const float2 sc2 = make_float2(scale_log2, scale_log2);
  const float2 nm2 = make_float2(-mref, -mref);
  float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};  // two chains of packed adds
#pragma unroll
  for (int c = 0; c < BN / 32; ++c) {
    uint32_t pk[16];
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
      const float2 a = fma2(make_float2(__uint_as_float(raw[c * 32 + e]), __uint_as_float(raw[c * 32 + e + 1])), sc2, nm2);
      const float2 pe = make_float2(fast_exp2(a.x), fast_exp2(a.y));
      sum2[(e >> 1) & 1] = add2(sum2[(e >> 1) & 1], pe);
      pk[e / 2] = pack_pair(pe.x, pe.y, IS_BF16);
    }
    tc::tmem_st16(s_addr + c * 16, pk);
    if (c * 32 + 32 == kSplit) {
      tc::tmem_wait_st();
      tc::fence_before_sync();
      tc::mbar_arrive(p_full);
    }
  }
  tc::tmem_wait_st();
  tc::fence_before_sync();
  tc::mbar_arrive(p_rest);
  l += (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
}

}  // namespace fa
}  // namespace ixb
