// Fused attention backward for sm_100a: gradients of softmax(Q K^T * scale [+ causal mask]) V
// with tcgen05 tensor-core MMAs, accumulators in tensor memory and operands brought in by
// TMA.  It takes the place of the vendor kernel behind torch.ops.npu_graph.npu_fa_backward
// (inductor_x/npu_fusion_attention_graph.py:38-42).
//
// With P = exp(S * scale - lse), dP = dO V^T, delta = rowsum(dO * O) and
// dS = P * (dP - delta):   dV = P^T dO,   dK = scale * dS^T Q,   dQ = scale * dS K.
// No atomics, one owner for every output, so the bits are the same from run to run:
//   fa_bwd_delta_kernel  delta[b, h, i] (half a warp per row)
//   fa_bwd_dkv_kernel    one CTA owns a 128-key tile and walks the query tiles that see it;
//                        it forms S^T = K Q^T and dP^T = V dO^T (thread <-> key, columns <->
//                        queries), so that P^T and dS^T - written back over S^T and dP^T as
//                        16-bit values - are the TMEM operands of dV += P^T dO and
//                        dK += dS^T Q, which stay in TMEM until the tile is finished.  With
//                        scratch, four warps copy the 16-bit dS^T to memory.  A CTA that has finished
//                        takes over a pending tile (cluster launch control): its K, V and first Q and dO
//                        arrive, and its first scores are formed, under the end of the one before
//   fa_bwd_dq_ds_kernel  one CTA owns two query tiles: dQ += dS K, with dS from memory
//   fa_bwd_dq_kernel     the same without scratch: S = Q K^T, dP = dO V^T (thread <-> query),
//                        dS over dP, dQ += dS K - the probabilities are computed once more, seven
//                        products instead of five
//
// Warp 0 is the TMA producer, warp 1 the MMA issuer; 4 * NG warps do the element-wise work in NG
// groups of four warps that split the 128 columns of a tile between them (a warp may only touch the
// 32 TMEM lanes of its quadrant; no row reduction is needed here - lse and delta come in
// precomputed - so the split costs nothing).  Every wait is bounded; a wait that gives up raises a
// flag in `status`, and the CTA exits when the copies and products under way have ended.
//
// Bound.  In a run of calls the power limit (1000 W, clocks down to 1.5 - 1.7 GHz): at 4 x 32 heads,
// 4096 keys, causal, bf16 a call took 1865 us (delta 60, dK/dV 1165 - 1190, dQ 825), 1800 with the
// reworked dK/dV (1000), 1625 with dS kept (dK/dV 1240, dQ 400); 8 heads without a mask, short enough
// for the full clock: 229, 226, 214; 8 x 16 heads of 1000, no mask: 315, 291, 265.  Keeping dS
// spares two of seven products and costs 4.4 GB to and from memory at the first of these sizes; what
// dK/dV loses to its stores (240 us) dQ gains nearly twice.
// Inside a step of dK/dV the chain is S -> P -> dV, next S: at the full clock 3100 cycles, of which the
// tensor core works 2048.  What shortened it: P handed over group by group, Q and dO in rings of
// their own whose copies are asked for before anything else, the statistics of a tile read ahead into
// registers (with both operands in shared memory a product takes all 128 bytes a cycle of it, and
// reads beside it are slow).  A tile took 13000 cycles besides its steps while each had a CTA of its own
// (the launch, tensor memory, the first copies, the results): calls in which tiles are taken over, before and
// after: 4 x 32 heads of 4096 causal 1590 and 1500 us, 10 x 16 of 1851 525 and 483, 8 x 32 of 1000 326 and 284,
// 8 x 16 of 1000 without a mask 246 and 226, 8 x 32 of 196 70 and 61.  Two tiles in flight would need more
// tensor memory than one SM has.
// Built, measured and dropped: a share of the exponentials on the fma pipe (1049 - 1070 against 1000:
// the ex2 unit is not the limit, power is); sixteen element-wise warps (the same); dS to memory by way
// of shared memory and bulk copies (171 against 162 for the 8 heads) or stored by the element-wise
// warps themselves (184); dS in tensor-memory columns of its own (dQ 1.51 -> 1.83 ms); P^T as a
// shared-memory operand (dK/dV 2.12 -> 2.36 ms); 64-query sub-tiles (30 % slower: an SS-form MMA with
// N = 64 takes 48 cycles, not 32).
#include <atomic>
#include "fa_maps.h"
#include "ixb/tcgen05.cuh"

namespace {

using namespace ixb;

constexpr int BM = 128;  // query rows per tile
constexpr int BN = 128;  // keys per tile
constexpr int HD = 128;  // head dimension
constexpr int kStages = 2;  // (the issuers pick stage descriptors with two-way selects: no local-memory arrays)
constexpr int kTileBytes = 128 * HD * 2;
constexpr int kHalfBytes = kTileBytes / 2;
constexpr int NG = 2;             // groups of element-wise warps; each takes 128 / NG columns of a tile
constexpr int GC = 128 / NG;      // columns per group
constexpr int kWorkers = 128 * NG;
constexpr int kThreads = 64 + kWorkers;
constexpr int kDkvThreads = 128 * (2 + NG);  // dK/dV: issuers, element-wise groups, dS stores: a warpgroup each
// Registers of the dK/dV kernel: launched with what 16 warps can have; the element-wise warps hold a
// tile's statistics besides its scores.
constexpr int kRegsLaunch = 128, kRegsIssue = 80, kRegsWork = 168, kRegsStore = 96;
static_assert(kRegsIssue + NG * kRegsWork + kRegsStore <= (2 + NG) * kRegsLaunch, "setmaxnreg draws on the block's own registers");
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColS = 0, kColDP = 128, kColAcc0 = 256, kColAcc1 = 384;
constexpr size_t kSmemBytes = (size_t)kTileBytes * 6 + 1024;

struct Out {
  void* ptr;
  long long sb, sh, ss;  // strides in elements
  bool wide;             // every row is a multiple of 32 bytes
};
struct BwdParams {
  const float* lse;    // [B, H, Sq] natural-log sum of exponentials of the forward
  const float* delta;  // [B, H, Sq] rowsum(dO * O)
  Out dq, dk, dv;
  int* status;
  int B, H, Sq, Sk;
  float scale, scale_log2;
  int causal;
  int head_group;
  unsigned char* ds;   // tiles of dS^T of the heads of this launch (see ds_tile), or null
  int bh0, n_bh;       // first head of this launch and how many (all of them where dS is not kept)
  int tiles_per_head;  // tiles of dS^T a head has
};

// dS^T goes to memory in tiles of 128 keys x 128 queries of 16-bit values, every tile in the form in
// which it is read back as a shared-memory operand: 16-byte pieces of 8 queries of one key, piece
// ((key / 32) * 16 + query / 8) * 32 + key % 32.  A warp (32 keys) stores 512 contiguous bytes an
// instruction, a tile is one 32 KB bulk copy.  Only tiles that some query of the tile sees are kept,
// key tile by key tile.
// Tile (kv, i) of a head: key tile kv sees query tiles from kv - hide on.
__host__ __device__ __forceinline__ int hidden_tiles(int causal, int Sq, int Sk, int n_kv_tiles) {
  return causal ? (Sk - Sq + 127) / 128 : n_kv_tiles;  // kv <= hide: every query tile
}
__host__ __device__ __forceinline__ long long ds_tile(int kv, int i, int n_q_tiles, int hide) {
  const long long u = kv > hide + 1 ? kv - 1 - hide : 0;  // query tiles that key tiles before kv do not see
  return (long long)kv * n_q_tiles - u * (u + 1) / 2 + i - (kv > hide ? kv - hide : 0);
}

__device__ __forceinline__ uint32_t pack_pair(float lo, float hi, bool is_bf16) {
  if (is_bf16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_pair(uint32_t w, bool is_bf16) {
  if (is_bf16) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}

// One arrival per warp: every lane has fenced its tensor-memory accesses, the warp
// synchronises, lane 0 arrives (the barrier counts warps, not threads).
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) tc::mbar_arrive(bar);
}

// ------------------------------------------------------------------------------ delta
template <bool IS_BF16>
__global__ void __launch_bounds__(256)
    fa_bwd_delta_kernel(const unsigned char* o, const unsigned char* dout, float* delta, int H, int Sq,
                        long long rows, long long o_sb, long long o_sh, long long o_ss, long long d_sb,
                        long long d_sh, long long d_ss) {
  // half a warp per row: 16 lanes x 16 bytes = the 128 16-bit values of a row
  const int lane = threadIdx.x & 31, sub = lane & 15;
  const long long row = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * 2 + (lane >> 4);
  float s = 0.f;
  if (row < rows) {
    const long long bh = row / Sq;
    const long long i = row - bh * Sq;
    const long long b = bh / H, h = bh - b * H;
    const uint4 a = ldg_stream(reinterpret_cast<const uint4*>(o + 2 * (b * o_sb + h * o_sh + i * o_ss) + sub * 16));
    const uint4 g = ldg_stream(reinterpret_cast<const uint4*>(dout + 2 * (b * d_sb + h * d_sh + i * d_ss) + sub * 16));
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = unpack_pair(aw[e], IS_BF16), y = unpack_pair(gw[e], IS_BF16);
      s = fmaf(x.x, y.x, fmaf(x.y, y.y, s));
    }
  }
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(kFull, s, off);
  if (sub == 0 && row < rows) delta[row] = s;
}

// --------------------------------------------------------------------- shared pieces
// CTA order: heads in groups of `head_group` (their operands stay in L2 while the group
// runs); inside a group tile `slot` of every head before tile `slot + 1` of any.
__device__ __forceinline__ void cta_order(int index, int n_tiles, int n_bh, int head_group, int* slot, int* bh) {
  const int per_group = n_tiles * head_group;
  const int group = index / per_group;
  const int in_group = index - group * per_group;
  const int left = n_bh - group * head_group;
  const int g_heads = left < head_group ? left : head_group;
  *slot = in_group / g_heads;
  *bh = group * head_group + in_group % g_heads;
}

__device__ __forceinline__ void load_tile(unsigned char* dst, const CUtensorMap* map, uint64_t* bar, int row0,
                                          int h, int b) {
  tc::tma_load_4d(dst, map, bar, 0, row0, h, b);
  tc::tma_load_4d(dst + kHalfBytes, map, bar, 64, row0, h, b);
}

// The products are issued by a whole warp through an elected lane (see tc::product_ss).
// D = A B^T, both operands K-major tiles of 128 x 128 (8 steps of 16 along the head dimension)
__device__ __forceinline__ void issue_ss(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
  tc::product_ss<kHalfBytes>(d, a_desc, b_desc, idesc);
}
// D (+)= A B with A in TMEM as 16-bit pairs (group g wrote its GC values of the reduced index
// as GC / 2 columns starting at column a + GC * g) and B a tile in MN-major form (16 rows =
// 2048 bytes a step)
__device__ __forceinline__ void issue_ts(uint32_t d, uint32_t a, uint64_t b_desc_mn, uint32_t idesc,
                                         bool accumulate) {
#pragma unroll
  for (int g = 0; g < NG; ++g)
    tc::product_ts<GC / 16>(d, a + g * GC, b_desc_mn + (uint32_t)(g * GC * 128 >> 4), idesc, (accumulate || g > 0) ? 1u : 0u);
}

// The part of it that group G's values make.
template <int G>
__device__ __forceinline__ void issue_ts_group(uint32_t d, uint32_t a, uint64_t b_desc_mn, uint32_t idesc, bool accumulate) {
  tc::product_ts<GC / 16>(d, a + G * GC, b_desc_mn + (uint32_t)(G * GC * 128 >> 4), idesc, accumulate ? 1u : 0u);
}

// GC accumulator columns of this thread's row -> 16-bit values in global memory
template <bool IS_BF16>
__device__ __forceinline__ void store_cols(uint32_t taddr, unsigned char* dst, float mult, bool live, bool wide) {
#pragma unroll
  for (int c = 0; c < GC / 32; ++c) {
    uint32_t acc[32];
    tc::tmem_ld32(taddr + c * 32, acc);
    tc::tmem_wait_ld();
    if (live) tc::store_row32<IS_BF16>(dst + c * 64, acc, mult, wide);
  }
}

// ------------------------------------------------------------------------------ dK, dV
// TMEM columns: [0,128) S^T then P^T, [128,256) dP^T then dS^T, [256,384) dV, [384,512) dK.
template <bool IS_BF16>
__global__ void __launch_bounds__(kDkvThreads, 1)
    fa_bwd_dkv_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                      const BwdParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* k_smem = smem;
  unsigned char* v_smem = smem + kTileBytes;
  unsigned char* q_smem = smem + 2 * kTileBytes;   // kStages tiles
  unsigned char* do_smem = smem + 4 * kTileBytes;  // kStages tiles

  __shared__ __align__(16) uint4 next_answer[2];
  __shared__ __align__(8) uint64_t next_wanted, next_full[2], next_taken[2], kv_full, kv_empty, q_full[kStages], q_empty[kStages],
      do_full[kStages], do_empty[kStages], s_full, dp_full, p_full[NG], ds_full, ds_read, acc_done, acc_empty, drained;
  // of a query tile: -lse in log2 units (-inf past the end: P = 0) and -delta
  __shared__ __align__(16) float nlse_s[kStages][BM], ndelta_s[kStages][BM];
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int failed;

  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0);  // known uniform to the compiler
  const int lane = threadIdx.x & 31;

  const int n_kv_tiles = (p.Sk + BN - 1) / BN;
  const int n_q_tiles = (p.Sq + BM - 1) / BM;
  const int hide = hidden_tiles(p.causal, p.Sq, p.Sk, n_kv_tiles);
  const bool keep_ds = p.ds != nullptr;
  const int diag = p.Sk - p.Sq;  // key j is visible to query i when j <= i + diag
  // a work item: a key tile of a (batch, head) and the query tiles that see it
  struct Item {
    int kt0, i0, n_it, bh, b, h, kv_tile;
    unsigned char* ds_head;
  };
  auto item_of = [&](int index) {
    Item w;
    cta_order(index, n_kv_tiles, p.n_bh, p.head_group, &w.kv_tile, &w.bh);  // early key tiles see the most queries
    w.ds_head = p.ds + (long long)w.bh * p.tiles_per_head * kTileBytes;
    w.bh += p.bh0;
    w.b = w.bh / p.H;
    w.h = w.bh % p.H;
    w.kt0 = w.kv_tile * BN;
    w.i0 = 0;
    if (p.causal) {
      const int first = w.kt0 - diag;  // first query that sees the first key of the tile
      w.i0 = first > 0 ? first / BM : 0;
    }
    w.n_it = n_q_tiles > w.i0 ? n_q_tiles - w.i0 : 0;  // (a key tile that no query sees is no item of any role's)
    return w;
  };

  if (threadIdx.x == 0) {
    mbar_init(&next_wanted, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&next_full[s], 1);
      mbar_init(&next_taken[s], 2 + kWorkers / 32 + 4);  // producer, issuer, element-wise and storing warps
    }
    mbar_init(&kv_full, 1);
    mbar_init(&kv_empty, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&q_full[s], 2);  // the copy and the statistics
      mbar_init(&q_empty[s], 1);
      mbar_init(&do_full[s], 1);
      mbar_init(&do_empty[s], 1);
    }
    mbar_init(&s_full, 1);
    mbar_init(&dp_full, 1);
    for (int g = 0; g < NG; ++g) mbar_init(&p_full[g], 4);
    mbar_init(&ds_full, kWorkers / 32);
    mbar_init(&ds_read, 4);
    mbar_init(&acc_done, 1);
    mbar_init(&acc_empty, kWorkers / 32);
    mbar_init(&drained, 1);
    failed = 0;
    mbar_init_fence();
  }
  if (warp == 1) tc::tmem_alloc(&tmem_base_slot, kTmemCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;

  // The item after item n of this block: answer n of the scheduler warp.  Taken by a whole warp.
  auto take_next = [&](int n, bool& ok) {
    ok = ok && __all_sync(kFull, mbar_wait(&next_full[n & 1], (n >> 1) & 1, &failed));
    if (!ok) return -1;
    const int index = __shfl_sync(kFull, tc::next_block(&next_answer[n & 1]), 0);
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(&next_taken[n & 1]);
    return index;
  };

  int kv_loads = 0, q_loads = 0, do_loads = 0;  // producer: items and query tiles it has asked for
  int asked = 0;                                // scheduler: the same
  if (warp < 4) tc::regs_dec<kRegsIssue>();
  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    bool ok = true;
    int step = 0;  // query tiles asked for, over all items
    for (int n = 0, index = blockIdx.x; index >= 0 && ok; ++n) {
      const Item w = item_of(index);
      if (w.n_it > 0) {
        if (kv_loads > 0) ok = __all_sync(kFull, mbar_wait(&kv_empty, (kv_loads - 1) & 1, &failed));
        if (!ok) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&kv_full, 2 * kTileBytes);
          load_tile(k_smem, &map_k, &kv_full, w.kt0, w.h, w.b);
          load_tile(v_smem, &map_v, &kv_full, w.kt0, w.h, w.b);
        }
        ++kv_loads;
      }
      // the statistics of a tile are read a tile ahead, so that nothing waits for that read
      float lse_r[4], delta_r[4];
      auto read_stats = [&](int qt0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int qi = qt0 + e * 32 + lane;
          const long long at = (long long)w.bh * p.Sq + qi;
          lse_r[e] = qi < p.Sq ? p.lse[at] * -kLog2e : -INFINITY;
          delta_r[e] = qi < p.Sq ? -p.delta[at] : 0.f;
        }
      };
      read_stats(w.i0 * BM);
      for (int it = 0; it < w.n_it && ok; ++it, ++step) {
        const int s = step % kStages, u = step / kStages;
        const int qt0 = (w.i0 + it) * BM;
        if (u > 0) ok = __all_sync(kFull, mbar_wait(&q_empty[s], (u - 1) & 1, &failed));
        if (!ok) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&q_full[s], kTileBytes);
          load_tile(q_smem + (size_t)s * kTileBytes, &map_q, &q_full[s], qt0, w.h, w.b);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          nlse_s[s][e * 32 + lane] = lse_r[e];
          ndelta_s[s][e * 32 + lane] = delta_r[e];
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&q_full[s]);
        q_loads = step + 1;
        if (it + 1 < w.n_it) read_stats(qt0 + BM);
        if (u > 0) ok = __all_sync(kFull, mbar_wait(&do_empty[s], (u - 1) & 1, &failed));
        if (!ok) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&do_full[s], kTileBytes);
          load_tile(do_smem + (size_t)s * kTileBytes, &map_do, &do_full[s], qt0, w.h, w.b);
        }
        do_loads = step + 1;
      }
      if (lane == 0) tc::mbar_arrive(&next_wanted);
      index = take_next(n, ok);
    }
    if (!ok && lane == 0) failed = 1;
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    constexpr uint32_t idesc_kk = tc::instr_desc(128, 128, IS_BF16 ? 1 : 0, 0, 0);
    constexpr uint32_t idesc_mn = tc::instr_desc(128, 128, IS_BF16 ? 1 : 0, 0, 1);
    const uint64_t k_desc = tc::smem_desc(smem_u32(k_smem), 16, 1024);
    const uint64_t v_desc = tc::smem_desc(smem_u32(v_smem), 16, 1024);
    const uint64_t q_desc = tc::smem_desc(smem_u32(q_smem), 16, 1024);
    const uint64_t do_desc = tc::smem_desc(smem_u32(do_smem), 16, 1024);
    const uint64_t q_desc_mn = tc::smem_desc(smem_u32(q_smem), kHalfBytes, 1024);
    const uint64_t do_desc_mn = tc::smem_desc(smem_u32(do_smem), kHalfBytes, 1024);
    constexpr uint32_t kStep = kTileBytes >> 4;  // one stage further, in descriptor units
    const uint32_t tmem = __shfl_sync(kFull, tmem_base, 0);
    const uint32_t t_s = tmem + kColS, t_dp = tmem + kColDP;
    const uint32_t t_dv = tmem + kColAcc0, t_dk = tmem + kColAcc1;
    auto wait = [&](uint64_t* bar, int parity) {
      const bool up = __all_sync(kFull, mbar_wait(bar, parity, &failed));
      tc::fence_after_sync();
      return up;
    };
    bool ok = true;
    int step = 0, items = 0;  // query tiles and items worked on so far
    for (int n = 0, index = blockIdx.x; index >= 0 && ok; ++n) {
      const Item w = item_of(index);
      // S^T = K Q^T and dP^T = V dO^T of query tile `at` (over all items); the last of an item free K and V
      auto scores = [&](int at) {
        const int s = at & 1;
        if (!wait(&q_full[s], (at >> 1) & 1)) return false;
        // (the tensor core runs its MMAs in order: P^T of the tile before has been consumed when this one starts)
        issue_ss(t_s, k_desc, q_desc + s * kStep, idesc_kk);
        tc::commit_elected(&s_full);
        return true;
      };
      auto score_gradients = [&](int at, bool last) {
        const int s = at & 1;
        if (!wait(&do_full[s], (at >> 1) & 1) || (keep_ds && at > 0 && !wait(&ds_read, (at - 1) & 1))) return false;
        issue_ss(t_dp, v_desc, do_desc + s * kStep, idesc_kk);
        tc::commit_elected(&dp_full);
        if (last) tc::commit_elected(&kv_empty);
        return true;
      };
      if (w.n_it > 0) {
        ok = wait(&kv_full, items & 1) && scores(step) && score_gradients(step, w.n_it == 1);
        for (int it = 0; it < w.n_it && ok; ++it, ++step) {
          const int s = step & 1;
          const bool next = it + 1 < w.n_it;
          // dV += P^T dO in two parts: of the two groups, which share the ex2 unit, one is ahead; the first product
          // of an item waits until the results of the one before have left the accumulators
          ok = (it > 0 || items == 0 || wait(&acc_empty, (items - 1) & 1)) && wait(&p_full[0], step & 1);
          if (!ok) break;
          issue_ts_group<0>(t_dv, t_s, do_desc_mn + s * kStep, idesc_mn, it > 0);
          ok = wait(&p_full[1], step & 1);
          if (!ok) break;
          issue_ts_group<1>(t_dv, t_s, do_desc_mn + s * kStep, idesc_mn, true);
          tc::commit_elected(&do_empty[s]);
          if (next) ok = scores(step + 1);
          ok = ok && wait(&ds_full, step & 1);
          if (!ok) break;
          issue_ts(t_dk, t_dp, q_desc_mn + s * kStep, idesc_mn, it > 0);  // dK += dS^T Q
          tc::commit_elected(&q_empty[s]);
          if (next) ok = score_gradients(step + 1, it + 2 == w.n_it);
        }
        if (ok) tc::commit_elected(&acc_done);
        ++items;
      }
      index = take_next(n, ok);
    }
    if (!ok && lane == 0) failed = 1;
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ scheduler
    // Asked for when the last copies of an item are under way, two steps before its end: soon enough for its K
    // and V, and not before - a block that asked at the start of a long item would keep a pending one from
    // those that finish first (2 x 16 heads of 583 causal keys 41.5 us so).
    bool ok = true;
    for (int n = 0; ok; ++n) {
      ok = __all_sync(kFull, mbar_wait(&next_wanted, n & 1, &failed));
      if (ok && n > 0) ok = __all_sync(kFull, mbar_wait(&next_taken[(n - 1) & 1], ((n - 1) >> 1) & 1, &failed));
      if (!ok) break;
      if (lane == 0) tc::request_next_block(&next_answer[n & 1], &next_full[n & 1]);
      asked = n + 1;
      ok = __all_sync(kFull, mbar_wait(&next_full[n & 1], (n >> 1) & 1, &failed));
      if (!ok || __shfl_sync(kFull, tc::next_block(&next_answer[n & 1]), 0) < 0) break;
    }
    if (!ok && lane == 0) failed = 1;
  } else if (warp >= 4 + 4 * NG) {
    tc::regs_dec<kRegsStore>();
    // ------------------------------------------------------------------ dS to memory
    // Warps of their own read the 16-bit dS^T once more from tensor memory: the element-wise warps
    // are what a step waits for, and shared memory, by way of which a bulk copy would go, is the
    // products' (see the head of this file).
    const int quad = warp & 3;
    const uint32_t dp_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + kColDP;
    bool ok = true;
    int step = 0;
    for (int n = 0, index = blockIdx.x; index >= 0 && ok; ++n) {
      const Item w = item_of(index);
      for (int it = 0; it < w.n_it && keep_ds; ++it, ++step) {
        ok = __all_sync(kFull, mbar_wait(&ds_full, step & 1, &failed));
        if (!ok) break;
        tc::fence_after_sync();
        uint32_t d[NG][GC / 2];
#pragma unroll
        for (int g = 0; g < NG; ++g) tc::tmem_ld32(dp_addr + GC * g, d[g]);
        tc::tmem_wait_ld();
        tc::fence_before_sync();
        warp_arrive(&ds_read, lane);
        uint4* dst = reinterpret_cast<uint4*>(w.ds_head + ds_tile(w.kv_tile, w.i0 + it, n_q_tiles, hide) * kTileBytes) +
                     quad * (BM / 8) * 32 + lane;
#pragma unroll
        for (int u = 0; u < BM / 8; ++u) {
          const uint32_t* v = &d[u * 8 / GC][(u * 4) % (GC / 2)];
          __stcs(dst + u * 32, make_uint4(v[0], v[1], v[2], v[3]));
        }
      }
      index = take_next(n, ok);
    }
    if (!ok) failed = 1;
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ element-wise work
    tc::regs_inc<kRegsWork>();
    const int g = (warp - 4) >> 2;  // group: query columns [GC g, GC g + GC) of a tile
    const int quad = warp & 3;
    const int row = quad * 32 + lane;  // key inside the tile
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t s_addr = lane_addr + kColS + GC * g;
    const uint32_t dp_addr = lane_addr + kColDP + GC * g;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    bool ok = true;
    int step = 0, items = 0;  // query tiles and items so far

    for (int n = 0, index = blockIdx.x; index >= 0 && ok; ++n) {
      const Item w = item_of(index);
      const int kt0 = w.kt0, kj = kt0 + row;
      for (int it = 0; it < w.n_it; ++it, ++step) {
        const int s = step & 1;
        const int qt0 = (w.i0 + it) * BM;
        // the tile's statistics come into registers ahead of its scores: shared memory is busy with
        // the products' operands, and every read of it is slow
        float4 stat[GC / 4];
        bool up = __all_sync(kFull, mbar_wait(&q_full[s], (step >> 1) & 1, &failed));
        if (up) {
#pragma unroll
          for (int e = 0; e < GC / 4; ++e) stat[e] = *reinterpret_cast<const float4*>(&nlse_s[s][GC * g + 4 * e]);
          up = __all_sync(kFull, mbar_wait(&s_full, step & 1, &failed));
        }
        if (!up) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
        // query column e of this group is visible to key kj when qt0 + GC g + e >= kj - diag; a row
        // past the last key has no gradients of its own, but its dS would meet zeros of K in dQ
        // (and need not be finite)
        const bool edge = (kt0 + BN > p.Sk) || (p.causal && (kt0 + BN - 1 > qt0 + diag));
        const int lo = !edge ? 0 : kj >= p.Sk ? GC : p.causal ? kj - diag - (qt0 + GC * g) : 0;
        uint32_t raw[GC];
#pragma unroll
        for (int c = 0; c < GC / 32; ++c) tc::tmem_ld32(s_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&raw[c * 32]));
        tc::tmem_wait_ld();
        float2 pr[GC / 2];
#pragma unroll
        for (int c = 0; c < GC / 32; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const float4 l4 = stat[c * 8 + e / 4];
            const float2 l2[2] = {make_float2(l4.x, l4.y), make_float2(l4.z, l4.w)};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int at = c * 32 + e + 2 * u;
              const float2 a = fma2(make_float2(__uint_as_float(raw[at]), __uint_as_float(raw[at + 1])), sc2, l2[u]);
              float2 x = make_float2(fast_exp2(a.x), fast_exp2(a.y));
              if (edge) {
                if (at < lo) x.x = 0.f;
                if (at + 1 < lo) x.y = 0.f;
              }
              pr[at / 2] = x;
              pk[e / 2 + u] = pack_pair(x.x, x.y, IS_BF16);
            }
          }
          // all of this group's S columns are in registers: P^T goes over their first half
          tc::tmem_st16(s_addr + c * 16, pk);
        }
        tc::tmem_wait_st();
        tc::fence_before_sync();
        warp_arrive(&p_full[g], lane);
#pragma unroll
        for (int e = 0; e < GC / 4; ++e) stat[e] = *reinterpret_cast<const float4*>(&ndelta_s[s][GC * g + 4 * e]);

        if (!__all_sync(kFull, mbar_wait(&dp_full, step & 1, &failed))) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
#pragma unroll
        for (int c = 0; c < GC / 32; ++c) tc::tmem_ld32(dp_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&raw[c * 32]));
        tc::tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < GC / 32; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const float4 d4 = stat[c * 8 + e / 4];
            const float2 d2[2] = {make_float2(d4.x, d4.y), make_float2(d4.z, d4.w)};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int at = c * 32 + e + 2 * u;
              const float2 x = mul2(pr[at / 2], add2(make_float2(__uint_as_float(raw[at]), __uint_as_float(raw[at + 1])), d2[u]));
              pk[e / 2 + u] = pack_pair(x.x, x.y, IS_BF16);
            }
          }
          tc::tmem_st16(dp_addr + c * 16, pk);
        }
        tc::tmem_wait_st();
        tc::fence_before_sync();
        warp_arrive(&ds_full, lane);
      }

      if (ok && w.n_it > 0) ok = mbar_wait(&acc_done, items & 1, &failed);
      ok = __all_sync(kFull, ok);
      if (ok) {
        tc::fence_after_sync();
        const bool live = kj < p.Sk;
        unsigned char* dv_row = reinterpret_cast<unsigned char*>(p.dv.ptr) +
                                2 * ((long long)w.b * p.dv.sb + (long long)w.h * p.dv.sh + (long long)kj * p.dv.ss) +
                                2 * GC * g;
        unsigned char* dk_row = reinterpret_cast<unsigned char*>(p.dk.ptr) +
                                2 * ((long long)w.b * p.dk.sb + (long long)w.h * p.dk.sh + (long long)kj * p.dk.ss) +
                                2 * GC * g;
        if (w.n_it > 0) {
          store_cols<IS_BF16>(lane_addr + kColAcc0 + GC * g, dv_row, 1.f, live, p.dv.wide);
          store_cols<IS_BF16>(lane_addr + kColAcc1 + GC * g, dk_row, p.scale, live, p.dk.wide);
          tc::fence_before_sync();
          warp_arrive(&acc_empty, lane);
          ++items;
        } else if (live) {
          // no query sees this key tile: the gradients are zero
          const uint4 z = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
          for (int e = 0; e < GC / 8; ++e) {
            reinterpret_cast<uint4*>(dv_row)[e] = z;
            reinterpret_cast<uint4*>(dk_row)[e] = z;
          }
        }
      }
      index = take_next(n, ok);
    }
    if (!ok) failed = 1;
  }

  tc::fence_before_sync();
  __syncthreads();
  if (failed) {  // (uniform: nobody writes it any more)
    // a role gave up: what the others have under way has to end before the block does
    if (threadIdx.x == 0) {
      tc::await_copies<1>(&kv_full, kv_loads);
      tc::await_copies<kStages>(q_full, q_loads);
      tc::await_copies<kStages>(do_full, do_loads);
    }
    if (warp == 1) tc::await_products(&drained);
    if (warp == 2 && lane == 0) tc::await_copies<2>(next_full, asked);
    __syncthreads();
  }
  if (threadIdx.x == 0 && failed && p.status != nullptr) atomicExch(p.status, 1);
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------------------ dQ
// TMEM columns: [0,128) S, [128,256) dP then dS (group g's GC values as GC / 2 columns at
// 128 + GC g), [256,384) dQ.
template <bool IS_BF16>
__global__ void __launch_bounds__(kThreads, 1)
    fa_bwd_dq_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                     const BwdParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* q_smem = smem;
  unsigned char* do_smem = smem + kTileBytes;
  unsigned char* k_smem = smem + 2 * kTileBytes;  // kStages tiles
  unsigned char* v_smem = smem + 4 * kTileBytes;  // kStages tiles

  __shared__ __align__(8) uint64_t qdo_full, k_full[kStages], k_empty[kStages], v_full[kStages],
      v_empty[kStages], s_full, dp_full, s_read, ds_full, acc_done, drained;
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int failed;

  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0);  // known uniform to the compiler
  const int lane = threadIdx.x & 31;

  const int n_q_tiles = (p.Sq + BM - 1) / BM;
  int slot, bh;
  cta_order((int)blockIdx.x, n_q_tiles, p.n_bh, p.head_group, &slot, &bh);
  const int q_tile = n_q_tiles - 1 - slot;  // late query tiles see the most keys: first
  const int b = bh / p.H, h = bh % p.H;
  const int qt0 = q_tile * BM;
  const int diag = p.Sk - p.Sq;
  int kv_end = p.Sk;
  if (p.causal) {
    const int lim = qt0 + BM + diag;
    kv_end = lim < p.Sk ? lim : p.Sk;
  }
  const int n_kv = (kv_end + BN - 1) / BN;

  if (threadIdx.x == 0) {
    mbar_init(&qdo_full, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    mbar_init(&s_full, 1);
    mbar_init(&dp_full, 1);
    mbar_init(&s_read, kWorkers / 32);
    mbar_init(&ds_full, kWorkers / 32);
    mbar_init(&acc_done, 1);
    mbar_init(&drained, 1);
    failed = 0;
    mbar_init_fence();
  }
  if (warp == 1) tc::tmem_alloc(&tmem_base_slot, kTmemCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;

  int k_loads = 0, v_loads = 0;  // producer: key and value tiles it has asked for
  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      bool ok = true;
      mbar_arrive_expect_tx(&qdo_full, 2 * kTileBytes);
      load_tile(q_smem, &map_q, &qdo_full, qt0, h, b);
      load_tile(do_smem, &map_do, &qdo_full, qt0, h, b);
      for (int j = 0; j < n_kv && ok; ++j) {
        const int s = j % kStages, n = j / kStages;
        if (n > 0) ok = mbar_wait(&k_empty[s], (n - 1) & 1, &failed);
        if (!ok) break;
        mbar_arrive_expect_tx(&k_full[s], kTileBytes);
        load_tile(k_smem + (size_t)s * kTileBytes, &map_k, &k_full[s], j * BN, h, b);
        k_loads = j + 1;
        if (n > 0) ok = mbar_wait(&v_empty[s], (n - 1) & 1, &failed);
        if (!ok) break;
        mbar_arrive_expect_tx(&v_full[s], kTileBytes);
        load_tile(v_smem + (size_t)s * kTileBytes, &map_v, &v_full[s], j * BN, h, b);
        v_loads = j + 1;
      }
      if (!ok) failed = 1;
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    {
      constexpr uint32_t idesc_kk = tc::instr_desc(128, 128, IS_BF16 ? 1 : 0, 0, 0);
      constexpr uint32_t idesc_mn = tc::instr_desc(128, 128, IS_BF16 ? 1 : 0, 0, 1);
      const uint64_t q_desc = tc::smem_desc(smem_u32(q_smem), 16, 1024);
      const uint64_t do_desc = tc::smem_desc(smem_u32(do_smem), 16, 1024);
      const uint64_t k_desc = tc::smem_desc(smem_u32(k_smem), 16, 1024);
      const uint64_t v_desc = tc::smem_desc(smem_u32(v_smem), 16, 1024);
      const uint64_t k_desc_mn = tc::smem_desc(smem_u32(k_smem), kHalfBytes, 1024);
      constexpr uint32_t kStep = kTileBytes >> 4;  // one stage further, in descriptor units
      const uint32_t tmem = __shfl_sync(kFull, tmem_base, 0);
      const uint32_t t_s = tmem + kColS, t_dp = tmem + kColDP, t_dq = tmem + kColAcc0;
      bool ok = __all_sync(kFull, mbar_wait(&qdo_full, 0, &failed));
      ok = ok && __all_sync(kFull, mbar_wait(&k_full[0], 0, &failed));
      ok = ok && __all_sync(kFull, mbar_wait(&v_full[0], 0, &failed));
      if (ok) {
        tc::fence_after_sync();
        issue_ss(t_s, q_desc, k_desc, idesc_kk);  // S = Q K^T
        tc::commit_elected(&s_full);
        issue_ss(t_dp, do_desc, v_desc, idesc_kk);  // dP = dO V^T
        tc::commit_elected(&dp_full);
        tc::commit_elected(&v_empty[0]);
      }
      for (int j = 0; j < n_kv && ok; ++j) {
        const int s = j & 1, s1 = (j + 1) & 1, n1 = (j + 1) >> 1;
        const bool next = j + 1 < n_kv;
        if (next) {
          // S(j) is in registers of the element-wise warps: its columns can take S(j+1)
          ok = __all_sync(kFull, mbar_wait(&s_read, j & 1, &failed));
          ok = ok && __all_sync(kFull, mbar_wait(&k_full[s1], n1 & 1, &failed));
          if (!ok) break;
          tc::fence_after_sync();
          issue_ss(t_s, q_desc, k_desc + s1 * kStep, idesc_kk);
          tc::commit_elected(&s_full);
        }
        ok = __all_sync(kFull, mbar_wait(&ds_full, j & 1, &failed));
        if (!ok) break;
        tc::fence_after_sync();
        issue_ts(t_dq, t_dp, k_desc_mn + s * kStep, idesc_mn, j > 0);  // dQ += dS K
        tc::commit_elected(&k_empty[s]);
        if (next) {
          ok = __all_sync(kFull, mbar_wait(&v_full[s1], n1 & 1, &failed));
          if (!ok) break;
          tc::fence_after_sync();
          issue_ss(t_dp, do_desc, v_desc + s1 * kStep, idesc_kk);  // after dQ(j): dS(j) has been consumed
          tc::commit_elected(&dp_full);
          tc::commit_elected(&v_empty[s1]);
        }
      }
      if (ok) tc::commit_elected(&acc_done);
      if (!ok && lane == 0) failed = 1;
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ element-wise work
    const int g = (warp - 2) >> 2;  // group: key columns [GC g, GC g + GC) of a tile
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const int qi = qt0 + row;
    const bool live = qi < p.Sq;
    const long long stat_at = (long long)bh * p.Sq + qi;
    const float lse2 = live ? p.lse[stat_at] * kLog2e : INFINITY;
    const float dl = live ? p.delta[stat_at] : 0.f;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t s_addr = lane_addr + kColS + GC * g;
    const uint32_t dp_addr = lane_addr + kColDP + GC * g;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    const float2 nl2 = make_float2(-lse2, -lse2);
    bool ok = true;

    for (int j = 0; j < n_kv; ++j) {
      if (!__all_sync(kFull, mbar_wait(&s_full, j & 1, &failed))) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
      uint32_t raw[GC];
#pragma unroll
      for (int c = 0; c < GC / 32; ++c) tc::tmem_ld32(s_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&raw[c * 32]));
      tc::tmem_wait_ld();
      tc::fence_before_sync();
      warp_arrive(&s_read, lane);
      const int col0 = j * BN + GC * g;
      const bool edge = (j * BN + BN > p.Sk) || (p.causal && (j * BN + BN - 1 > qt0 + diag));
      int lim = GC - 1;  // last visible key of this row, relative to this group's columns
      if (edge) {
        int last = p.Sk - 1;
        if (p.causal && qi + diag < last) last = qi + diag;
        lim = last - col0;
      }
      float pr[GC];
#pragma unroll
      for (int e = 0; e < GC; e += 2) {
        const float2 a = fma2(make_float2(__uint_as_float(raw[e]), __uint_as_float(raw[e + 1])), sc2, nl2);
        pr[e] = fast_exp2(a.x);
        pr[e + 1] = fast_exp2(a.y);
        if (edge) {
          if (e > lim) pr[e] = 0.f;
          if (e + 1 > lim) pr[e + 1] = 0.f;
        }
      }
      if (!__all_sync(kFull, mbar_wait(&dp_full, j & 1, &failed))) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
#pragma unroll
      for (int c = 0; c < GC / 32; ++c) {
        uint32_t d[32];
        tc::tmem_ld32(dp_addr + c * 32, d);
        tc::tmem_wait_ld();
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const float x0 = pr[c * 32 + e] * (__uint_as_float(d[e]) - dl);
          const float x1 = pr[c * 32 + e + 1] * (__uint_as_float(d[e + 1]) - dl);
          pk[e / 2] = pack_pair(x0, x1, IS_BF16);
        }
        tc::tmem_st16(dp_addr + c * 16, pk);
      }
      tc::tmem_wait_st();
      tc::fence_before_sync();
      warp_arrive(&ds_full, lane);
    }

    if (ok) ok = mbar_wait(&acc_done, 0, &failed);
    ok = __all_sync(kFull, ok);
    if (ok) {
      tc::fence_after_sync();
      unsigned char* dq_row = reinterpret_cast<unsigned char*>(p.dq.ptr) +
                              2 * ((long long)b * p.dq.sb + (long long)h * p.dq.sh + (long long)qi * p.dq.ss) +
                              2 * GC * g;
      store_cols<IS_BF16>(lane_addr + kColAcc0 + GC * g, dq_row, p.scale, live, p.dq.wide);
    } else {
      failed = 1;
    }
  }

  tc::fence_before_sync();
  __syncthreads();
  if (failed) {  // (as above)
    if (threadIdx.x == 0) {
      tc::await_copies<1>(&qdo_full, 1);
      tc::await_copies<kStages>(k_full, k_loads);
      tc::await_copies<kStages>(v_full, v_loads);
    }
    if (warp == 1) tc::await_products(&drained);
    __syncthreads();
  }
  if (threadIdx.x == 0 && failed && p.status != nullptr) atomicExch(p.status, 1);
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------ dQ from kept dS
// One CTA owns two query tiles of a head and walks the key tiles they see: dQ += dS K, with the
// tiles of dS^T as the first operand (MN-major, no swizzle) and K in MN-major form.  Bound: the 32 KB
// of dS a product reads; two query tiles share a K tile, which comes from L2.  2.2 GB of dS (4 x 32
// heads of 4096, causal) in 400 us, 5500 GB/s.  Pending items are taken over as in the dK/dV kernel, so that
// dS keeps coming while the results of an item leave: whole calls 8 x 32 heads of 196 61.0 -> 58.0 us, 12 x 32
// of 136 causal 73.3 -> 68.2, 8 x 16 of 1000 226 -> 220, 4 x 32 of 4096 causal 1520 -> 1507.
// TMEM: two sets of 2 x 128 columns, used by the items in turn.
constexpr int kQT = 2;        // query tiles a CTA
constexpr int kDsStages = 4;  // tiles of dS^T in flight
constexpr int kDsThreads = 64 + 128 + 32;  // producer and issuer, results, scheduler
// TAKE: there are more items than SMs.  Where there are not, nothing is pending: without the loop over items
// (TAKE = false) 2 x 8 heads of 2048 causal take 22.7 us in this kernel, with it 23.4.
template <bool IS_BF16, bool TAKE>
__global__ void __launch_bounds__(kDsThreads, 1)
    fa_bwd_dq_ds_kernel(const __grid_constant__ CUtensorMap map_k, const BwdParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* k_smem = smem;                    // kStages tiles
  unsigned char* ds_smem = smem + 2 * kTileBytes;  // kDsStages tiles

  __shared__ __align__(16) uint4 next_answer[2];
  __shared__ __align__(8) uint64_t next_wanted, next_full[2], next_taken[2], k_full[kStages], k_empty[kStages],
      ds_full[kDsStages], ds_empty[kDsStages], acc_full[2], acc_empty[2], drained;
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int failed;

  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0);  // known uniform to the compiler
  const int lane = threadIdx.x & 31;

  const int n_q_tiles = (p.Sq + BM - 1) / BM;
  const int n_kv_tiles = (p.Sk + BN - 1) / BN;
  const int n_slots = (n_q_tiles + kQT - 1) / kQT;
  const int hide = hidden_tiles(p.causal, p.Sq, p.Sk, n_kv_tiles);
  struct Item {
    int first, tiles;  // query tiles
    int n_kv0, n_kv;   // key tiles that the first query tile sees, and that either sees
    int b, h;
    const unsigned char* ds_head;
  };
  auto item_of = [&](int index) {
    Item w;
    int slot, bh;
    cta_order(index, n_slots, p.n_bh, p.head_group, &slot, &bh);
    bh = p.n_bh - 1 - bh;  // the last heads first: some of their dS is still in L2
    w.first = (n_slots - 1 - slot) * kQT;  // late query tiles see the most keys: first
    w.tiles = min(kQT, n_q_tiles - w.first);
    w.ds_head = p.ds + (long long)bh * p.tiles_per_head * kTileBytes;
    bh += p.bh0;
    w.b = bh / p.H;
    w.h = bh % p.H;
    w.n_kv0 = p.causal ? min(n_kv_tiles, w.first + hide + 1) : n_kv_tiles;
    w.n_kv = p.causal ? min(n_kv_tiles, w.first + w.tiles + hide) : n_kv_tiles;
    return w;
  };

  if (threadIdx.x == 0) {
    mbar_init(&next_wanted, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&next_full[s], 1);
      mbar_init(&next_taken[s], 2 + 4);  // producer, issuer and the warps of the results
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 4);
    }
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < kDsStages; ++s) {
      mbar_init(&ds_full[s], 1);
      mbar_init(&ds_empty[s], 1);
    }
    mbar_init(&drained, 1);
    failed = 0;
    mbar_init_fence();
  }
  if (warp == 1) tc::tmem_alloc(&tmem_base_slot, (TAKE ? 2 : 1) * kQT * 128);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;

  // The item after item n of this block: answer n of the scheduler warp.  Taken by a whole warp.
  auto take_next = [&](int n, bool& ok) {
    if (!TAKE) return -1;
    ok = ok && __all_sync(kFull, mbar_wait(&next_full[n & 1], (n >> 1) & 1, &failed));
    if (!ok) return -1;
    const int index = __shfl_sync(kFull, tc::next_block(&next_answer[n & 1]), 0);
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(&next_taken[n & 1]);
    return index;
  };

  int k_loads = 0, ds_loads = 0;  // producer: key and dS tiles it has asked for
  int asked = 0;                  // scheduler: the same
  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    bool ok = true;
    for (int i = 0, index = blockIdx.x; (TAKE ? index >= 0 : i == 0) && ok; ++i) {
      const Item w = item_of(index);
      int mine = 1;
      if (lane == 0) {
        bool good = true;
        for (int j = 0; j < w.n_kv && good; ++j) {
          const int s = k_loads & 1, n = k_loads >> 1;
          if (n > 0) good = mbar_wait(&k_empty[s], (n - 1) & 1, &failed);
          if (!good) break;
          mbar_arrive_expect_tx(&k_full[s], kTileBytes);
          load_tile(k_smem + (size_t)s * kTileBytes, &map_k, &k_full[s], j * BN, w.h, w.b);
          ++k_loads;
          if (TAKE && j + 1 == w.n_kv) tc::mbar_arrive(&next_wanted);
          const unsigned char* tile = w.ds_head + ds_tile(j, w.first, n_q_tiles, hide) * kTileBytes;
          for (int t = j < w.n_kv0 ? 0 : 1; t < w.tiles; ++t, ++ds_loads) {
            const int u = ds_loads & (kDsStages - 1), m = ds_loads / kDsStages;
            if (m > 0) good = mbar_wait(&ds_empty[u], (m - 1) & 1, &failed);
            if (!good) break;
            mbar_arrive_expect_tx(&ds_full[u], kTileBytes);
            bulk_g2s(ds_smem + u * kTileBytes, tile + t * kTileBytes, kTileBytes, &ds_full[u]);
          }
        }
        mine = good ? 1 : 0;
      }
      ok = __shfl_sync(kFull, mine, 0) != 0;
      index = take_next(i, ok);
    }
    if (!ok && lane == 0) failed = 1;
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    constexpr uint32_t idesc = tc::instr_desc(128, 128, IS_BF16 ? 1 : 0, 1, 1);
    const uint64_t k_desc = tc::smem_desc(smem_u32(k_smem), kHalfBytes, 1024);
    // 8 keys to the next 8: 128 bytes; 8 queries to the next 8: 32 pieces
    const uint64_t ds_desc = tc::smem_desc_plain(smem_u32(ds_smem), 128, 32 * 16);
    constexpr uint32_t kStep = kTileBytes >> 4;
    const uint32_t tmem = __shfl_sync(kFull, tmem_base, 0);
    bool ok = true;
    int m = 0, n = 0;  // tiles of K and of dS consumed
    for (int i = 0, index = blockIdx.x; (TAKE ? index >= 0 : i == 0) && ok; ++i) {
      const Item w = item_of(index);
      // items use the two sets of accumulators in turn: the results of one leave under the products of the next
      const uint32_t acc = tmem + (i & 1) * (kQT * 128);
      if (i > 1) ok = __all_sync(kFull, mbar_wait(&acc_empty[i & 1], ((i >> 1) - 1) & 1, &failed));
      tc::fence_after_sync();
      for (int j = 0; j < w.n_kv && ok; ++j, ++m) {
        const int s = m & 1;
        ok = __all_sync(kFull, mbar_wait(&k_full[s], (m >> 1) & 1, &failed));
        for (int t = j < w.n_kv0 ? 0 : 1; t < w.tiles && ok; ++t, ++n) {
          const int u = n & (kDsStages - 1);
          ok = __all_sync(kFull, mbar_wait(&ds_full[u], (n / kDsStages) & 1, &failed));
          if (!ok) break;
          tc::fence_after_sync();
          // 16 keys a step: 256 bytes inside 32 keys of a dS tile, 16 rows (2048 bytes) of K
#pragma unroll
          for (int kq = 0; kq < 4; ++kq)
            tc::product_ss_steps<2, 256, 2048>(acc + 128 * t, ds_desc + u * kStep + kq * (kTileBytes / 4 >> 4),
                                               k_desc + s * kStep + kq * (2 * 2048 >> 4), idesc, j > 0 || kq > 0 ? 1u : 0u);
          tc::commit_elected(&ds_empty[u]);
        }
        if (ok) tc::commit_elected(&k_empty[s]);
      }
      if (ok) tc::commit_elected(&acc_full[i & 1]);
      index = take_next(i, ok);
    }
    if (!ok && lane == 0) failed = 1;
    __syncwarp();
  } else if (warp == 6) {
    // ------------------------------------------------------------------ scheduler (as in the dK/dV kernel)
    bool ok = true;
    for (int n = 0; ok && TAKE; ++n) {
      ok = __all_sync(kFull, mbar_wait(&next_wanted, n & 1, &failed));
      if (ok && n > 0) ok = __all_sync(kFull, mbar_wait(&next_taken[(n - 1) & 1], ((n - 1) >> 1) & 1, &failed));
      if (!ok) break;
      if (lane == 0) tc::request_next_block(&next_answer[n & 1], &next_full[n & 1]);
      asked = n + 1;
      ok = __all_sync(kFull, mbar_wait(&next_full[n & 1], (n >> 1) & 1, &failed));
      if (!ok || __shfl_sync(kFull, tc::next_block(&next_answer[n & 1]), 0) < 0) break;
    }
    if (!ok && lane == 0) failed = 1;
  } else {
    // ------------------------------------------------------------------ results
    const int quad = warp & 3;
    bool ok = true;
    for (int i = 0, index = blockIdx.x; (TAKE ? index >= 0 : i == 0) && ok; ++i) {
      const Item w = item_of(index);
      ok = __all_sync(kFull, mbar_wait(&acc_full[i & 1], (i >> 1) & 1, &failed));
      if (!ok) break;
      tc::fence_after_sync();
      const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (i & 1) * (kQT * 128);
      for (int t = 0; t < w.tiles; ++t) {
        const int qi = (w.first + t) * BM + quad * 32 + lane;
        unsigned char* dq_row = reinterpret_cast<unsigned char*>(p.dq.ptr) +
                                2 * ((long long)w.b * p.dq.sb + (long long)w.h * p.dq.sh + (long long)qi * p.dq.ss);
#pragma unroll
        for (int g = 0; g < NG; ++g)
          store_cols<IS_BF16>(lane_addr + 128 * t + GC * g, dq_row + 2 * GC * g, p.scale, qi < p.Sq, p.dq.wide);
      }
      tc::fence_before_sync();
      warp_arrive(&acc_empty[i & 1], lane);
      index = take_next(i, ok);
    }
    if (!ok && lane == 0) failed = 1;
  }

  tc::fence_before_sync();
  __syncthreads();
  if (failed) {  // (as above)
    if (threadIdx.x == 0) {
      tc::await_copies<kStages>(k_full, k_loads);
      tc::await_copies<kDsStages>(ds_full, ds_loads);
    }
    if (warp == 1) tc::await_products(&drained);
    if (warp == 6 && lane == 0) tc::await_copies<2>(next_full, asked);
    __syncthreads();
  }
  if (threadIdx.x == 0 && failed && p.status != nullptr) atomicExch(p.status, 1);
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, (TAKE ? 2 : 1) * kQT * 128);
  }
}

// `regs`: the registers a thread that a kernel with a register split has to be launched with, or 0.
template <class K>
int opt_in_smem(K kern, std::atomic<bool>& done, int regs = 0) {
  if (!done.load(std::memory_order_acquire)) {
    if (regs != 0) {
      cudaFuncAttributes at;
      cudaError_t e = cudaFuncGetAttributes(&at, kern);
      if (e != cudaSuccess) return ixb_host::cuda_status(e);
      if (at.numRegs != regs) return IXB_ERR_UNSUPPORTED;
    }
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e != cudaSuccess) return ixb_host::cuda_status(e);
    done.store(true, std::memory_order_release);
  }
  return IXB_OK;
}

// Tiles of dS^T one head has.
long long tiles_of_head(int Sq, int Sk, int causal) {
  const int n_q = (int)((Sq + (long long)BM - 1) / BM), n_kv = (int)((Sk + (long long)BN - 1) / BN);
  return ds_tile(n_kv - 1, n_q - 1, n_q, hidden_tiles(causal, Sq, Sk, n_kv)) + 1;
}

}  // namespace

extern "C" size_t ixb_fa_bwd_scratch_bytes(int32_t B, int32_t H, int32_t Sq, int32_t Sk, int causal, size_t limit) {
  if (B <= 0 || H <= 0 || Sq <= 0 || Sk <= 0 || (causal && Sk < Sq)) return 0;
  const long long n_bh = (long long)B * H, tiles = tiles_of_head(Sq, Sk, causal != 0);
  const long long fit = (long long)(limit / kTileBytes) / tiles;  // heads within the limit
  if (fit <= 0 || tiles > 0x7fffffffLL) return 0;
  const long long launches = (n_bh + fit - 1) / fit;
  return (size_t)((n_bh + launches - 1) / launches * tiles) * kTileBytes;
}

extern "C" int ixb_fa_bwd_scratch(int dtype, const void* q, const void* k, const void* v, const void* o,
                                  const void* dout, const float* lse, void* dq, void* dk, void* dv, float* delta,
                                  void* scratch, size_t scratch_bytes, int32_t B, int32_t H, int32_t Sq, int32_t Sk,
                                  int32_t D, const int64_t* q_strides, const int64_t* k_strides,
                                  const int64_t* v_strides, const int64_t* o_strides, const int64_t* do_strides,
                                  const int64_t* dq_strides, const int64_t* dk_strides, const int64_t* dv_strides,
                                  float scale, int causal, int32_t* status, ixb_stream stream) {
  if (B < 0 || H < 0 || Sq < 0 || Sk < 0) return IXB_ERR_ARG;
  if (B == 0 || H == 0 || Sq == 0 || Sk == 0) return IXB_OK;
  if (!q || !k || !v || !o || !dout || !lse || !dq || !dk || !dv || !delta) return IXB_ERR_ARG;
  if (!ixb_host::aligned16(scratch)) return IXB_ERR_ALIGN;
  if (dtype != IXB_BF16 && dtype != IXB_F16) return IXB_ERR_DTYPE;
  if (D != HD) return IXB_ERR_SHAPE;
  if (causal && Sk < Sq) return IXB_ERR_SHAPE;
  if (!(scale > 0.f)) return IXB_ERR_ARG;
  const void* ptrs[8] = {q, k, v, o, dout, dq, dk, dv};
  const int64_t* strs[8] = {q_strides, k_strides, v_strides, o_strides, do_strides, dq_strides, dk_strides,
                            dv_strides};
  for (int t = 0; t < 8; ++t) {
    if (strs[t] == nullptr) return IXB_ERR_ARG;
    if (!ixb_host::aligned16(ptrs[t])) return IXB_ERR_ALIGN;
    for (int i = 0; i < 3; ++i)
      if (strs[t][i] <= 0 || (strs[t][i] * 2) % 16 != 0) return IXB_ERR_ALIGN;
  }
  const long long n_q_tiles = (Sq + BM - 1) / BM, n_kv_tiles = (Sk + BN - 1) / BN;
  const long long n_bh = (long long)B * H;
  if (n_q_tiles * n_bh > 0x7fffffffLL || n_kv_tiles * n_bh > 0x7fffffffLL) return IXB_ERR_SHAPE;
  const int is_bf16 = dtype == IXB_BF16;
  CUtensorMap mq, mk, mv, mdo;
  if (int st = ixb_host::make_fa_map(&mq, q, is_bf16, B, H, Sq, q_strides[0], q_strides[1], q_strides[2])) return st;
  if (int st = ixb_host::make_fa_map(&mk, k, is_bf16, B, H, Sk, k_strides[0], k_strides[1], k_strides[2])) return st;
  if (int st = ixb_host::make_fa_map(&mv, v, is_bf16, B, H, Sk, v_strides[0], v_strides[1], v_strides[2])) return st;
  if (int st = ixb_host::make_fa_map(&mdo, dout, is_bf16, B, H, Sq, do_strides[0], do_strides[1], do_strides[2]))
    return st;
  BwdParams p;
  p.lse = lse;
  p.delta = delta;
  p.dq = Out{dq, dq_strides[0], dq_strides[1], dq_strides[2], ixb_host::rows_aligned32(dq, dq_strides)};
  p.dk = Out{dk, dk_strides[0], dk_strides[1], dk_strides[2], ixb_host::rows_aligned32(dk, dk_strides)};
  p.dv = Out{dv, dv_strides[0], dv_strides[1], dv_strides[2], ixb_host::rows_aligned32(dv, dv_strides)};
  p.status = status;
  p.B = B;
  p.H = H;
  p.Sq = Sq;
  p.Sk = Sk;
  p.scale = scale;
  p.scale_log2 = scale * kLog2e;
  p.causal = causal ? 1 : 0;
  static const int group_env = [] { const char* e = getenv("IXB_FA_HEAD_GROUP"); return e != nullptr ? atoi(e) : 0; }();
  p.head_group = group_env > 0 ? group_env : (causal ? 8 : 1);

  auto kern_delta = is_bf16 ? fa_bwd_delta_kernel<true> : fa_bwd_delta_kernel<false>;
  auto kern_dkv = is_bf16 ? fa_bwd_dkv_kernel<true> : fa_bwd_dkv_kernel<false>;
  auto kern_dq = is_bf16 ? fa_bwd_dq_kernel<true> : fa_bwd_dq_kernel<false>;
  auto kern_dq_ds = is_bf16 ? fa_bwd_dq_ds_kernel<true, true> : fa_bwd_dq_ds_kernel<false, true>;
  auto kern_dq_ds_one = is_bf16 ? fa_bwd_dq_ds_kernel<true, false> : fa_bwd_dq_ds_kernel<false, false>;
  static std::atomic<bool> configured[4][2][64];
  int devid = 0;
  cudaGetDevice(&devid);
  if (int st = opt_in_smem(kern_dkv, configured[0][is_bf16][devid & 63], kRegsLaunch)) return st;
  if (int st = opt_in_smem(kern_dq, configured[1][is_bf16][devid & 63])) return st;
  if (int st = opt_in_smem(kern_dq_ds, configured[2][is_bf16][devid & 63])) return st;
  if (int st = opt_in_smem(kern_dq_ds_one, configured[3][is_bf16][devid & 63])) return st;

  // The heads go in as many equal launches as the scratch asks for; without room for one head's dS the
  // probabilities are recomputed for dQ.
  const long long tiles = tiles_of_head(Sq, Sk, p.causal);
  const long long fit = scratch != nullptr && tiles <= 0x7fffffffLL ? (long long)(scratch_bytes / kTileBytes) / tiles : 0;
  const long long launches = fit > 0 ? (n_bh + fit - 1) / fit : 1;
  const long long heads = (n_bh + launches - 1) / launches;
  p.ds = fit > 0 ? static_cast<unsigned char*>(scratch) : nullptr;
  p.tiles_per_head = fit > 0 ? (int)tiles : 0;

  const ixb_devinfo* dev = ixb_host::current_device();
  if (dev == nullptr) return IXB_ERR_CUDA;
  const int sms = dev->sm_count;
  cudaStream_t cs = (cudaStream_t)stream;
  const long long rows = n_bh * Sq;
  kern_delta<<<(unsigned)((rows + 15) / 16), 256, 0, cs>>>(
      static_cast<const unsigned char*>(o), static_cast<const unsigned char*>(dout), delta, H, Sq, rows,
      o_strides[0], o_strides[1], o_strides[2], do_strides[0], do_strides[1], do_strides[2]);
  for (long long at = 0; at < n_bh; at += heads) {
    p.bh0 = (int)at;
    p.n_bh = (int)(heads < n_bh - at ? heads : n_bh - at);
    kern_dkv<<<(unsigned)(n_kv_tiles * p.n_bh), kDkvThreads, kSmemBytes, cs>>>(mq, mk, mv, mdo, p);
    const long long slots = (n_q_tiles + kQT - 1) / kQT * p.n_bh;
    if (fit > 0)
      (slots > sms ? kern_dq_ds : kern_dq_ds_one)<<<(unsigned)slots, kDsThreads, kSmemBytes, cs>>>(mk, p);
    else
      kern_dq<<<(unsigned)(n_q_tiles * p.n_bh), kThreads, kSmemBytes, cs>>>(mq, mk, mv, mdo, p);
  }
  return ixb_host::cuda_status(cudaGetLastError());
}

extern "C" int ixb_fa_bwd(int dtype, const void* q, const void* k, const void* v, const void* o,
                          const void* dout, const float* lse, void* dq, void* dk, void* dv, float* delta,
                          int32_t B, int32_t H, int32_t Sq, int32_t Sk, int32_t D, const int64_t* q_strides,
                          const int64_t* k_strides, const int64_t* v_strides, const int64_t* o_strides,
                          const int64_t* do_strides, const int64_t* dq_strides, const int64_t* dk_strides,
                          const int64_t* dv_strides, float scale, int causal, int32_t* status,
                          ixb_stream stream) {
  return ixb_fa_bwd_scratch(dtype, q, k, v, o, dout, lse, dq, dk, dv, delta, nullptr, 0, B, H, Sq, Sk, D, q_strides,
                            k_strides, v_strides, o_strides, do_strides, dq_strides, dk_strides, dv_strides, scale,
                            causal, status, stream);
}
