// Fused attention forward for sm_100a: softmax(Q K^T * scale [+ causal mask]) V with
// tcgen05 tensor-core MMAs, accumulators in tensor memory and operands brought in by TMA.
// It takes the place of the vendor kernel behind torch.ops.npu_graph.npu_fa
// (inductor_x/npu_fusion_attention_graph.py:20-35).
//
// A work item is two 128-row query tiles (A, B) of one (batch, head) with the key/value tiles
// (128 keys each) that they can see.  The grid has one block per item, but a block that has
// finished takes over pending ones (cluster launch control) and keeps its tensor memory,
// barriers and operand rings, so that the loads and the first scores of the next item run
// under the epilogue of the one before it.  Twelve warps:
//   warp 0     TMA producer: Q of the item, K_j / V_j into two-stage rings
//   warp 1     MMA issuer: S_t(j) = Q_t K_j^T into tile t's TMEM buffer, then
//              O_t += P_t(j) V_j with P read straight from TMEM (it overwrites S as 16-bit
//              values).  The two tiles alternate, so the tensor core works on one tile
//              while the other tile's softmax runs.
//   warp 2     scheduler: asks for the next item while this one is worked on (warp 3 idles)
//   warps 4-7  softmax of tile A, warps 8-11 softmax of tile B: thread <-> query row.
//              The row of scores is read once and stays in registers for the maximum and the
//              exponentials; P goes back in two parts, so that the product starts under the
//              last quarter of the exponentials.  The O accumulator is rescaled only when the
//              maximum has grown by more than 2^8 since the last rescale (the final division
//              by the running sum makes a stale reference exact).
// Hand-offs are mbarriers; every wait is bounded and a wait that gives up raises a flag in
// `status`; the CTA exits when the copies and products under way have ended.
//
// TMEM columns: [0,128) S/P of A, [128,256) S/P of B, [256,384) O of A, [384,512) O of B.
//
// Bound: the tensor core.  A step's products of both tiles take it 2048 cycles and the ex2 unit
// needs as many for their exponentials; what is lost beside that is the chain scores -> softmax
// -> P -> product of each tile.  Measured at 8 x 32 heads, 4096 keys, causal, bf16 (one GPU, one
// run): 1138 us with a single lane issuing, the scores read twice from tensor memory and a block
// per item; 963 us with the warp-wide issue, the row in registers and P handed over in two parts
// (at 64 keys instead of 96: 945 against 933 below); 933 us with items taken over by running
// blocks - 966, 1142, 1179 TFLOP/s.  The products alone take 803 us, everything but the
// exponentials 858 us.  16 x 16 heads of 1000 keys, fp16: 177, 156, 138 us; 127 - 133 with whole sectors
// stored and only those columns of an edge tile looked at that some row does not see (512 keys: 52 and
// 50).  An item of eight key tiles takes 29400 cycles there, 2870 a step, of which the tensor core works
// 2048, and 6500 between the last scores of one item and the first of the next: all SMs store and load at
// once.  Built, measured and dropped: O by way of shared memory, a line a store (512 keys 48, but 128
// keys 19.5 against 18.7 and 300 keys 38.3 against 36.3); the next item's first scores behind the
// last product of the first tile (no difference); one, two, three of eight exponentials on the fma pipe
// (1000 keys 130, 131, 134 against 129, 4096 causal keys 973 - 1009, 1020 - 1038, 1093 against 985 - 1006:
// power, not the ex2 unit, is the limit there); a warpgroup of its own for the results (8 x 32 heads of 4096
// causal 941 -> 952, of 16 x 16 of 1000 127 -> 128, small calls up to 8 % slower); the next item asked for at the
// start of items of up to four steps (3 x 32 heads of 459 causal 17.7 -> 20.2), or at once where all items are of one
// length (30 x 32 of 128 34.0 -> 34.3).
#include <atomic>
#include <cmath>
#include "host.h"
#include "fa_maps.h"
#include "ixb/fa_softmax.cuh"

namespace {

using namespace ixb;

using namespace ixb::fa;

constexpr int kStages = 2;  // (the issuer picks stage descriptors with two-way selects)
// Registers: the block starts with kRegsLaunch a thread (all that 12 warps can have); the first
// warpgroup gives up what it does not need so that a softmax thread holds its row of 128 scores.
constexpr int kRegsLaunch = 168, kRegsIssue = 80, kRegsSoftmax = 208;
static_assert(kRegsIssue + NQ * kRegsSoftmax <= (1 + NQ) * kRegsLaunch, "setmaxnreg draws on the block's own registers");
constexpr size_t kSmemBytes = (size_t)kTileBytes * (NQ + 2 * kStages) + 1024;

struct FaParams {
  void* o;
  float* lse;            // [B, H, Sq] natural-log sum of exponentials, may be null
  int* status;           // device word set to 1 if a wait gave up, may be null
  long long o_stride_b, o_stride_h, o_stride_s;  // elements
  int B, H, Sq, Sk;
  float scale_log2;      // softmax scale * log2(e), > 0
  int causal;
  int wide;        // the rows of o are multiples of 32 bytes
  int head_group;  // heads whose CTAs are dispatched together (see the CTA order in the kernel)
};

template <bool IS_BF16>
__global__ void __launch_bounds__(kThreads, 1)
    fa_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                  const __grid_constant__ CUtensorMap map_v, const FaParams p) {
  extern __shared__ unsigned char smem_raw[];
  // operand tiles want 1024-byte alignment for the 128-byte swizzle
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* q_smem = smem;
  unsigned char* k_smem = smem + kTileBytes * NQ;
  unsigned char* v_smem = smem + kTileBytes * (NQ + kStages);

  __shared__ __align__(16) uint4 next_answer[2];
  __shared__ __align__(8) uint64_t q_full, q_empty, next_wanted, next_full[2], next_taken[2], k_full[kStages],
      k_empty[kStages], v_full[kStages], v_empty[kStages], s_full[NQ], p_full[NQ], p_rest[NQ], pv_done[NQ], drained;
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int failed;

  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0);  // known uniform to the compiler
  const int lane = threadIdx.x & 31;

  // Order of the work.  Heads are taken in groups of p.head_group (their K and V stay in L2 while
  // the group runs); inside a group the query blocks go from the last one to the first, all heads
  // of the group at each: under a causal mask the late blocks see the most keys, so the blocks
  // still running when the grid drains are the short ones.
  struct Item {
    int q0, b, h;
    int n_kv_t[NQ];  // key tiles each query tile walks (0 for a tile past the end of the sequence)
    int n_kv;
  };
  const int diag = p.Sk - p.Sq;  // key j is visible to query row i when j <= i + diag
  auto item_of = [&](int index) {
    Item w;
    const int n_q_blocks = (p.Sq + BM * NQ - 1) / (BM * NQ);
    const int per_group = n_q_blocks * p.head_group;
    const int group = index / per_group;
    const int in_group = index - group * per_group;
    const int left = p.B * p.H - group * p.head_group;
    const int g_heads = left < p.head_group ? left : p.head_group;
    const int bh = group * p.head_group + in_group % g_heads;
    w.b = bh / p.H;
    w.h = bh % p.H;
    w.q0 = (n_q_blocks - 1 - in_group / g_heads) * BM * NQ;
    w.n_kv = 0;
#pragma unroll
    for (int t = 0; t < NQ; ++t) {
      const int qt0 = w.q0 + t * BM;
      int kv_end = p.Sk;
      if (p.causal) {
        const int lim = qt0 + BM + diag;
        kv_end = lim < p.Sk ? lim : p.Sk;
      }
      w.n_kv_t[t] = qt0 < p.Sq ? (kv_end + BN - 1) / BN : 0;
      w.n_kv = w.n_kv_t[t] > w.n_kv ? w.n_kv_t[t] : w.n_kv;
    }
    return w;
  };

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    mbar_init(&q_empty, 1);
    mbar_init(&next_wanted, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&next_full[s], 1);
      mbar_init(&next_taken[s], 2 + NQ * 4);  // producer, issuer and the softmax warps
    }
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int t = 0; t < NQ; ++t) {
      mbar_init(&s_full[t], 1);
      mbar_init(&p_full[t], 128);
      mbar_init(&p_rest[t], 128);
      mbar_init(&pv_done[t], 1);
    }
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

  int q_loads = 0, k_loads = 0, v_loads = 0;  // producer, lane 0: what it has asked for
  int asked = 0;                              // scheduler: the same
  if (warp < 4) {
    tc::regs_dec<kRegsIssue>();
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      bool ok = true;
      int step = 0;  // key tiles loaded so far, over all items
      for (int n = 0, index = blockIdx.x; index >= 0 && ok; ++n) {
        const Item w = item_of(index);
        int mine = 1;
        if (lane == 0) {
          bool good = n == 0 || mbar_wait(&q_empty, (n - 1) & 1, &failed);
          if (good) {
            ++q_loads;
            mbar_arrive_expect_tx(&q_full, kTileBytes * NQ);
#pragma unroll
            for (int t = 0; t < NQ; ++t) {
              // rows past the end of the tensor are zero-filled by the copy engine
              tc::tma_load_4d(q_smem + t * kTileBytes, &map_q, &q_full, 0, w.q0 + t * BM, w.h, w.b);
              tc::tma_load_4d(q_smem + t * kTileBytes + kHalfBytes, &map_q, &q_full, 64, w.q0 + t * BM, w.h, w.b);
            }
          }
          for (int j = 0; j < w.n_kv && good; ++j) {
            const int s = (step + j) & 1, u = (step + j) >> 1;
            good = u == 0 || mbar_wait(&k_empty[s], (u - 1) & 1, &failed);
            if (!good) break;
            unsigned char* kd = k_smem + (size_t)s * kTileBytes;
            mbar_arrive_expect_tx(&k_full[s], kTileBytes);
            tc::tma_load_4d(kd, &map_k, &k_full[s], 0, j * BN, w.h, w.b);
            tc::tma_load_4d(kd + kHalfBytes, &map_k, &k_full[s], 64, j * BN, w.h, w.b);
            k_loads = step + j + 1;
            if (j + 1 == w.n_kv) tc::mbar_arrive(&next_wanted);
            good = u == 0 || mbar_wait(&v_empty[s], (u - 1) & 1, &failed);
            if (!good) break;
            unsigned char* vd = v_smem + (size_t)s * kTileBytes;
            mbar_arrive_expect_tx(&v_full[s], kTileBytes);
            tc::tma_load_4d(vd, &map_v, &v_full[s], 0, j * BN, w.h, w.b);
            tc::tma_load_4d(vd + kHalfBytes, &map_v, &v_full[s], 64, j * BN, w.h, w.b);
            v_loads = step + j + 1;
          }
          mine = good ? 1 : 0;
        }
        ok = __shfl_sync(kFull, mine, 0) != 0;
        step += w.n_kv;
        index = take_next(n, ok);
      }
      if (!ok && lane == 0) failed = 1;
    } else if (warp == 1) {
      // -------------------------------------------------------------------- MMA issuer
      // The whole warp runs this role and an elected lane issues (see tc::product_ss).
      constexpr uint32_t idesc_qk = tc::instr_desc(BM, BN, IS_BF16 ? 1 : 0, 0, 0);
      constexpr uint32_t idesc_pv = tc::instr_desc(BM, HD, IS_BF16 ? 1 : 0, 0, 1);
      const uint32_t tmem = __shfl_sync(kFull, tmem_base, 0);
      const uint64_t q_desc = tc::smem_desc(smem_u32(q_smem), 16, 1024);
      const uint64_t k_desc = tc::smem_desc(smem_u32(k_smem), 16, 1024);
      const uint64_t v_desc = tc::smem_desc(smem_u32(v_smem), kHalfBytes, 1024);
      // tile t, stage s: the address field moves by whole tiles and cannot carry out of it
      auto issue_qk = [&](int t, int stage) {
        tc::product_ss<kHalfBytes>(tmem + kColS + t * 128, q_desc + (uint32_t)(t * (kTileBytes >> 4)),
                                   k_desc + (uint32_t)(stage * (kTileBytes >> 4)), idesc_qk);
        tc::commit_elected(&s_full[t]);
      };
      bool ok = true;
      int step = 0;             // key tiles consumed so far, over all items
      int products[NQ] = {0, 0};  // P tiles consumed so far
      for (int n = 0, index = blockIdx.x; index >= 0 && ok; ++n) {
        const Item w = item_of(index);
        ok = __all_sync(kFull, mbar_wait(&q_full, n & 1, &failed)) &&
             __all_sync(kFull, mbar_wait(&k_full[step & 1], (step >> 1) & 1, &failed));
        if (!ok) break;
        tc::fence_after_sync();
#pragma unroll
        for (int t = 0; t < NQ; ++t)
          if (w.n_kv_t[t] > 0) issue_qk(t, step & 1);
        tc::commit_elected(&k_empty[step & 1]);
        if (w.n_kv == 1) tc::commit_elected(&q_empty);
        for (int j = 0; j < w.n_kv; ++j) {
          const int s = (step + j) & 1, u = (step + j) >> 1;
          const int s1 = (step + j + 1) & 1, u1 = (step + j + 1) >> 1;
          ok = __all_sync(kFull, mbar_wait(&v_full[s], u & 1, &failed));
          if (j + 1 < w.n_kv) ok = ok && __all_sync(kFull, mbar_wait(&k_full[s1], u1 & 1, &failed));
          if (!ok) break;
#pragma unroll
          for (int t = 0; t < NQ; ++t) {
            const bool do_pv = j < w.n_kv_t[t], do_qk = j + 1 < w.n_kv_t[t];
            if (do_pv) {
              // O_t += P_t V_j: the first kSplit keys of P, then the rest - the product starts
              // while the last exponentials of the tile are still being formed
              ok = ok && __all_sync(kFull, mbar_wait(&p_full[t], products[t] & 1, &failed));
              if (!ok) break;
              tc::fence_after_sync();
              const uint64_t vd = v_desc + (uint32_t)(s * (kTileBytes >> 4));
              const uint32_t o = tmem + kColO + t * 128, pa = tmem + kColS + t * 128;
              tc::product_ts<kSplit / 16>(o, pa, vd, idesc_pv, j > 0);
              ok = __all_sync(kFull, mbar_wait(&p_rest[t], products[t] & 1, &failed));
              if (!ok) break;
              tc::fence_after_sync();
              // (16 keys of V are 2048 bytes of a 64-column box)
              tc::product_ts<(BN - kSplit) / 16>(o, pa + kSplit / 2, vd + (uint32_t)(kSplit / 16 * 2048 >> 4), idesc_pv, 1u);
              ++products[t];
              // only the last product of the tile needs a signal of its own: every earlier one
              // is covered by the commit behind the scores that follow it (a commit tracks all
              // MMAs issued before it)
              if (!do_qk) tc::commit_elected(&pv_done[t]);
            }
            // P_t(j) has been consumed by the MMAs just issued (the tensor core runs them in
            // order), so tile t's buffer can take S_t(j+1)
            if (do_qk) issue_qk(t, s1);
          }
          if (!ok) break;
          tc::commit_elected(&v_empty[s]);
          if (j + 1 < w.n_kv) tc::commit_elected(&k_empty[s1]);
          if (j + 2 == w.n_kv) tc::commit_elected(&q_empty);  // the item's last scores are issued
        }
        step += w.n_kv;
        index = take_next(n, ok);
      }
      if (!ok && lane == 0) failed = 1;
      __syncwarp();
    } else if (warp == 2) {
      // -------------------------------------------------------------------- scheduler
      // Asked for when the last K of an item is under way, two steps before its end: soon enough for its Q, and not
      // before - a block that asked at the start of a long item would keep a pending one from those that
      // finish first.
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
    }
  } else {
    // ----------------------------------------------------------- softmax + epilogue
    tc::regs_inc<kRegsSoftmax>();
    const int t = (warp >> 2) - 1;           // query tile of this warp group
    const int quad = warp & 3;               // TMEM lane quadrant this warp may touch
    const int row = quad * 32 + lane;        // row inside the query tile
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t s_addr = lane_addr + kColS + t * 128;
    const uint32_t o_addr = lane_addr + kColO + t * 128;
    bool ok = true;
    int seen = 0;   // score tiles of this query tile so far, over all items
    int closed = 0; // items in which this query tile had work
    for (int n = 0, index = blockIdx.x; index >= 0 && ok; ++n) {
      const Item w = item_of(index);
      const int qt0 = w.q0 + t * BM;
      const int qi = qt0 + row;
      const int my_n_kv = t ? w.n_kv_t[1] : w.n_kv_t[0];
      float m_used = -INFINITY;  // reference maximum (scaled, log2 domain)
      float l = 0.f;             // running sum of exp2(s - m_used)
      for (int j = 0; j < my_n_kv; ++j) {
        if (!__all_sync(kFull, mbar_wait(&s_full[t], seen & 1, &failed))) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
        const int col0 = j * BN;
        const bool edge = (col0 + BN > p.Sk) || (p.causal && (col0 + BN - 1 > qt0 + diag));
        // last visible key of this row, relative to the tile
        int lim = BN - 1;
        if (edge) {
          int last = p.Sk - 1;
          if (p.causal && qi + diag < last) last = qi + diag;
          lim = last - col0;
        }
        softmax_tile<IS_BF16>(s_addr, o_addr, edge, lim, j == 0, p.scale_log2, m_used, l, &p_full[t], &p_rest[t]);
        ++seen;
      }
      if (ok && my_n_kv > 0) {
        ok = __all_sync(kFull, mbar_wait(&pv_done[t], closed & 1, &failed));  // the tile's last product
        ++closed;
      }
      if (ok) {
        tc::fence_after_sync();
        const float inv = (l > 0.f) ? 1.f / l : 0.f;
        const bool live = qi < p.Sq;
        unsigned char* orow = reinterpret_cast<unsigned char*>(p.o) +
                              2 * ((long long)w.b * p.o_stride_b + (long long)w.h * p.o_stride_h +
                                   (long long)qi * p.o_stride_s);
        if (my_n_kv > 0) {
#pragma unroll
          for (int c = 0; c < HD / 32; ++c) {
            uint32_t o[32];
            tc::tmem_ld32(o_addr + c * 32, o);
            tc::tmem_wait_ld();
            if (live) tc::store_row32<IS_BF16>(orow + c * 64, o, inv, p.wide != 0);
          }
          if (live && p.lse != nullptr) {
            const float lse = l == 0.f ? -INFINITY : (m_used + log2f(l)) * 0.69314718055994530942f;  // (l may be NaN)
            p.lse[((long long)w.b * p.H + w.h) * p.Sq + qi] = lse;
          }
        }
      }
      // (the next item's scores may be written meanwhile, but its first product waits for this
      // warp's probabilities, which come after the reads of O above)
      tc::fence_before_sync();
      index = take_next(n, ok);
    }
    if (!ok && lane == 0) failed = 1;
  }

  tc::fence_before_sync();
  __syncthreads();
  if (failed) {  // (uniform: nobody writes it any more)
    // a role gave up: what the others have under way has to end before the block does
    if (threadIdx.x == 0) {
      tc::await_copies<1>(&q_full, q_loads);
      tc::await_copies<kStages>(k_full, k_loads);
      tc::await_copies<kStages>(v_full, v_loads);
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

// Heads whose blocks are dispatched together.
// Without a mask every query block of a head reads all of its K and V, so the heads go one
// after the other (group of 1: blockIdx order = head-major, as a 2-D grid would give).
// Under a causal mask heads run in groups, the long query blocks of all of them first: what a group's
// long blocks find of K and V in L2 against the SMs that wait for the last group's long blocks at the end.
// One group where the K and V of all heads stay in L2, else equal groups of about 40 MB.  Groups of
// 8 heads -> this: 1 x 32 heads of 2048 keys 60 -> 49 us, 2 x 32 87 -> 73, 2 x 16 of 4096 179 -> 145,
// 3 x 12 of 5014 295 -> 240, 2 x 8 of 8192 315 -> 272, 4 x 32 of 2048 145 -> 138, 8 x 32 of 4096 the same.
// Three query tiles make a block of one tile and a block of two, the block of one first.  With as many keys as
// queries both have three tile products: neither is the long one, and what is left of groups is that both
// blocks read the same K and V.  Groups of 8 heads and one group: 96 heads of 300 18.6 and 19.7 us, 128 18.7 and 20.3,
// 192 25.1 and 25.8, 256 31.0 and 31.7; of 384 18.6 and 20.4, 20.6 and 20.6, 26.8 and 26.8, 32.9 and 32.9.  With more
// keys the block of two has more products (two at three key tiles, n - 3 at n), and which is better goes by how the
// blocks fall on the SMs at first, by what stays in L2 with more keys: 300 x 384 128 heads 23.0 and 24.1, 144 24.6 and
// 22.7, 256 37.1 and 35.5; 300 x 500 128 heads 25.7 and 24.7, 160 31.0 and 32.9; 300 x 1000 128 heads 39.0 and 37.0, 320
// 84.9 and 78.0; 261 x 700 256 heads 61.6 and 53.4.
// Where all blocks run at once no order is the better one for the end, and neighbours read the same K and V in
// groups of 8: 1 x 32 heads 1024 x 4096 58.1 us (in one group 59.6), 4 x 8 1000 x 3000 45.6 (46.1), 2 x 16 900 x 2000 32.8 (33.0).
int head_group_of(int B, int H, int Sq, int Sk, int causal) {
  static const int group_env = [] { const char* v = getenv("IXB_FA_HEAD_GROUP"); return v != nullptr ? atoi(v) : 0; }();
  if (group_env > 0) return group_env;
  if (!causal) return 1;
  const double all = (double)B * H, mb = Sk * (2. * HD * 2 / (1 << 20));  // heads, and MB of K and V of each
  const bool alike = Sq == Sk && ((long long)Sq + BM - 1) / BM == 3;
  const ixb_devinfo* dev = ixb_host::current_device();
  if (dev != nullptr && ((long long)Sq + BM * NQ - 1) / (BM * NQ) * all <= dev->sm_count) return 8;
  const double groups = alike ? ceil(all / 8) : all * mb <= 96 ? 1 : ceil(all / (mb < 5 ? floor(40 / mb) : 8));
  return (int)ceil(all / groups);
}

}  // namespace

extern "C" int ixb_fa_fwd_plan(int32_t B, int32_t H, int32_t Sq, int32_t Sk, int causal, int32_t* heads, int32_t* blocks) {
  if (B <= 0 || H <= 0 || Sq <= 0 || Sk <= 0 || heads == nullptr || blocks == nullptr) return IXB_ERR_ARG;
  *heads = head_group_of(B, H, Sq, Sk, causal);
  *blocks = ixb_host::fa_split_size(B, H, Sq, Sk);
  return IXB_OK;
}

extern "C" int ixb_fa_fwd(int dtype, const void* q, const void* k, const void* v, void* o, float* lse,
                          int32_t B, int32_t H, int32_t Sq, int32_t Sk, int32_t D,
                          const int64_t* q_strides, const int64_t* k_strides,
                          const int64_t* v_strides, const int64_t* o_strides, float scale,
                          int causal, int32_t* status, ixb_stream stream) {
  if (B < 0 || H < 0 || Sq < 0 || Sk < 0) return IXB_ERR_ARG;
  if (B == 0 || H == 0 || Sq == 0) return IXB_OK;
  if (!q || !k || !v || !o || !q_strides || !k_strides || !v_strides || !o_strides) return IXB_ERR_ARG;
  if (dtype != IXB_BF16 && dtype != IXB_F16) return IXB_ERR_DTYPE;
  if (D != HD) return IXB_ERR_SHAPE;
  if (Sk <= 0) return IXB_ERR_SHAPE;
  if (causal && Sk < Sq) return IXB_ERR_SHAPE;  // some rows would see no key at all
  if ((long long)B * H > 65535) return IXB_ERR_SHAPE;
  const void* ptrs[4] = {q, k, v, o};
  const int64_t* strs[4] = {q_strides, k_strides, v_strides, o_strides};
  for (int t = 0; t < 4; ++t) {
    if (!ixb_host::aligned16(ptrs[t])) return IXB_ERR_ALIGN;
    for (int i = 0; i < 3; ++i)
      if (strs[t][i] <= 0 || (strs[t][i] * 2) % 16 != 0) return IXB_ERR_ALIGN;
  }
  const int is_bf16 = dtype == IXB_BF16;
  CUtensorMap mq, mk, mv;
  if (int st = ixb_host::make_fa_map(&mq, q, is_bf16, B, H, Sq, q_strides[0], q_strides[1], q_strides[2])) return st;
  if (int st = ixb_host::make_fa_map(&mk, k, is_bf16, B, H, Sk, k_strides[0], k_strides[1], k_strides[2])) return st;
  if (int st = ixb_host::make_fa_map(&mv, v, is_bf16, B, H, Sk, v_strides[0], v_strides[1], v_strides[2])) return st;
  FaParams p;
  p.o = o;
  p.lse = lse;
  p.status = status;
  p.o_stride_b = o_strides[0];
  p.o_stride_h = o_strides[1];
  p.o_stride_s = o_strides[2];
  p.B = B;
  p.H = H;
  p.Sq = Sq;
  p.Sk = Sk;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal ? 1 : 0;
  p.wide = ixb_host::rows_aligned32(o, o_strides) ? 1 : 0;
  p.head_group = head_group_of(B, H, Sq, Sk, causal);
  if (!(scale > 0.f)) return IXB_ERR_ARG;  // the row maximum is taken before scaling
  if (const int cluster = ixb_host::fa_split_size(B, H, Sq, Sk))
    return ixb_host::fa_split(cluster, is_bf16, mq, mk, mv, o, lse, B, H, Sq, Sk, o_strides, scale, causal, status, (cudaStream_t)stream);
  const dim3 grid((unsigned)(((Sq + BM * NQ - 1) / (BM * NQ)) * (long long)B * H));
  auto kern = is_bf16 ? fa_fwd_kernel<true> : fa_fwd_kernel<false>;
  // the shared-memory opt-in is a property of (kernel, device): set once per device
  static std::atomic<bool> configured[2][64];
  int devid = 0;
  cudaGetDevice(&devid);
  std::atomic<bool>& done = configured[is_bf16][devid & 63];
  if (!done.load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e != cudaSuccess) return ixb_host::cuda_status(e);
    // the softmax warps' setmaxnreg waits for registers the block owns: never launch a build
    // that was given fewer at launch than the split adds up to (the Makefile fails on one; this
    // is for objects built without it)
    cudaFuncAttributes at;
    e = cudaFuncGetAttributes(&at, kern);
    if (e != cudaSuccess) return ixb_host::cuda_status(e);
    if (at.numRegs != kRegsLaunch) return IXB_ERR_UNSUPPORTED;
    done.store(true, std::memory_order_release);
  }
  kern<<<grid, kThreads, kSmemBytes, (cudaStream_t)stream>>>(mq, mk, mv, p);
  return ixb_host::cuda_status(cudaGetLastError());
}
