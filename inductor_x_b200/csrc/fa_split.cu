// Attention forward for few query rows, or few heads: fa_fwd.cu gives a block two query tiles and all the
// keys they see, which leaves most SMs without work when there are fewer such blocks than SMs.  Here a
// cluster of 1, 2, 4 or 8 blocks takes ONE query tile of one (batch, head) and shares its keys: each block
// has two tiles of scores in tensor memory as there, but of the same query tile and of different key
// tiles - slot s = 2 * rank + t of a cluster walks the key tiles s, s + slots, ...  At the end every slot
// leaves its row maxima, sums and 32-bit accumulators in shared memory, and the blocks of the cluster add
// them up row by row through distributed shared memory: one launch, no scratch, the same bits every time.
//
//   warp 0     TMA producer: Q, then K and V tiles; a tile of each in flight for each slot
//   warp 1     MMA issuer, the slots in turn
//   warps 4-7  softmax of slot 0, warps 8-11 of slot 1: thread <-> query row (softmax_tile)
//   all        after a cluster barrier warps 4-11 merge the rows of the tile, a warp a row
//
// Every mbarrier wait is bounded and raises a flag in `status`; the hardware barriers are reached by every
// warp whatever happened to it.
//
// Bound: latency.  A block lives for the launch, the first copies (2 us together), 1.5 us a step of two key
// tiles, and the merge.  When it is taken, and what it measured, stands at fa_split_size.
#include <atomic>
#include <cmath>
#include "host.h"
#include "fa_maps.h"
#include "ixb/fa_softmax.cuh"

namespace {

using namespace ixb;
using namespace ixb::fa;

// Registers: the block starts with kRegsLaunch a thread (all that 12 warps can have); the first
// warpgroup gives up what it does not need so that a softmax thread holds its row of 128 scores.
constexpr int kRegsLaunch = 168, kRegsIssue = 80, kRegsSoftmax = 208;
static_assert(kRegsIssue + NQ * kRegsSoftmax <= (1 + NQ) * kRegsLaunch, "setmaxnreg draws on the block's own registers");
constexpr int kMaxCluster = 8;
constexpr size_t kSmemBytes = (size_t)kTileBytes * 5 + 1024;
static_assert(NQ * BM * HD * sizeof(float) <= (size_t)kTileBytes * 5, "the accumulators take the place of the operands");

struct SplitParams {
  void* o;
  float* lse;            // [B, H, Sq], may be null
  int* status;           // may be null
  long long o_stride_b, o_stride_h, o_stride_s;  // elements
  int B, H, Sq, Sk;
  float scale_log2;
  int causal;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(const void* local_smem, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local_smem)), "r"(rank));
  return remote;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <bool IS_BF16, int CLUSTER>
__global__ void __launch_bounds__(kThreads, 1)
    fa_split_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const SplitParams p) {
  constexpr int kSlots = NQ * CLUSTER;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* q_smem = smem;
  unsigned char* k_smem = smem + kTileBytes;       // a tile for each slot
  unsigned char* v_smem = smem + kTileBytes * 3;

  __shared__ __align__(8) uint64_t q_full, k_full[NQ], k_empty[NQ], v_full[NQ], v_empty[NQ], s_full[NQ], p_full[NQ], p_rest[NQ],
      pv_done[NQ], drained;
  __shared__ float m_row[NQ][BM], l_row[NQ][BM];
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int failed;

  const int warp = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0);  // known uniform to the compiler
  const int lane = threadIdx.x & 31;
  const int rank = CLUSTER > 1 ? (int)cluster_rank() : 0;

  // late (long) query tiles of a head first
  const int n_q_tiles = (p.Sq + BM - 1) / BM;
  const int item = (int)blockIdx.x / CLUSTER;
  const int bh = item / n_q_tiles, b = bh / p.H, h = bh % p.H;
  const int q0 = (n_q_tiles - 1 - item % n_q_tiles) * BM;
  const int diag = p.Sk - p.Sq;  // key j is visible to query row i when j <= i + diag
  int kv_end = p.Sk;
  if (p.causal && q0 + BM + diag < kv_end) kv_end = q0 + BM + diag;
  const int n_kv = (kv_end + BN - 1) / BN;
  auto tiles_of = [&](int t) {
    const int s = NQ * rank + t;
    return n_kv > s ? (n_kv - s + kSlots - 1) / kSlots : 0;
  };
  const int n_t[NQ] = {tiles_of(0), tiles_of(1)};  // (n_t[0] is n_t[1] or one more)

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int t = 0; t < NQ; ++t) {
      mbar_init(&k_full[t], 1);
      mbar_init(&k_empty[t], 1);
      mbar_init(&v_full[t], 1);
      mbar_init(&v_empty[t], 1);
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

  int q_loads = 0, k_loads[NQ] = {0, 0}, v_loads[NQ] = {0, 0};  // producer, thread 0: what it has asked for
  float m_used = -INFINITY, l = 0.f;                            // softmax warps: this thread's row
  const int t_own = (warp >> 2) - 1;                            // and the slot it belongs to
  const int row_own = (warp & 3) * 32 + lane;
  const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
  if (warp < 4) {
    tc::regs_dec<kRegsIssue>();
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0 && n_t[0] > 0) {
        bool good = true;
        q_loads = 1;
        mbar_arrive_expect_tx(&q_full, kTileBytes);
        tc::tma_load_4d(q_smem, &map_q, &q_full, 0, q0, h, b);  // rows past the end are zero-filled
        tc::tma_load_4d(q_smem + kHalfBytes, &map_q, &q_full, 64, q0, h, b);
        for (int k = 0; k < n_t[0] && good; ++k) {
#pragma unroll
          for (int t = 0; t < NQ; ++t) {
            if (k >= n_t[t] || !good) continue;
            const int key0 = (NQ * rank + t + k * kSlots) * BN;
            good = k == 0 || mbar_wait(&k_empty[t], (k - 1) & 1, &failed);
            if (!good) continue;
            unsigned char* kd = k_smem + t * kTileBytes;
            mbar_arrive_expect_tx(&k_full[t], kTileBytes);
            tc::tma_load_4d(kd, &map_k, &k_full[t], 0, key0, h, b);
            tc::tma_load_4d(kd + kHalfBytes, &map_k, &k_full[t], 64, key0, h, b);
            k_loads[t] = k + 1;
          }
#pragma unroll
          for (int t = 0; t < NQ; ++t) {
            if (k >= n_t[t] || !good) continue;
            const int key0 = (NQ * rank + t + k * kSlots) * BN;
            good = k == 0 || mbar_wait(&v_empty[t], (k - 1) & 1, &failed);
            if (!good) continue;
            unsigned char* vd = v_smem + t * kTileBytes;
            mbar_arrive_expect_tx(&v_full[t], kTileBytes);
            tc::tma_load_4d(vd, &map_v, &v_full[t], 0, key0, h, b);
            tc::tma_load_4d(vd + kHalfBytes, &map_v, &v_full[t], 64, key0, h, b);
            v_loads[t] = k + 1;
          }
        }
        if (!good) failed = 1;
      }
      __syncwarp();
    } else if (warp == 1 && n_t[0] > 0) {
      // -------------------------------------------------------------------- MMA issuer
      // The whole warp runs this role and an elected lane issues (see tc::product_ss).
      constexpr uint32_t idesc_qk = tc::instr_desc(BM, BN, IS_BF16 ? 1 : 0, 0, 0);
      constexpr uint32_t idesc_pv = tc::instr_desc(BM, HD, IS_BF16 ? 1 : 0, 0, 1);
      const uint32_t tmem = __shfl_sync(kFull, tmem_base, 0);
      const uint64_t q_desc = tc::smem_desc(smem_u32(q_smem), 16, 1024);
      const uint64_t k_desc = tc::smem_desc(smem_u32(k_smem), 16, 1024);
      const uint64_t v_desc = tc::smem_desc(smem_u32(v_smem), kHalfBytes, 1024);
      auto wait = [&](uint64_t* bar, int parity) {
        const bool up = __all_sync(kFull, mbar_wait(bar, parity, &failed));
        tc::fence_after_sync();
        return up;
      };
      auto issue_qk = [&](int t) {
        tc::product_ss<kHalfBytes>(tmem + kColS + t * 128, q_desc, k_desc + (uint32_t)(t * (kTileBytes >> 4)), idesc_qk);
        tc::commit_elected(&s_full[t]);
        tc::commit_elected(&k_empty[t]);
      };
      bool ok = wait(&q_full, 0);
#pragma unroll
      for (int t = 0; t < NQ; ++t) {
        if (!ok || n_t[t] == 0) continue;
        ok = wait(&k_full[t], 0);
        if (ok) issue_qk(t);
      }
      for (int k = 0; k < n_t[0] && ok; ++k) {
#pragma unroll
        for (int t = 0; t < NQ; ++t) {
          if (!ok || k >= n_t[t]) continue;
          ok = wait(&v_full[t], k & 1) && wait(&p_full[t], k & 1);
          if (!ok) continue;
          const uint64_t vd = v_desc + (uint32_t)(t * (kTileBytes >> 4));
          const uint32_t o = tmem + kColO + t * 128, pa = tmem + kColS + t * 128;
          tc::product_ts<kSplit / 16>(o, pa, vd, idesc_pv, k > 0);
          ok = wait(&p_rest[t], k & 1);
          if (!ok) continue;
          // (16 keys of V are 2048 bytes of a 64-column box)
          tc::product_ts<(BN - kSplit) / 16>(o, pa + kSplit / 2, vd + (uint32_t)(kSplit / 16 * 2048 >> 4), idesc_pv, 1u);
          tc::commit_elected(&v_empty[t]);
          if (k + 1 < n_t[t]) {
            ok = wait(&k_full[t], (k + 1) & 1);
            if (ok) issue_qk(t);  // (P of this tile has been consumed by the MMAs just issued: they run in order)
          } else {
            tc::commit_elected(&pv_done[t]);
          }
        }
      }
      if (!ok && lane == 0) failed = 1;
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------------------- softmax
    tc::regs_inc<kRegsSoftmax>();
    const uint32_t s_addr = lane_addr + kColS + t_own * 128, o_addr = lane_addr + kColO + t_own * 128;
    const int mine = t_own ? n_t[1] : n_t[0];
    const int qi = q0 + row_own;
    bool ok = true;
    for (int k = 0; k < mine; ++k) {
      ok = __all_sync(kFull, mbar_wait(&s_full[t_own], k & 1, &failed));
      if (!ok) break;
      tc::fence_after_sync();
      const int col0 = (NQ * rank + t_own + k * kSlots) * BN;
      const bool edge = (col0 + BN > p.Sk) || (p.causal && (col0 + BN - 1 > q0 + diag));
      int lim = BN - 1;  // last visible key of this row, relative to the tile
      if (edge) {
        int last = p.Sk - 1;
        if (p.causal && qi + diag < last) last = qi + diag;
        lim = last - col0;
      }
      softmax_tile<IS_BF16>(s_addr, o_addr, edge, lim, k == 0, p.scale_log2, m_used, l, &p_full[t_own], &p_rest[t_own]);
    }
    if (ok && mine > 0) ok = __all_sync(kFull, mbar_wait(&pv_done[t_own], 0, &failed));  // the slot's last product
    if (!ok && lane == 0) failed = 1;
  }

  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const bool gave_up = failed != 0;  // (uniform: nobody writes it any more)
  if (gave_up) {
    // a role gave up: what the others have under way has to end before the block does
    if (threadIdx.x == 0) {
      tc::await_copies<1>(&q_full, q_loads);
#pragma unroll
      for (int t = 0; t < NQ; ++t) {
        tc::await_copies<1>(&k_full[t], k_loads[t]);
        tc::await_copies<1>(&v_full[t], v_loads[t]);
      }
      if (p.status != nullptr) atomicExch(p.status, 1);
    }
    if (warp == 1) tc::await_products(&drained);
    __syncthreads();
  }
  // Every product has ended and every copy has been consumed: the accumulators take the operands' place,
  // row after row, their 16-byte pieces swizzled by the row (a thread writes a row, a warp reads one).
  float4* o_smem = reinterpret_cast<float4*>(smem);
  constexpr int kPieces = HD / 4;
  const int rows = p.Sq - q0 < BM ? p.Sq - q0 : BM;
  if (warp >= 4) {
    m_row[t_own][row_own] = gave_up ? -INFINITY : m_used;
    l_row[t_own][row_own] = gave_up ? 0.f : l;
    if (!gave_up && (t_own ? n_t[1] : n_t[0]) > 0) {
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tc::tmem_ld32(lane_addr + kColO + t_own * 128 + c * 32, o);
        tc::tmem_wait_ld();
        if (row_own < rows) {
#pragma unroll
          for (int e = 0; e < 8; ++e)
            o_smem[(t_own * BM + row_own) * kPieces + ((c * 8 + e) ^ lane)] =
                make_float4(__uint_as_float(o[4 * e]), __uint_as_float(o[4 * e + 1]), __uint_as_float(o[4 * e + 2]),
                            __uint_as_float(o[4 * e + 3]));
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncwarp();
  if constexpr (CLUSTER > 1) cluster_sync_all();
  else __syncthreads();
  if (warp >= 4) {
    unsigned char* base = reinterpret_cast<unsigned char*>(p.o) + 2 * ((long long)b * p.o_stride_b + (long long)h * p.o_stride_h);
    // several rows at a time (with more blocks a warp has fewer): one by one every row waits for its loads
    // and its two folds, 3 us for 128 rows of one block
    constexpr int kRows = CLUSTER <= 2 ? 4 : 8 / CLUSTER, kStep = 8 * CLUSTER;
    for (int r0 = rank * 8 + warp - 4; r0 < rows; r0 += kRows * kStep) {
      float w[kRows], top[kRows], total[kRows];
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        // lane s: the statistics of slot s
        const int r = r0 + i * kStep;
        float m = -INFINITY, ls = 0.f;
        if (lane < kSlots && r < rows) {
          if constexpr (CLUSTER > 1) {
            m = ld_cluster_f32(map_to_rank(&m_row[lane % NQ][r], lane / NQ));
            ls = ld_cluster_f32(map_to_rank(&l_row[lane % NQ][r], lane / NQ));
          } else {
            m = m_row[lane][r];
            ls = l_row[lane][r];
          }
        }
        top[i] = m;  // (-inf: the slot saw nothing of the row, or nothing but NaN, which its sum says)
        total[i] = ls;
      }
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const float m = top[i];
        top[i] = warp_max_fast(m);
        w[i] = m == -INFINITY ? 0.f : fast_exp2(m - top[i]);
        total[i] = warp_reduce<SumOp>(w[i] * total[i]);
      }
      float4 acc[kRows];
#pragma unroll
      for (int i = 0; i < kRows; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int s = 0; s < kSlots; ++s) {
        float4 v[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const int r = r0 + i * kStep;
          const float4* piece = &o_smem[(s % NQ * BM + r) * kPieces + (lane ^ (r & 31))];
          // (a slot without a key tile wrote nothing; every other one counts whatever it weighs, since no weight
          // makes a NaN or an infinity of it go away)
          v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (s < n_kv && r < rows) v[i] = CLUSTER > 1 ? ld_cluster_f32x4(map_to_rank(piece, s / NQ)) : *piece;
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const float ws = __shfl_sync(kFull, w[i], s);
          acc[i].x = fmaf(ws, v[i].x, acc[i].x);
          acc[i].y = fmaf(ws, v[i].y, acc[i].y);
          acc[i].z = fmaf(ws, v[i].z, acc[i].z);
          acc[i].w = fmaf(ws, v[i].w, acc[i].w);
        }
      }
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const int r = r0 + i * kStep;
        if (r >= rows) break;
        const float inv = total[i] == 0.f ? 0.f : 1.f / total[i];  // (a sum may be NaN)
        uint2 out;
        out.x = tc::round_pair<IS_BF16>(acc[i].x * inv, acc[i].y * inv);
        out.y = tc::round_pair<IS_BF16>(acc[i].z * inv, acc[i].w * inv);
        *reinterpret_cast<uint2*>(base + 2 * (long long)(q0 + r) * p.o_stride_s + lane * 8) = out;
        if (lane == 0 && p.lse != nullptr)
          p.lse[((long long)b * p.H + h) * p.Sq + q0 + r] =
              total[i] == 0.f ? -INFINITY : (top[i] + log2f(total[i])) * 0.69314718055994530942f;
      }
    }
  }
  // nobody leaves while another block of the cluster reads its shared memory
  __syncwarp();
  if constexpr (CLUSTER > 1) cluster_sync_all();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// The opt-ins of a kernel on the current device, asked for once: a property of (kernel, device).
template <bool IS_BF16, int CLUSTER>
int configure(int devid) {
  auto kern = fa_split_kernel<IS_BF16, CLUSTER>;
  static std::atomic<bool> configured[64];
  std::atomic<bool>& done = configured[devid & 63];
  if (!done.load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e != cudaSuccess) return ixb_host::cuda_status(e);
    cudaFuncAttributes at;  // (as in fa_fwd.cu: the softmax warps wait for registers the block has to own)
    e = cudaFuncGetAttributes(&at, kern);
    if (e != cudaSuccess) return ixb_host::cuda_status(e);
    if (at.numRegs != kRegsLaunch) return IXB_ERR_UNSUPPORTED;
    done.store(true, std::memory_order_release);
  }
  return IXB_OK;
}

template <int CLUSTER>
cudaLaunchConfig_t launch_config(long long blocks, cudaLaunchAttribute* attr, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = CLUSTER;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CLUSTER > 1 ? 1 : 0;
  return cfg;
}

template <bool IS_BF16, int CLUSTER>
int launch_split(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const SplitParams& p, cudaStream_t stream) {
  int devid = 0;
  cudaGetDevice(&devid);
  if (int st = configure<IS_BF16, CLUSTER>(devid)) return st;
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = launch_config<CLUSTER>((long long)((p.Sq + BM - 1) / BM) * p.B * p.H * CLUSTER, &attr, stream);
  return ixb_host::cuda_status(cudaLaunchKernelEx(&cfg, fa_split_kernel<IS_BF16, CLUSTER>, mq, mk, mv, p));
}

// Blocks of clusters of this size that the current device runs at a time (0: none), asked for once.
template <int CLUSTER>
int room_for(int devid) {
  static std::atomic<int> known[64];  // one more than the number
  std::atomic<int>& room = known[devid & 63];
  int n = room.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = launch_config<CLUSTER>(CLUSTER, &attr, nullptr);
    int clusters = 0;
    if (configure<true, CLUSTER>(devid) != IXB_OK ||
        cudaOccupancyMaxActiveClusters(&clusters, fa_split_kernel<true, CLUSTER>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      clusters = 0;
    }
    n = 1 + clusters * CLUSTER;
    room.store(n, std::memory_order_relaxed);
  }
  return n - 1;
}
int room_for(int cluster, int devid, int sms) {
  return cluster == 1 ? sms : cluster == 2 ? room_for<2>(devid) : cluster == 4 ? room_for<4>(devid) : room_for<8>(devid);
}

}  // namespace

namespace ixb_host {

// Whether, and over how many blocks, the keys of a query tile are shared.  Times in us of both kernels, as
// measured on one B200 at 148 SMs (40 shapes, 1 to 256 heads, within 15 % where it matters):
//   fa_fwd_kernel  5.5 + 1.6 a key tile of its longest item; with one query tile an item (Sq <= 128) 5.3 +
//                  1.41, and 3.4 more for every further round of items
//   this one       5 for one row of the tile to 8.5 for all 128 (the merge), 1.6 for each key tile of a
//                  slot; or what reading K and V takes at 6.2 TB/s
// in one wave of blocks (148 SMs; clusters of 2, 4 and 8 find room for 148, 132 and 120 blocks there, room_for), or for
// Sq <= 128 in several.  Taken where it promises 7 %.  1 x 12 heads 18 x 3086: 40.4 -> 11 - 12 us; 1 x 32, 1 x 8192: 95.7
// -> 27; 3 x 16, 97 x 1840: 26.6 -> 16; 16 x 12, 1 x 2879: 74 -> 59; causal 1 x 4 of 2000: 30.5 -> 16.8, of 4096:
// 55.9 -> 34.4; 1 x 12 of 1000 without a mask 19.4 -> 15.5.  Where it is not taken: 2 x 8 of 2048 32.9 against
// 42.9 (two waves), 4 x 4 of 1288 causal 22.7 against 25.7, 2 x 4 of 128 6.9 against 8.5.  A causal mask changes
// neither time: the last query tile of a call sees every key, and it ends last.
int fa_split_size(int B, int H, int Sq, int Sk) {
  static const int forced = [] {
    const char* v = getenv("IXB_FA_SPLIT");
    const int n = v != nullptr ? atoi(v) : -1;
    return n == 0 || n == 1 || n == 2 || n == 4 || n == 8 ? n : -1;
  }();
  if (forced >= 0) return forced;
  const ixb_devinfo* dev = current_device();
  int devid = 0;
  if (dev == nullptr || cudaGetDevice(&devid) != cudaSuccess) return 0;
  const int sms = dev->sm_count;
  const double heads = (double)B * H;
  const double n_q = (Sq + BM - 1) / BM, n_kv = (Sk + BN - 1) / BN;  // (the last query tile sees every key)
  const bool one = Sq <= BM;
  const double rounds = ceil(((Sq + 2 * BM - 1) / (2 * BM)) * heads / sms);
  if (rounds > 1 && !one) return 0;
  const double plain = one ? 5.3 + rounds * 1.41 * n_kv + (rounds - 1) * 3.4 : 5.5 + 1.6 * n_kv;
  const double read = heads * Sk * 2 * HD * 2 / 6.2e6;
  double best = 0.93 * plain;
  int cluster = 0;
  for (int c = 1; c <= kMaxCluster; c *= 2) {
    auto time = [&](int room) {  // with room for so many blocks at a time
      const double waves = ceil(n_q * heads * c / room);
      if (waves > 1 && !one) return (double)INFINITY;
      const double t = waves * (5 + 3.5 * (one ? Sq : BM) / BM + 1.6 * ceil(n_kv / (2 * c)));
      return t > read ? t : read;
    };
    if (!(time(sms) < best)) continue;  // (and worse with less room)
    const int room = room_for(c, devid, sms);
    if (room <= 0) continue;
    const double t = time(room);
    if (t < best) {
      best = t;
      cluster = c;
    }
  }
  return cluster;
}

int fa_split(int cluster, int is_bf16, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, void* o, float* lse,
             int B, int H, int Sq, int Sk, const int64_t* o_strides, float scale, int causal, int32_t* status, cudaStream_t stream) {
  SplitParams p;
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
#define IXB_SPLIT_CASE(C) \
  if (cluster == C) return is_bf16 ? launch_split<true, C>(mq, mk, mv, p, stream) : launch_split<false, C>(mq, mk, mv, p, stream);
  IXB_SPLIT_CASE(1)
  IXB_SPLIT_CASE(2)
  IXB_SPLIT_CASE(4)
  IXB_SPLIT_CASE(8)
#undef IXB_SPLIT_CASE
  return IXB_ERR_UNSUPPORTED;
}

}  // namespace ixb_host
