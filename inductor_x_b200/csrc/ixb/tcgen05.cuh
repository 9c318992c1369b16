// Inline-PTX wrappers for the 5th-generation tensor core path of sm_100a: tensor-memory
// (TMEM) allocation, tcgen05.mma issue with shared-memory / TMEM operands, completion
// through mbarriers, TMEM <-> register moves, and tiled TMA loads.
#pragma once
#include <cuda.h>

#include "tma.cuh"

namespace ixb {
namespace tc {

// ---- shared-memory matrix descriptor (SM100 format, version 1) ---------------------
// start address, leading-dimension and stride-dimension byte offsets are stored without
// their 4 least significant bits.  layout_type 2 = 128-byte swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t smem_addr, uint32_t lbo_bytes,
                                              uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3fffu);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3fffu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3fffu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}

// the same without a swizzle: 8 x 8 blocks of 128 contiguous bytes
__device__ __forceinline__ uint64_t smem_desc_plain(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return smem_desc(smem_addr, lbo_bytes, sbo_bytes) & ~((uint64_t)7 << 61);
}

// ---- instruction descriptor for kind::f16 (fp32 accumulate) ---------------------------
// is_bf16: operand format (0 = f16, 1 = bf16); *_mn_major: 0 = K-major, 1 = MN-major.
__host__ __device__ constexpr uint32_t instr_desc(int m, int n, int is_bf16, int a_mn_major,
                                                  int b_mn_major) {
  return (1u << 4) | ((uint32_t)is_bf16 << 7) | ((uint32_t)is_bf16 << 10) |
         ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// ---- TMEM allocation (whole warp) ---------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ---- one 128 x 128 x 128 product, issued by a whole converged warp -----------------------
// Every lane runs the issuing loop and one elected lane executes the instructions: the
// operands then stay warp-uniform.  In a loop that a single lane runs (`if (lane == 0)`) the
// compiler has to move each operand of each MMA from a per-lane register first, which costs
// issue slots that the arithmetic warps beside it win.
// D = A B^T, both operands K-major tiles (two boxes of 64 columns, `kBox` bytes apart): 8 steps
// of 16 along the reduced axis, 32 bytes a step inside the 128-byte swizzled row.
template <int kBox>
__device__ __forceinline__ void product_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n\t"
      ".reg .pred e, f, t;\n\t"
      ".reg .b64 a1, a2, a3, a4, a5, a6, a7, b1, b2, b3, b4, b5, b6, b7;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 f, 0, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "add.s64 a1, %1, 2;\n\tadd.s64 b1, %2, 2;\n\t"
      "add.s64 a2, %1, 4;\n\tadd.s64 b2, %2, 4;\n\t"
      "add.s64 a3, %1, 6;\n\tadd.s64 b3, %2, 6;\n\t"
      "add.s64 a4, %1, %4;\n\tadd.s64 b4, %2, %4;\n\t"
      "add.s64 a5, a4, 2;\n\tadd.s64 b5, b4, 2;\n\t"
      "add.s64 a6, a4, 4;\n\tadd.s64 b6, b4, 4;\n\t"
      "add.s64 a7, a4, 6;\n\tadd.s64 b7, b4, 6;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, f;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, t;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, t;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, t;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a4, b4, %3, t;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a5, b5, %3, t;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a6, b6, %3, t;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a7, b7, %3, t;\n\t"
      "}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(kBox >> 4)
      : "memory");
}
// D (+)= A B over N steps of 16 of the reduced index: A in TMEM as 16-bit pairs (8 columns a
// step), B a tile in MN-major form (16 rows = 2048 bytes a step)
template <int N> __device__ __forceinline__ void product_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                                            uint32_t idesc, uint32_t accumulate) {
  static_assert(N == 2 || N == 4 || N == 6 || N == 8, "whole pairs of steps");
  asm volatile(
      "{\n\t"
      ".reg .pred e, f, t;\n\t"
      ".reg .b32 a;\n\t"
      ".reg .b64 b;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 f, %4, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "add.u32 a, %1, 8;\n\tadd.s64 b, %2, 128;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, f;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n\t"
      "}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
  if constexpr (N > 2) product_ts<N - 2>(d_tmem, a_tmem + 16, b_desc + 256, idesc, 1u);
}
// D (+)= A B over N steps of 16 of the reduced index, both operands in shared memory, kA and kB bytes a step
template <int N, int kA, int kB>
__device__ __forceinline__ void product_ss_steps(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate) {
  static_assert(N % 2 == 0, "whole pairs of steps");
  asm volatile(
      "{\n\t"
      ".reg .pred e, f, t;\n\t"
      ".reg .b64 a, b;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 f, %4, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "add.s64 a, %1, %5;\n\tadd.s64 b, %2, %6;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, f;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "n"(kA >> 4), "n"(kB >> 4)
      : "memory");
  if constexpr (N > 2) product_ss_steps<N - 2, kA, kB>(d_tmem, a_desc + 2 * (kA >> 4), b_desc + 2 * (kB >> 4), idesc, 1u);
}
// By the elected lane of a converged warp, the one that issued the products: the mbarrier gets one
// arrival when every MMA issued so far by this lane has finished.
__device__ __forceinline__ void commit_elected(uint64_t* bar) {
  asm volatile(
      "{\n\t"
      ".reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
      "}" ::"r"(smem_u32(bar))
      : "memory");
}

// ---- TMEM <-> registers: 32 lanes x 32 columns of 32 bits, thread i <-> lane base+i ---
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
      "%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
      "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
      "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
      "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ---- 32 accumulators of one row to memory as 16-bit values ----------------------------------------
// A lane stores its own row, so the lanes of a warp touch 32 lines an instruction, and the waits of the
// other roles queue behind in the load/store unit: a store moves a whole 32-byte sector where the
// rows allow it (`wide`: `dst` is a multiple of 32 bytes), half of one otherwise.
template <bool IS_BF16> __device__ __forceinline__ uint32_t round_pair(float lo, float hi) {
  if constexpr (IS_BF16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}
template <bool IS_BF16>
__device__ __forceinline__ void store_row32(unsigned char* dst, const uint32_t (&acc)[32], float mult, bool wide) {
  uint32_t w[16];
#pragma unroll
  for (int k = 0; k < 16; ++k)
    w[k] = round_pair<IS_BF16>(__uint_as_float(acc[2 * k]) * mult, __uint_as_float(acc[2 * k + 1]) * mult);
  if (wide) {
#pragma unroll
    for (int k = 0; k < 16; k += 8)
      asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + 4 * k), "r"(w[k]), "r"(w[k + 1]),
                   "r"(w[k + 2]), "r"(w[k + 3]), "r"(w[k + 4]), "r"(w[k + 5]), "r"(w[k + 6]), "r"(w[k + 7])
                   : "memory");
  } else {
#pragma unroll
    for (int k = 0; k < 16; k += 4)
      *reinterpret_cast<uint4*>(dst + 4 * k) = make_uint4(w[k], w[k + 1], w[k + 2], w[k + 3]);
  }
}

// ---- leaving after a wait that gave up --------------------------------------------------------
// A block must not leave while copies into its shared memory or MMAs on its operands are under way.
// Bounded like every wait, and without a look at the abort flag, which is up by then.
// The last copies into a ring of STAGES tiles, `issued` of them so far (one thread).
template <int STAGES> __device__ __forceinline__ void await_copies(uint64_t* full, int issued) {
#pragma unroll
  for (int s = 1; s <= STAGES; ++s) {
    const int last = issued - s;
    if (last >= 0) mbar_wait(&full[last % STAGES], (last / STAGES) & 1);
  }
}
// Every product this warp has issued; `bar` (one arrival) is used for nothing else (whole warp).
__device__ __forceinline__ void await_products(uint64_t* bar) {
  __syncwarp();
  commit_elected(bar);
  __all_sync(kFull, mbar_wait(bar, 0));
}

// ---- register split between warpgroups (whole warpgroup) -------------------------------
template <int N> __device__ __forceinline__ void regs_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N> __device__ __forceinline__ void regs_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

// ---- work of blocks that have not started yet (one thread) -----------------------------------
// Asks for the index of a block of this grid that the hardware has not launched; the answer
// (16 bytes) lands in shared memory and completes 16 bytes on `bar`.  A running block that
// takes over a pending one keeps its tensor memory, barriers and pipelines.
__device__ __forceinline__ void request_next_block(void* answer, uint64_t* bar) {
  mbar_arrive_expect_tx(bar, 16);
  asm volatile(
      "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
          smem_u32(answer)),
      "r"(smem_u32(bar))
      : "memory");
}
// blockIdx.x of the block taken over, or -1 when none was left
__device__ __forceinline__ int next_block(const void* answer) {
  int taken, x = 0;
  asm volatile(
      "{\n\t"
      ".reg .b128 h;\n\t"
      ".reg .pred p;\n\t"
      "ld.shared.b128 h, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.s32 %0, 1, 0, p;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t"
      "}"
      : "=r"(taken), "+r"(x)
      : "r"(smem_u32(answer))
      : "memory");
  // the copy engine may write the next answer over this one once the reader says so
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  return taken ? x : -1;
}

// ---- tiled TMA load, rank 4, this CTA only --------------------------------------------
// c0 is the innermost coordinate; c0 * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar,
                                            int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace tc
}  // namespace ixb
