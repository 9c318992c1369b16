// Kernel templates instantiated by generated functor modules.  The code generator
// classifies a fused node group into one of these families and emits a `Body` struct
// whose single method is straight-line code over gen_vec / gen_ops types:
//
//   pointwise_gen_kernel<Body>   Body::tile(xbase, nvalid): kVec consecutive elements of
//                                the flattened iteration space per call (128-bit access
//                                where an operand is contiguous along it)
//   row_gen_kernel<Body,...>     Body::row(ctx, x): one reduced row held in the registers of
//                                a team (same work split as row.cuh)
//   outer_gen_kernel<Body,...>   Body::tile(ctx, xbase, nvalid): reductions whose reduced axis
//                                is not stride-1; threads map along the kept axis and the
//                                body loops over the reduced index
//
// They play the role of the decorators the reference attaches to every emitted kernel,
// pointwise_npu_index / persistent_reduction_npu_index / reduction_npu_index
// (inductor_x/npu_triton_heuristics.py:545-611).
#pragma once
#include <atomic>

#include "gen_ops.cuh"
#include "row.cuh"
#include "tma.cuh"

namespace ixb {
namespace gen {

// ---- element access by storage type -------------------------------------------------
template <class T> struct Mem;
template <> struct Mem<float> {
  using val = float;
  static __device__ __forceinline__ float ld(const float* p) { return *p; }
  static __device__ __forceinline__ void st(float* p, float v) { *p = v; }
};
template <> struct Mem<f16> {
  using val = float;
  static __device__ __forceinline__ float ld(const f16* p) { return __half2float(*p); }
  static __device__ __forceinline__ void st(f16* p, float v) { *p = __float2half_rn(v); }
};
template <> struct Mem<bf16> {
  using val = float;
  static __device__ __forceinline__ float ld(const bf16* p) { return __bfloat162float(*p); }
  static __device__ __forceinline__ void st(bf16* p, float v) { *p = __float2bfloat16_rn(v); }
};
template <> struct Mem<double> {
  using val = float;
  static __device__ __forceinline__ float ld(const double* p) { return (float)*p; }
  static __device__ __forceinline__ void st(double* p, float v) { *p = (double)v; }
};
template <> struct Mem<long long> {
  using val = long long;
  static __device__ __forceinline__ long long ld(const long long* p) { return *p; }
  static __device__ __forceinline__ void st(long long* p, long long v) { *p = v; }
};
template <> struct Mem<int> {
  using val = long long;
  static __device__ __forceinline__ long long ld(const int* p) { return *p; }
  static __device__ __forceinline__ void st(int* p, long long v) { *p = (int)v; }
};
template <> struct Mem<short> {
  using val = long long;
  static __device__ __forceinline__ long long ld(const short* p) { return *p; }
  static __device__ __forceinline__ void st(short* p, long long v) { *p = (short)v; }
};
template <> struct Mem<signed char> {
  using val = long long;
  static __device__ __forceinline__ long long ld(const signed char* p) { return *p; }
  static __device__ __forceinline__ void st(signed char* p, long long v) { *p = (signed char)v; }
};
template <> struct Mem<unsigned char> {
  using val = long long;
  static __device__ __forceinline__ long long ld(const unsigned char* p) { return *p; }
  static __device__ __forceinline__ void st(unsigned char* p, long long v) { *p = (unsigned char)v; }
};
template <> struct Mem<bool> {
  using val = bool;
  static __device__ __forceinline__ bool ld(const bool* p) { return *p; }
  static __device__ __forceinline__ void st(bool* p, bool v) { *p = v; }
};

template <class V, int N> struct vec_of;
template <int N> struct vec_of<float, N> { using type = typename fres<N>::type; };
template <int N> struct vec_of<long long, N> { using type = typename ires<N>::type; };
template <int N> struct vec_of<bool, N> { using type = typename bres<N>::type; };

// conversions the store side needs: any value kind -> the element kind of the buffer
template <class V> struct Cast;
template <> struct Cast<float> {
  static __device__ __forceinline__ float from(float v) { return v; }
  static __device__ __forceinline__ float from(double v) { return (float)v; }
  static __device__ __forceinline__ float from(long long v) { return (float)v; }
  static __device__ __forceinline__ float from(bool v) { return v ? 1.f : 0.f; }
};
template <> struct Cast<long long> {
  static __device__ __forceinline__ long long from(float v) { return (long long)v; }
  static __device__ __forceinline__ long long from(double v) { return (long long)v; }
  static __device__ __forceinline__ long long from(long long v) { return v; }
  static __device__ __forceinline__ long long from(bool v) { return v ? 1 : 0; }
};
template <> struct Cast<bool> {
  static __device__ __forceinline__ bool from(float v) { return v != 0.f; }
  static __device__ __forceinline__ bool from(double v) { return v != 0.0; }
  static __device__ __forceinline__ bool from(long long v) { return v != 0; }
  static __device__ __forceinline__ bool from(bool v) { return v; }
};

// iota: xbase, xbase+1, ...
template <int N> __device__ __forceinline__ vi<N> iota(long long base) {
  vi<N> r;
#pragma unroll
  for (int i = 0; i < N; ++i) r.v[i] = base + i;
  return r;
}
template <class A> __device__ __forceinline__ auto lane0(const A& a) { return at(a, 0); }

// gather: one scalar access per element, predicated by `mask` (false -> `other`)
template <class T, class I, class M>
__device__ __forceinline__ auto gather(const T* p, const I& idx, const M& mask,
                                       typename Mem<T>::val other) {
  using V = typename Mem<T>::val;
  constexpr int N = rank2<I, M>::n;
  typename vec_of<V, N>::type r;
  if constexpr (N == 0) {
    r = at(mask, 0) ? Mem<T>::ld(p + at(idx, 0)) : other;
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) r.v[i] = at(mask, i) ? Mem<T>::ld(p + at(idx, i)) : other;
  }
  return r;
}
template <class T, class I, class M, class A>
__device__ __forceinline__ void scatter(T* p, const I& idx, const M& mask, const A& val) {
  using V = typename Mem<T>::val;
  constexpr int N = rank3<I, M, A>::n;
  if constexpr (N == 0) {
    if (at(mask, 0)) Mem<T>::st(p + at(idx, 0), Cast<V>::from(at(val, 0)));
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (at(mask, i)) Mem<T>::st(p + at(idx, i), Cast<V>::from(at(val, i)));
  }
}

// scatter with accumulation (store mode "atomic_add": index_put(accumulate=True), scatter_add
// and the outer split of the reference, inductor_x/codegen/triton.py:904-905): one atomic add
// per valid element, in the storage type of the destination
__device__ __forceinline__ void atomic_add(float* p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add(f16* p, float v) { atomicAdd(p, __float2half_rn(v)); }
__device__ __forceinline__ void atomic_add(bf16* p, float v) { atomicAdd(p, __float2bfloat16_rn(v)); }
__device__ __forceinline__ void atomic_add(double* p, float v) { atomicAdd(p, (double)v); }
__device__ __forceinline__ void atomic_add(long long* p, long long v) {
  atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
}
__device__ __forceinline__ void atomic_add(int* p, long long v) { atomicAdd(p, (int)v); }
template <class T, class I, class M, class A>
__device__ __forceinline__ void scatter_add(T* p, const I& idx, const M& mask, const A& val) {
  using V = typename Mem<T>::val;
  constexpr int N = rank3<I, M, A>::n;
  if constexpr (N == 0) {
    if (at(mask, 0)) atomic_add(p + at(idx, 0), Cast<V>::from(at(val, 0)));
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (at(mask, i)) atomic_add(p + at(idx, i), Cast<V>::from(at(val, i)));
  }
}

// contiguous run of N elements starting at p: 128-bit accesses when the address allows.  A
// complete run that starts off a 16-byte boundary is cut out of the aligned words that cover it
// (each of them holds at least one element of the run, so nothing beyond its 16 bytes is read).
// FAST: the caller knows the run is complete and 16-byte aligned (full tile, aligned base
// pointer checked on the host, index proven a multiple of the vector), so the access is
// unconditional - no branch separates the loads of an unrolled loop and they overlap.
// STREAM: the run is read once and nothing near it is (a gathered table row): no L1 allocation.
// CUT = false leaves out the form for runs off a boundary (element by element then): for loads that
// are made once per thread, where the extra code costs the rows that follow more than it gives.
// softmax -> LayerNorm with it in all, in none, in the shared-memory table of rows that do not fill
// their team only, as it is used: 16384 x 4096 bf16 60.1, 59.4, 59.4 us; 20011 x 1537 fp16 59.4,
// 58.3, 58.3; 9000 x 3001 fp32 78.0, 76.7, 76.7; 5000 x 5003 bf16 47.5, 48.2, 47.5.
template <class T, int N, bool FAST = false, bool STREAM = false, bool CUT = true>
__device__ __forceinline__ typename vec_of<typename Mem<T>::val, N>::type ldvec(const T* p, int nvalid) {
  using V = typename Mem<T>::val;
  typename vec_of<V, N>::type r;
  constexpr int kPer = 16 / sizeof(T);
  if constexpr ((N % kPer) == 0 && (sizeof(T) == 2 || sizeof(T) == 4) && std::is_same<V, float>::value) {
    if (FAST || (nvalid >= N && (reinterpret_cast<uintptr_t>(p) & 15u) == 0)) {
#pragma unroll
      for (int c = 0; c < N / kPer; ++c) {
        if constexpr (STREAM) unpack<T>(ldg_stream(p + c * kPer), &r.v[c * kPer]);
        else unpack<T>(ldg_keep(p + c * kPer), &r.v[c * kPer]);  // may be re-read: keep in L1
      }
      return r;
    }
    if (CUT && nvalid >= N && !STREAM) {
      // (plain loads, as the element-wise ones they replace: a later pass of a looped row may read
      // what an earlier one stored)
      const int s = off_boundary(p);
      const uint4* a = reinterpret_cast<const uint4*>(p - s);
      uint4 lo = a[0];
#pragma unroll
      for (int c = 0; c < N / kPer; ++c) {
        const uint4 hi = a[c + 1];
        unpack<T>(shift_words<T>(lo, hi, s), &r.v[c * kPer]);
        lo = hi;
      }
      return r;
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) r.v[i] = i < nvalid ? Mem<T>::ld(p + i) : V();
  return r;
}
// A run of N elements as the raw 128-bit words it was loaded as: what a thread holds while
// several independent loads are in flight, before any of them is widened.
template <class T, int N> struct RawVec {
  static constexpr int kWords = N * (int)sizeof(T) / 16;
  static_assert(kWords >= 1 && kWords * 16 == N * (int)sizeof(T), "whole 128-bit words");
  uint4 q[kWords];
};
// complete, 16-byte aligned run (the caller has established both), read once: no L1 allocation
template <class T, int N> __device__ __forceinline__ RawVec<T, N> ldraw(const T* p) {
  RawVec<T, N> r;
#pragma unroll
  for (int c = 0; c < RawVec<T, N>::kWords; ++c) r.q[c] = ldg_stream(p + c * (16 / (int)sizeof(T)));
  return r;
}
// Placed after a batch of ldraw calls: the words of `raw` cannot be consumed before this
// point, and (volatile statements keep their order) this point comes after every load of the
// batch - so all of them are issued before the first result is waited for.
template <class T, int N> __device__ __forceinline__ void pin(RawVec<T, N>& raw) {
#pragma unroll
  for (int c = 0; c < RawVec<T, N>::kWords; ++c)
    asm volatile("" : "+r"(raw.q[c].x), "+r"(raw.q[c].y), "+r"(raw.q[c].z), "+r"(raw.q[c].w));
}
template <class T, int N>
__device__ __forceinline__ typename vec_of<typename Mem<T>::val, N>::type widen_raw(const RawVec<T, N>& raw) {
  typename vec_of<typename Mem<T>::val, N>::type r;
  constexpr int kPer = 16 / (int)sizeof(T);
#pragma unroll
  for (int c = 0; c < RawVec<T, N>::kWords; ++c) unpack<T>(raw.q[c], &r.v[c * kPer]);
  return r;
}
template <class T, int N, bool FAST = false, class A>
__device__ __forceinline__ void stvec(T* p, int nvalid, const A& val) {
  using V = typename Mem<T>::val;
  constexpr int kPer = 16 / sizeof(T);
  if constexpr ((N % kPer) == 0 && (sizeof(T) == 2 || sizeof(T) == 4) && std::is_same<V, float>::value) {
    if (FAST || (nvalid >= N && (reinterpret_cast<uintptr_t>(p) & 15u) == 0)) {
      float f[N];
#pragma unroll
      for (int i = 0; i < N; ++i) f[i] = Cast<float>::from(at(val, i));
#pragma unroll
      for (int c = 0; c < N / kPer; ++c) stg_stream(p + c * kPer, pack<T>(&f[c * kPer]));
      return;
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < nvalid) Mem<T>::st(p + i, Cast<V>::from(at(val, i)));
}

// One element shared by all the elements a thread owns (an index or a per-row scale whose
// address does not change inside a vector): a single load, returned as a scalar, so that
// everything computed from it is scalar too.
template <class T>
__device__ __forceinline__ typename Mem<T>::val ld_uniform(const T* p, long long idx, bool valid,
                                                           typename Mem<T>::val other) {
  return valid ? Mem<T>::ld(p + idx) : other;
}
// Indirect access whose direct part is contiguous along the vector.  If every indirect
// operand turned out to be a scalar (it came from ld_uniform), the N elements are adjacent
// and move as one 128-bit access; otherwise one access per element.
template <class T, int N, bool FAST, class I, class M, class... U>
__device__ __forceinline__ auto igather(const T* p, const I& idx, const M& mask, typename Mem<T>::val other,
                                        int nvalid, const U&... indirect) {
  if constexpr (((rank<U>::n == 0) && ...) && rank<I>::n == N) {
    return ldvec<T, N, FAST, true>(p + at(idx, 0), nvalid);
  } else {
    return gather(p, idx, mask, other);
  }
}

// The same for rows off a 16-byte boundary (vectors that end with their row): the run is cut out of the words
// that cover it, which the lanes beside this one read as well.
template <class T, int N, class I, class M, class... U>
__device__ __forceinline__ auto igather_row(const T* p, const I& idx, const M& mask, typename Mem<T>::val other,
                                            int nvalid, const U&... indirect) {
  if constexpr (((rank<U>::n == 0) && ...) && rank<I>::n == N) return ldvec<T, N>(p + at(idx, 0), nvalid);
  else return gather(p, idx, mask, other);
}

// ---- bounds check of indirect indices (debug builds) ---------------------------------------
// A module generated with IXB_DEBUG_BOUNDS checks every data-dependent index against the
// extent it addresses (the reference asserts them on the device,
// inductor_x/codegen/triton.py:1666-1710).  A violation is counted, one offending value is
// kept, and the index is replaced by 0 so that the access stays inside the buffer; the
// launcher reads the two words after the launch and raises on the host.  Nothing traps.
#ifdef IXB_DEBUG_BOUNDS
static __device__ unsigned long long g_bounds_status[2];  // [violations, one offending index]
__device__ __forceinline__ long long checked_one(long long x, long long size) {
  if (x < 0 || x >= size) {
    atomicAdd(&g_bounds_status[0], 1ull);
    atomicExch(&g_bounds_status[1], (unsigned long long)x);
    return 0;
  }
  return x;
}
template <class I> __device__ __forceinline__ auto checked_index(const I& idx, long long size) {
  return map1<typename ires<rank<I>::n>::type>([size](long long x) { return checked_one(x, size); }, idx);
}
// host: fetch and clear the status words of this module (synchronises the device)
inline int read_bounds_status(unsigned long long* out) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_bounds_status, 2 * sizeof(unsigned long long));
  if (e != cudaSuccess) return (int)e;
  const unsigned long long zero[2] = {0ull, 0ull};
  return (int)cudaMemcpyToSymbol(g_bounds_status, zero, sizeof(zero));
}
#endif

// ---- pointwise family -------------------------------------------------------------------
// CTAs of `kern` that fit on the device at once.  Persistent kernels launch exactly this
// many (or fewer, if the work is smaller): a grid of a few waves would leave the last wave
// partly empty.
template <class K> inline long long resident_ctas(K kern, int threads) {
  int dev = 0, sms = 148, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, 0) != cudaSuccess || n < 1) n = 1;
  return (long long)sms * n;
}

// true when every pointer argument of a generated module is 16-byte aligned
inline bool pointers_aligned(void* const* ptrs, int n) {
  for (int i = 0; i < n; ++i)
    if (reinterpret_cast<uintptr_t>(ptrs[i]) & 15u) return false;
  return true;
}

template <class Body, bool ALIGNED>
__global__ void __launch_bounds__(256) pointwise_gen_kernel(const Body body, const long long xnumel) {
  constexpr int V = Body::kVec;
  const long long ntiles = (xnumel + V - 1) / V;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += stride) {
    // Body::first_of maps the thread's slot to the first element of its vector: t * V, or the
    // transposing order (consecutive lanes along the axis the loads are contiguous in)
    const long long xbase = body.first_of(t);
    const long long left = xnumel - xbase;
    if (ALIGNED && left >= V) body.template tile<true>(xbase, V);
    else body.template tile<false>(xbase, left >= V ? V : (int)left);
  }
}
// ---- rows of odd length ----------------------------------------------------------------------
// The flat index in rows of LB elements, LB no whole number of vectors: the vectors are those of the flat
// index, cut at the ends of the rows, so that inside a vector a per-column operand or a gathered row is one run
// and a per-row operand one value.  Of the two parts of a vector that two rows share each is stored
// element by element.
template <class Body, int LB, bool ALIGNED>
__global__ void __launch_bounds__(256) pointwise_rows_gen_kernel(const Body body, const long long slots) {
  constexpr int V = Body::kVec, K = (LB + V - 1 + V - 1) / V;  // vectors that a row may touch
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < slots; t += (long long)gridDim.x * blockDim.x) {
    const unsigned row = (unsigned)t / K, k = (unsigned)t % K;
    const long long first = (long long)row * LB;
    int x = (int)k * V - (int)((unsigned)first % V), n = V;
    if (x < 0) {
      n += x;
      x = 0;
    }
    if (x + n > LB) n = LB - x;
    if (n <= 0) continue;
    // one form for the whole warp: lanes at an end of a row would have the others wait for a second pass over the body
    // (gelu(x + w) of 2^24 bf16 in rows of 333 39.5 -> 30.4 us, gather of such rows 9.4 -> 8.7)
    if (ALIGNED && __all_sync(__activemask(), n == V)) body.template tile<true>(first + x, V);
    else body.template tile<false>(first + x, n);
  }
}

// ---- transposes: a register tile per thread ---------------------------------------------------
// A pointwise group that stores along the flat index but reads an operand that is contiguous
// along another digit C of it (a transpose) gives every thread a V x kC micro-tile of that
// operand: V 128-bit loads, each kC consecutive elements along C (one for each of the V
// positions of the thread's vector along the flat index), then kC output vectors - element ci
// of every loaded row is the operand of output vector ci.  Both sides move 128 bits per access
// and the extraction costs what widening a half would cost anyway.  Lanes are arranged 4 along
// the flat index by 8 along C, so a warp reads four full 128-byte lines per load instruction
// and writes 64-byte runs.  This is what the reference's second set of index variables and
// `.permute(1, 0)` on the tile are for (inductor_x/codegen/triton.py:856-888, 1303-1332).
template <class U, int V> struct TileRaw {
  static constexpr int kC = 16 / (int)sizeof(U);
  uint4 q[V];
};
template <class U, int V, class I>
__device__ __forceinline__ void fetch_tile(TileRaw<U, V>& r, const U* p, const I& idx) {
#pragma unroll
  for (int j = 0; j < V; ++j) r.q[j] = ldg_stream(p + at(idx, j));
}
template <class U> __device__ __forceinline__ float tile_elem(const uint4& q, int ci);
template <> __device__ __forceinline__ float tile_elem<float>(const uint4& q, int ci) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  return __uint_as_float(w[ci]);
}
template <> __device__ __forceinline__ float tile_elem<bf16>(const uint4& q, int ci) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  return __uint_as_float((ci & 1) ? (w[ci >> 1] & 0xffff0000u) : (w[ci >> 1] << 16));
}
template <> __device__ __forceinline__ float tile_elem<f16>(const uint4& q, int ci) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  const __half2 h = *reinterpret_cast<const __half2*>(&w[ci >> 1]);
  return (ci & 1) ? __high2float(h) : __low2float(h);
}
// element ci of every row of the tile, widened: the operand of output vector ci
template <class U, int V> __device__ __forceinline__ vf<V> take(const TileRaw<U, V>& t, int ci) {
  vf<V> r;
#pragma unroll
  for (int j = 0; j < V; ++j) r.v[j] = tile_elem<U>(t.q[j], ci);
  return r;
}

template <class Body>
__global__ void __launch_bounds__(256) pointwise_tile_gen_kernel(const Body body, const long long xnumel) {
  constexpr int V = Body::kVec;
  constexpr int C = Body::kTileC;
  const long long ntiles = xnumel / ((long long)V * C);     // exact by construction of the order
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += stride) {
    const long long x0 = body.first_of_tile(t);
    typename Body::Tile raw;
    body.fetch_tile(x0, raw);
#pragma unroll
    for (int ci = 0; ci < C; ++ci) body.template tile<true, true>(x0 + ci * Body::kStepC, V, raw, ci);
  }
}
// Grid of a kernel that moves every byte once and holds nothing from one vector to the next: a block
// for every 256 vectors, which the hardware starts in order as others end.  Blocks that are resident for the
// whole launch and stride through the tensor drift apart instead, and the DRAM pages that are open
// at a time spread over all they have reached: a copy of 512 MB takes 160 us this way and 178 - 186
// (148 x 8 and x 4 blocks) the other, the transpose of 4096 x 512 x 128 fp16 157 against 199, an inner
// permute of the same size 170.5 against 175.5.  Rows gathered through an index are in no order anyway and
// keep the resident grid (23.8 against 26.0 us for 262144 rows of 256 bytes out of 2^20), and so does what stays in L2
// (Body::kStream: the threads from which this holds, 0 for never; the generator's _stream_threads says how it is chosen).
template <class Body> inline long long stream_grid(long long threads, long long resident) {
  long long grid = (threads + 255) / 256;
  const long long most = Body::kStream > 0 && threads >= Body::kStream ? 0x7fffffffLL : resident;
  if (grid > most) grid = most;
  return grid < 1 ? 1 : grid;
}
// ---- transposes by way of shared memory ---------------------------------------------------------
// The same where the extents do not divide into register tiles or rows start off a 16-byte boundary on
// either side.  A block has NK vectors of up to 120 (60 of 32 bits) output rows; of each of the NK * V + V - 1
// source rows these may want it copies the aligned words that hold some element of it (16 words a row
// at most, cp.async), and an output vector is gathered from the V rows.  Output vectors are those of memory:
// a row's first one begins before the row where the row does not begin on a boundary, so that what
// is stored is whole 16-byte words but for the ends of a row.  Words are swizzled by the row's vector:
// the lanes of a warp, eight vectors by four rows of output, read eight rows V apart without a bank conflict
// (rows off a boundary shift against each other by a word now and then).  Bound: the gathering, a
// shared load and some ten instructions an element.  Measured: see launch_pointwise_smem.
constexpr int kTileWords = 16;
template <class U, int V, int ROWS, int STRIDE> struct TileSmem {
  const uint4* words = nullptr;  // [ROWS + V][kTileWords], the last V of them never written
  int row = 0, col = 0;          // of the vector's first element
  int off = 0;                   // elements between the first word of row 0 and its first element
};
template <class U, int V, int ROWS, int STRIDE>
__device__ __forceinline__ vf<V> take(const TileSmem<U, V, ROWS, STRIDE>& t, int) {
  constexpr int kPer = 16 / (int)sizeof(U);
  const unsigned char* from = reinterpret_cast<const unsigned char*>(t.words + t.row * kTileWords);
  const int off = t.off + t.row * (STRIDE % kPer);
  vf<V> r;
#pragma unroll
  for (int j = 0; j < V; ++j) {  // (elements past the end of a row come from the rows behind the tile, and are masked)
    const int pos = ((off + j * (STRIDE % kPer)) & (kPer - 1)) + t.col;
    const int key = (t.row + j) / V & 7;
    r.v[j] = Mem<U>::ld(reinterpret_cast<const U*>(from + j * (16 * kTileWords) + ((pos * (int)sizeof(U)) ^ (key * 16))));
  }
  return r;
}
// Source rows of one operand into shared memory: row r of the tile begins at from + (r - first) * STRIDE;
// rows [lo, hi) of it exist, and `count` elements of each are wanted.
template <class U, int V, int ROWS, int STRIDE>
__device__ __forceinline__ TileSmem<U, V, ROWS, STRIDE> copy_tile(uint4* words, const U* from, int lo, int hi, int count) {
  constexpr int kPer = 16 / (int)sizeof(U);
  for (int i = threadIdx.x; i < ROWS * kTileWords; i += blockDim.x) {
    const int r = i / kTileWords, w = i % kTileWords;
    if (r < lo || r >= hi) continue;
    const U* row = from + (long long)r * STRIDE;
    const int off = off_boundary(row);
    if (w * kPer < off + count)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(words + r * kTileWords + (w ^ ((r / V) & 7)))),
                   "l"(row - off + w * kPer)
                   : "memory");
  }
  TileSmem<U, V, ROWS, STRIDE> t;
  t.words = words;
  t.off = off_boundary(from);
  return t;
}
// LB, DC, LC: digits of the flat index (output rows of LB elements, the loads' axis LC of them DC apart)
template <class Body, int LB, long long DC, int LC, int NK>
__global__ void __launch_bounds__(256) pointwise_smem_gen_kernel(const Body body) {
  constexpr int V = Body::kVec, TX = NK * V, ROWS = TX + V - 1;
  constexpr int NX = (LB + V - 1 + TX - 1) / TX;
  constexpr int NC = (LC + Body::kTileCols - 1) / Body::kTileCols, TC = (LC + NC - 1) / NC;
  __shared__ uint4 words[Body::kTileOps][(ROWS + V) * kTileWords];
  unsigned b = blockIdx.x;
  const int c0 = (int)(b % NC) * TC;
  b /= NC;
  const int x0 = (int)(b % NX) * TX;
  b /= NX;
  const unsigned mid = b % (unsigned)(DC / LB), outer = b / (unsigned)(DC / LB);
  const long long first = (long long)outer * (DC * LC) + c0 * DC + (long long)mid * LB;  // flat index of (x 0, c0)
  const int cols = LC - c0 < TC ? LC - c0 : TC;
  // row r of the tile is element x0 - (V - 1) + r of the output rows
  typename Body::Tile raw = body.copy_tiles(words, first, x0 - (V - 1), cols);
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int it = threadIdx.x >> 5; it < (cols + 3) / 4 * (NK / 8); it += 8) {
    const int c = it / (NK / 8) * 4 + (lane >> 3), k = it % (NK / 8) * 8 + (lane & 7);
    if (c >= cols) continue;
    const long long row = first + c * DC;
    int x = x0 + k * V - (int)((unsigned long long)row % V), n = V;
    if (x < 0) {
      n += x;
      x = 0;
    }
    if (x + n > LB) n = LB - x;
    if (n <= 0) continue;
    raw.at(x - (x0 - (V - 1)), c);
    if (n == V) body.template tile<true, true>(row + x, V, raw);
    else body.template tile<false, true>(row + x, n, raw);
  }
}

template <class Body> int launch_pointwise(const Body& body, long long xnumel, void* stream, bool aligned);
template <class Body, int LB> int launch_pointwise_rows(const Body& body, long long xnumel, void* stream, bool aligned) {
  if (xnumel <= 0) return 0;
  const long long slots = xnumel / LB * ((LB + 2 * (Body::kVec - 1)) / Body::kVec);
  if (slots > 0x7fffffffLL) return (int)cudaErrorInvalidValue;  // (the generator keeps the index below 2^31, and rows past a vector)
  static const long long cap_a = resident_ctas(pointwise_rows_gen_kernel<Body, LB, true>, 256);
  static const long long cap_u = resident_ctas(pointwise_rows_gen_kernel<Body, LB, false>, 256);
  const long long grid = stream_grid<Body>(slots, aligned ? cap_a : cap_u);
  if (aligned) pointwise_rows_gen_kernel<Body, LB, true><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(body, slots);
  else pointwise_rows_gen_kernel<Body, LB, false><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(body, slots);
  return (int)cudaGetLastError();
}
// Per-element gathers -> by way of shared memory: 200 x 1000 x 1000 fp16 775 -> 122 us (the floor of its bytes),
// 300 x 701 x 333 fp32 345 -> 88 (86), 500 x 511 x 513 bf16 472 -> 138 (80: rows off a boundary on both sides),
// 3000 x 100 x 100 fp16 118 -> 39 (18: a fifth of the rows' last vectors are parts), 2000 x 64 x 65 29 -> 10.6 (5).
template <class Body, int LB, long long DC, int LC, int NK>
int launch_pointwise_smem(const Body& body, long long xnumel, void* stream, bool aligned) {
  if (xnumel <= 0) return 0;
  constexpr int TX = NK * Body::kVec, NX = (LB + Body::kVec - 1 + TX - 1) / TX, NC = (LC + Body::kTileCols - 1) / Body::kTileCols;
  const long long blocks = xnumel / LB / LC * NX * NC;
  if (!aligned || blocks > 0x7fffffffLL) return launch_pointwise(body, xnumel, stream, aligned);
  pointwise_smem_gen_kernel<Body, LB, DC, LC, NK><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(body);
  return (int)cudaGetLastError();
}
// tiles when every pointer is 16-byte aligned, the plain kernel (per-element gathers) otherwise
template <class Body> int launch_pointwise_tile(const Body& body, long long xnumel, void* stream, bool aligned) {
  if (xnumel <= 0) return 0;
  if (!aligned) return launch_pointwise(body, xnumel, stream, false);
  static const long long cap = resident_ctas(pointwise_tile_gen_kernel<Body>, 256);
  const long long grid = stream_grid<Body>(xnumel / ((long long)Body::kVec * Body::kTileC), cap);
  pointwise_tile_gen_kernel<Body><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(body, xnumel);
  return (int)cudaGetLastError();
}

template <class Body> int launch_pointwise(const Body& body, long long xnumel, void* stream, bool aligned = false) {
  if (xnumel <= 0) return 0;
  static const long long cap_a = resident_ctas(pointwise_gen_kernel<Body, true>, 256);
  static const long long cap_u = resident_ctas(pointwise_gen_kernel<Body, false>, 256);
  const long long grid = stream_grid<Body>((xnumel + Body::kVec - 1) / Body::kVec, aligned ? cap_a : cap_u);
  if (aligned) pointwise_gen_kernel<Body, true><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(body, xnumel);
  else pointwise_gen_kernel<Body, false><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(body, xnumel);
  return (int)cudaGetLastError();
}

// ---- persistent row family ---------------------------------------------------------------
// The generated body sees a context that maps vector element e = i * kVec + j of this
// thread to column vec_col(i) + j of the row, exactly as RowCtx does for the prebuilt bodies.
// COLS is the row length when it is known at compile time (0: at run time, or walked in chunks).
// Vectors that every thread of the team has inside the row - all of them when the length is
// TEAM * VPT * kVec (FULL), all but the last one or two of an odd length - then need no validity
// test and fold in packed pairs; without it every element of an odd row paid one per fold.
//
// A generated row body has four parts:
//   Consts / init(c, k)            operands that do not change from row to row (per-column
//                                  scales and shifts): loaded and widened once per thread
//   Raw / fetch(c, x, raw)         the 128-bit vectors of the operands streamed once per row,
//                                  requested one row ahead of the arithmetic
//   row<STAGED>(c, k, x, raw, cols) the math of row x; STAGED says whether `raw` was fetched
//                                  (aligned operands) or the body loads for itself; `cols` holds
//                                  the thread's part of sums over the rows (Cols, clear, flush)
//   prefetch(c, x)                 L2 prefetch of the streamed operands of a later row

// raw 128-bit vectors of one row-shaped operand of storage type U, as one thread holds them
template <class U, int VPT, int KVEC> struct RawRow {
  static constexpr int kChunks = KVEC * (int)sizeof(U) / 16;  // 128-bit words per vector
  static_assert(kChunks >= 1, "staged operands are at least as wide as the row's vector type");
  uint4 q[VPT][kChunks];
};

// the same for rows that may start anywhere: the aligned words that cover the thread's vectors,
// one more than the vectors themselves fill
template <class U, int VPT, int KVEC> struct RawRowU {
  static constexpr int kChunks = KVEC * (int)sizeof(U) / 16;
  static_assert(kChunks >= 1, "staged operands are at least as wide as the row's vector type");
  uint4 q[VPT][kChunks + 1];
};

// exact 64-bit integer reduction operators
struct ISum {
  static __device__ __forceinline__ long long id() { return 0; }
  static __device__ __forceinline__ long long f(long long a, long long b) { return a + b; }
};
struct IProd {
  static __device__ __forceinline__ long long id() { return 1; }
  static __device__ __forceinline__ long long f(long long a, long long b) { return a * b; }
};
struct IMax {
  static __device__ __forceinline__ long long id() { return (long long)0x8000000000000000ull; }
  static __device__ __forceinline__ long long f(long long a, long long b) { return a > b ? a : b; }
};
struct IMin {
  static __device__ __forceinline__ long long id() { return 0x7fffffffffffffffLL; }
  static __device__ __forceinline__ long long f(long long a, long long b) { return a < b ? a : b; }
};

// references to up to two float vectors (operands of the online-softmax riders)
template <int E, int K> struct VecRefs {
  const vf<E>* p[K > 0 ? K : 1];
};
template <int E> __device__ __forceinline__ VecRefs<E, 0> refs() { return VecRefs<E, 0>{{nullptr}}; }
template <int E> __device__ __forceinline__ VecRefs<E, 1> refs(const vf<E>& a) { return VecRefs<E, 1>{{&a}}; }
template <int E> __device__ __forceinline__ VecRefs<E, 2> refs(const vf<E>& a, const vf<E>& b) {
  return VecRefs<E, 2>{{&a, &b}};
}

// one warp-level sum of K values: every lane receives every total
template <int K> __device__ __forceinline__ void warp_sum(float (&v)[K]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] += __shfl_xor_sync(kFull, v[k], o);
}
// Two or three sums of a warp: lanes 0, 8 and 16 hold them.  Each step that halves the lanes a value is
// spread over halves the values as well: six shuffles in place of ten or fifteen.
__device__ __forceinline__ float warp_sum_split(float a, float b, float c) {
  const int lane = threadIdx.x & 31;
  // lanes of the upper half go on with c (and nothing beside it), the others with a and b
  const bool up = lane & 16;
  const float other = __shfl_xor_sync(kFull, up ? a : c, 16);
  const float a1 = (up ? c : a) + other;
  const float b1 = b + __shfl_xor_sync(kFull, b, 16);   // (of use to the lower half alone)
  const bool odd = lane & 8;
  const float send = odd ? a1 : (up ? a1 : b1);
  const float got = __shfl_xor_sync(kFull, send, 8);
  float t = (up ? a1 : (odd ? b1 : a1)) + got;
  t += __shfl_xor_sync(kFull, t, 4);
  t += __shfl_xor_sync(kFull, t, 2);
  t += __shfl_xor_sync(kFull, t, 1);
  return t;
}
// NaN-propagating maximum / minimum of a warp in one instruction
__device__ __forceinline__ float warp_max_nan(float v) {
  float r;
  asm volatile("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_min_nan(float v) {
  float r;
  asm volatile("redux.sync.min.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
template <class Op> __device__ __forceinline__ float warp_all(float v) {
  if constexpr (std::is_same<Op, MaxOp>::value) return warp_max_nan(v);
  else if constexpr (std::is_same<Op, MinOp>::value) return warp_min_nan(v);
  else return warp_reduce<Op>(v);
}

// SHIFT: the thread's vectors are those of memory, not of the row: vector 0 of lane 0 is the aligned one
// that holds the row's first element, `off` elements into it, and column vec_col(0) is -off there.
template <typename T, int TEAM, int TEAMS, int VPT, int COLS = 0, bool SHIFT = false>
struct GenRowCtx : RowCtx<T, TEAM, TEAMS, VPT, false> {
  using Base = RowCtx<T, TEAM, TEAMS, VPT, false>;
  static constexpr int kE = VPT * Base::kVec;
  static constexpr bool FULL = !SHIFT && COLS == TEAM * VPT * Base::kVec;
  // vector i of every thread lies inside the row
  static __device__ __forceinline__ constexpr bool full(int i) {
    return COLS >= (i + 1) * TEAM * Base::kVec && !(SHIFT && i == 0);
  }
  __device__ __forceinline__ int ncols() const { return COLS > 0 ? COLS : this->cols; }
  static constexpr int kGroup = TEAM < 32 ? TEAM : 32;  // lanes of one warp that share a row
  static constexpr int kW = Base::kWarpsPerTeam;        // warps per team (0 for sub-warp teams)
  static constexpr int kChains = (kE / 2) >= 4 ? 4 : ((kE / 2) >= 2 ? 2 : 1);  // accumulator chains
  // Teams narrower than a warp share their warp's control flow: a team whose row index
  // ran past the end repeats the last row with `live` false, which masks its stores.
  bool live = true;
  // Rows longer than the team holds are walked in chunks of kCap columns (looped reduction):
  // chunk0 is the first column of the current chunk.  vec_col shadows the base-class version,
  // so every access below is relative to the chunk.
  int chunk0 = 0;
  static constexpr int kCap = TEAM * VPT * Base::kVec;
  int off = 0;
  __device__ __forceinline__ int vec_col(int i) const {
    return chunk0 + (this->lane + i * TEAM) * Base::kVec - (SHIFT ? off : 0);
  }
  __device__ __forceinline__ int nchunks() const { return (this->cols + kCap - 1) / kCap; }
  __device__ __forceinline__ void set_chunk(int chunk) { chunk0 = chunk * kCap; }
  // Per-column operands that are not kept in registers live in a CTA-wide shared-memory
  // table, widened to fp32 once at start-up.  Slot s is laid out [quad][vector] (a quad = four
  // floats) so that consecutive lanes read consecutive 16-byte words: no bank conflicts.
  const float4* ktab = nullptr;
  static constexpr int kQuads = Base::kVec / 4 > 0 ? Base::kVec / 4 : 1;
  static constexpr int kTabVecs = TEAM * VPT;   // vectors of one row at full capacity

  template <int SLOT, class U> __device__ __forceinline__ void fill_sconst(const U* rowp) const {
    static_assert(Base::kVec % 4 == 0, "shared-memory operands need whole quads per vector");
    float4* tab = const_cast<float4*>(ktab) + SLOT * kQuads * kTabVecs;
    if constexpr (SHIFT) {
      for (int v = threadIdx.x; v < kTabVecs; v += blockDim.x)
#pragma unroll
        for (int q = 0; q < kQuads; ++q) {
          float part[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int col = v * Base::kVec + 4 * q + j - off;
            part[j] = (unsigned)col < (unsigned)ncols() ? Cast<float>::from(Mem<U>::ld(rowp + col)) : 0.f;
          }
          tab[q * kTabVecs + v] = make_float4(part[0], part[1], part[2], part[3]);
        }
      return;
    }
    for (int v = threadIdx.x; v < kTabVecs; v += blockDim.x) {
      const int c0 = v * Base::kVec;
      const int left = this->cols - c0;
      const auto part = ldvec<U, Base::kVec, false, false, !FULL>(rowp + (left > 0 ? c0 : 0), left > 0 ? left : 0);
#pragma unroll
      for (int q = 0; q < kQuads; ++q)
        tab[q * kTabVecs + v] = make_float4(part.v[4 * q], part.v[4 * q + 1], part.v[4 * q + 2], part.v[4 * q + 3]);
    }
  }
  template <int SLOT> __device__ __forceinline__ vf<kE> sconst() const {
    const float4* tab = ktab + SLOT * kQuads * kTabVecs;
    vf<kE> r;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = this->lane + i * TEAM;
#pragma unroll
      for (int q = 0; q < kQuads; ++q) {
        const float4 f = tab[q * kTabVecs + v];
        r.v[i * Base::kVec + 4 * q] = f.x;
        r.v[i * Base::kVec + 4 * q + 1] = f.y;
        r.v[i * Base::kVec + 4 * q + 2] = f.z;
        r.v[i * Base::kVec + 4 * q + 3] = f.w;
      }
    }
    return r;
  }

  __device__ __forceinline__ bool leader() const { return this->lane == 0 && live; }
  // element j of vector i lies inside the row
  __device__ __forceinline__ bool inside(int i, int j) const {
    // (one test with a constant each, where the length is one: the first vector of a row off a boundary can only
    // begin before it and the others only end behind it, a row of whole vectors ends with one)
    if constexpr (SHIFT && COLS >= TEAM * Base::kVec) return full(i) || (i == 0 ? this->vec_col(0) >= -j : this->vec_col(i) < COLS - j);
    if constexpr (!SHIFT && COLS > 0 && COLS % Base::kVec == 0) return full(i) || this->vec_col(i) < COLS;
    if constexpr (SHIFT) return full(i) || (unsigned)(this->vec_col(i) + j) < (unsigned)ncols();
    return full(i) || this->vec_col(i) + j < ncols();
  }
  // vector i may hold elements that are not the row's
  __device__ __forceinline__ bool cut(int i) const {
    if constexpr (SHIFT && COLS >= TEAM * Base::kVec) return !full(i) && (i == 0 ? this->vec_col(0) < 0 : this->vec_col(i) > COLS - Base::kVec);
    return !full(i) && ((SHIFT && this->vec_col(i) < 0) || this->vec_col(i) + Base::kVec > ncols());
  }
  __device__ __forceinline__ vi<kE> rindex() const {
    vi<kE> r;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j) r.v[i * Base::kVec + j] = this->vec_col(i) + j;
    return r;
  }
  __device__ __forceinline__ vb<kE> rmask() const {
    vb<kE> r;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j) r.v[i * Base::kVec + j] = live && inside(i, j);
    return r;
  }
  // row-contiguous operand of storage type U starting at `rowp`
  template <bool CUT = true, class U> __device__ __forceinline__ auto load_row(const U* rowp) const {
    using V = typename Mem<U>::val;
    typename vec_of<V, kE>::type r;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c0 = this->vec_col(i);
      if (SHIFT && cut(i)) {
#pragma unroll
        for (int j = 0; j < Base::kVec; ++j)
          r.v[i * Base::kVec + j] = inside(i, j) ? Mem<U>::ld(rowp + c0 + j) : V();
        continue;
      }
      const int left = full(i) ? Base::kVec : ncols() - c0;
      auto part = ldvec<U, Base::kVec, false, false, CUT>(rowp + c0, left > 0 ? left : 0);
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j) r.v[i * Base::kVec + j] = part.v[j];
    }
    return r;
  }
  // the same operand as raw 128-bit vectors (aligned rows only; vectors past the end of a
  // ragged row read as zero): requested a row ahead, widened when the row is worked on
  template <class U> __device__ __forceinline__ void fetch_row(const U* rowp, RawRow<U, VPT, Base::kVec>& raw) const {
    constexpr int kC = RawRow<U, VPT, Base::kVec>::kChunks;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c0 = this->vec_col(i);
#pragma unroll
      for (int k = 0; k < kC; ++k) {
        if constexpr (SHIFT) {
          // (the words at the two ends are written by the blocks of the neighbouring rows as well, in
          // place as it may be: no __ldg)
          constexpr int kPer = 16 / (int)sizeof(U);
          const int w0 = c0 + k * kPer;
          raw.q[i][k] = (full(i) || (w0 + kPer > 0 && w0 < ncols())) ? ldg_word_stream(rowp + w0) : make_uint4(0, 0, 0, 0);
        } else {
          raw.q[i][k] = (full(i) || c0 < ncols()) ? ldg_stream(reinterpret_cast<const uint4*>(rowp + c0) + k)
                                                 : make_uint4(0, 0, 0, 0);
        }
      }
    }
  }
  template <class U> __device__ __forceinline__ vf<kE> widen(const RawRow<U, VPT, Base::kVec>& raw) const {
    constexpr int kC = RawRow<U, VPT, Base::kVec>::kChunks;
    constexpr int kPer = 16 / (int)sizeof(U);
    vf<kE> r;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int k = 0; k < kC; ++k) unpack<U>(raw.q[i][k], &r.v[i * Base::kVec + k * kPer]);
    if constexpr (SHIFT) {
#pragma unroll
      for (int i = 0; i < VPT; ++i)
        if (cut(i)) {
#pragma unroll
          for (int j = 0; j < Base::kVec; ++j)
            if (!inside(i, j)) r.v[i * Base::kVec + j] = 0.f;
        }
    }
    return r;
  }
  // Rows that start off a 16-byte boundary (an odd row length moves every row) where the block cannot
  // keep to one offset (SHIFT) - run-time lengths, operands of several pitches: the words that
  // cover a thread's vectors are fetched aligned - the one it shares with the next lane comes
  // out of L1 - and shifted into place when the row is worked on.  Only words that hold an
  // element of the row are read.  Element-wise loads of such rows touch every line eight times
  // and cannot be requested a row ahead: softmax -> LayerNorm of 20011 x 1537 fp16 took 104 us
  // with them, 90 us this way, 73 us with the length known at compile time (COLS), 59 us in the
  // launch shape that measures best (six teams of 64 threads with four vectors each), 57 us with
  // plain loads of the per-column operands.
  template <class U> __device__ __forceinline__ void fetch_row(const U* rowp, RawRowU<U, VPT, Base::kVec>& raw) const {
    constexpr int kC = RawRowU<U, VPT, Base::kVec>::kChunks;
    constexpr int kPer = 16 / (int)sizeof(U);
    const int off = off_boundary(rowp);     // whole vectors lie between the row start and any other vector
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c0 = this->vec_col(i) - off;   // column of the first element of the first word
#pragma unroll
      for (int k = 0; k <= kC; ++k) {
        const bool need = (full(i) || (c0 + off < ncols() && c0 + k * kPer < ncols())) && (k < kC || off > 0);
        raw.q[i][k] = need ? ldg_shared_word(rowp + (c0 + k * kPer)) : make_uint4(0, 0, 0, 0);
      }
    }
  }
  template <class U> __device__ __forceinline__ vf<kE> widen(const RawRowU<U, VPT, Base::kVec>& raw, const U* rowp) const {
    constexpr int kC = RawRowU<U, VPT, Base::kVec>::kChunks;
    constexpr int kPer = 16 / (int)sizeof(U);
    const int off = off_boundary(rowp);
    vf<kE> r;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
#pragma unroll
      for (int k = 0; k < kC; ++k)
        unpack<U>(shift_words<U>(raw.q[i][k], raw.q[i][k + 1], off), &r.v[i * Base::kVec + k * kPer]);
      if (!full(i) && this->vec_col(i) + Base::kVec > ncols()) {     // what follows the row is not its business
#pragma unroll
        for (int j = 0; j < Base::kVec; ++j)
          if (!inside(i, j)) r.v[i * Base::kVec + j] = 0.f;
      }
    }
    return r;
  }
  template <bool STAGED, class U>
  __device__ __forceinline__ vf<kE> operand(const RawRowU<U, VPT, Base::kVec>& raw, const U* rowp) const {
    if constexpr (STAGED) return widen<U>(raw, rowp);
    else return load_row(rowp);
  }
  // Store to such a row: a lane owns the aligned word that ends in its vector, i.e. the last
  // elements of the vector before it (from the lane before it) and the first of its own.  The
  // ends of a warp's run and of the row are written element by element.
  template <class U, class A> __device__ __forceinline__ void put_row_any(U* rowp, const A& val) const {
    if constexpr (std::is_same<typename Mem<U>::val, float>::value && (sizeof(U) == 2 || sizeof(U) == 4) &&
                  std::is_same<A, vf<kE>>::value) {
      constexpr int kPer = 16 / (int)sizeof(U);
      constexpr int kC = Base::kVec / kPer;
      const int off = off_boundary(rowp);
      const int wl = this->lane & (kGroup - 1);
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        uint4 w[kC + 1];       // the vector's words behind the last word of the lane before
#pragma unroll
        for (int k = 0; k < kC; ++k) w[k + 1] = pack<U>(&val.v[i * Base::kVec + k * kPer]);
        w[0].x = __shfl_up_sync(kFull, w[kC].x, 1, kGroup);
        w[0].y = __shfl_up_sync(kFull, w[kC].y, 1, kGroup);
        w[0].z = __shfl_up_sync(kFull, w[kC].z, 1, kGroup);
        w[0].w = __shfl_up_sync(kFull, w[kC].w, 1, kGroup);
        if (!live) continue;
#pragma unroll
        for (int k = 0; k < kC; ++k) {
          const int col = this->vec_col(i) + k * kPer - off;
          const uint4 v = off == 0 ? w[k + 1] : shift_words<U>(w[k], w[k + 1], kPer - off);
          const int first = (k > 0 || wl > 0) ? 0 : off;
          if (first == 0 && (full(i) || col + kPer <= ncols())) stg_stream(rowp + col, v);
          else put_elements(rowp + col, v, first, ncols() - col);
        }
        // the last lane of a run has nobody behind it to write the end of its vector
        if (off > 0 && wl == kGroup - 1) {
          const int col = this->vec_col(i) + Base::kVec - off;
          const int left = ncols() - col;
          put_elements(rowp + col, shift_words<U>(w[kC], w[kC], kPer - off), 0, left < off ? left : off);
        }
      }
    } else {
      store_row(rowp, val);
    }
  }
  // a streamed operand inside row(): from the fetched vectors, or loaded on the spot
  template <bool STAGED, class U>
  __device__ __forceinline__ vf<kE> operand(const RawRow<U, VPT, Base::kVec>& raw, const U* rowp) const {
    if constexpr (STAGED) return widen<U>(raw);
    else return load_row(rowp);
  }
  // ask L2 for the lines of a row-contiguous operand this thread will load later: the
  // thread whose vector opens a 128-byte line (or the row itself) issues the prefetch
  template <class U> __device__ __forceinline__ void prefetch_row(const U* rowp) const {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c0 = this->vec_col(i);
      const U* p = rowp + c0;
      const bool opens = (reinterpret_cast<unsigned long long>(p) & 127ull) < Base::kVec * sizeof(U) || c0 <= 0;
      if (c0 < this->cols && opens) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
    }
  }
  template <class U, class A> __device__ __forceinline__ void store_row(U* rowp, const A& val) const {
    using V = typename Mem<U>::val;
    if (!live) return;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c0 = this->vec_col(i);
      if (SHIFT && cut(i)) {
#pragma unroll
        for (int j = 0; j < Base::kVec; ++j)
          if (inside(i, j)) Mem<U>::st(rowp + c0 + j, Cast<V>::from(at(val, i * Base::kVec + j)));
        continue;
      }
      const int left = full(i) ? Base::kVec : ncols() - c0;
      typename vec_of<V, Base::kVec>::type part;
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j) part.v[j] = Cast<V>::from(at(val, i * Base::kVec + j));
      stvec<U, Base::kVec>(rowp + c0, left > 0 ? left : 0, part);
    }
  }
  // aligned rows: one 128-bit streaming store per vector, no address test
  template <bool STAGED, class U, class A> __device__ __forceinline__ void put_row(U* rowp, const A& val) const {
    if constexpr (STAGED && std::is_same<typename Mem<U>::val, float>::value && (sizeof(U) == 2 || sizeof(U) == 4) &&
                  std::is_same<A, vf<kE>>::value) {
      if (!live) return;
      constexpr int kPer = 16 / (int)sizeof(U);
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int c0 = this->vec_col(i);
        if (SHIFT && cut(i)) {
          if (c0 >= ncols()) continue;
#pragma unroll
          for (int j = 0; j < Base::kVec; ++j)
            if (inside(i, j)) Mem<U>::st(rowp + c0 + j, val.v[i * Base::kVec + j]);
          continue;
        }
        if (full(i) || c0 < ncols()) {
#pragma unroll
          for (int k = 0; k < Base::kVec / kPer; ++k)
            stg_stream(rowp + c0 + k * kPer, pack<U>(&val.v[i * Base::kVec + k * kPer]));
        }
      }
    } else {
      store_row(rowp, val);
    }
  }

  // rows that may start off a boundary: whole vectors of memory where the block works in those
  template <bool STAGED, class U, class A> __device__ __forceinline__ void put_row_shifted(U* rowp, const A& val) const {
    if constexpr (SHIFT) put_row<STAGED>(rowp, val);
    else put_row_any(rowp, val);
  }

  // ---- sums over the rows -----------------------------------------------------------------
  // What this thread has summed for its columns, over the teams of the block (team after team, through
  // `tab`, which nothing else uses any more) and into the block's row of partial sums.
  __device__ __forceinline__ void flush_column(const vf<kE>& sum, float4* tab, float* partial) const {
    vf<kE> a = sum;
#pragma unroll 1
    for (int t = 0; t < TEAMS; ++t) {
      if (TEAMS > 1) __syncthreads();
      if (this->team != t) continue;
#pragma unroll
      for (int i = 0; i < VPT; ++i)
#pragma unroll
        for (int q = 0; q < kQuads; ++q) {
          float4& mine = tab[q * kTabVecs + this->lane + i * TEAM];
          float* v = &a.v[i * Base::kVec + 4 * q];
          if (t > 0) {
            const float4 p = mine;
            v[0] += p.x;
            v[1] += p.y;
            v[2] += p.z;
            v[3] += p.w;
          }
          if (t < TEAMS - 1) {
            mine = make_float4(v[0], v[1], v[2], v[3]);
          } else if (!SHIFT && !cut(i)) {
            *reinterpret_cast<float4*>(partial + this->vec_col(i) + 4 * q) = make_float4(v[0], v[1], v[2], v[3]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (inside(i, 4 * q + j)) partial[this->vec_col(i) + 4 * q + j] = v[j];
          }
        }
    }
    if (TEAMS > 1) __syncthreads();
  }

  // ---- team exchange --------------------------------------------------------------------
  // Partial results cross warps through one 16-byte slot per warp; after the team barrier
  // lane l of every warp reads the slot of warp l mod kW and a shuffle tree over kW lanes
  // folds them, so the cost per thread does not grow with the number of warps in the team.
  // In teams of four warps every thread reads all the slots instead, which saves two rounds of shuffles (and
  // the three sums of a warp are folded together, warp_sum_split): softmax -> LayerNorm of 16384 x 4096 bf16
  // 59.2 -> 56.5 us.  Two warps: no difference (20011 x 1537 fp16 46.9, 47.1); 8 and 16: 1 to 3 % slower (rows
  // of 4096 fp32 44.3, 45.4; 2238 x 7081 fp16 35.2, 36.3).
  __device__ __forceinline__ float* slot_base() { return this->red + this->phase * kW * 4; }
  template <class Op> __device__ __forceinline__ float xreduce(float v) {
    if constexpr (TEAM < 32) {
      return lane_group_reduce<Op, TEAM>(v);
    } else {
      v = warp_all<Op>(v);
      if constexpr (kW > 1) {
        float* slot = slot_base();
        if constexpr (kW == 4) {
          if ((this->lane & 31) == 0) slot[this->lane >> 5] = v;
          team_barrier(this->team + 1, TEAM);
          const float4 q = *reinterpret_cast<const float4*>(slot);
          v = Op::combine(Op::combine(q.x, q.z), Op::combine(q.y, q.w));
        } else {
          if ((this->lane & 31) == 0) slot[(this->lane >> 5) * 4] = v;
          team_barrier(this->team + 1, TEAM);
          v = slot[(this->lane & (kW - 1)) * 4];
          v = lane_group_reduce<Op, kW>(v);
        }
        this->phase ^= 1;
      }
      return v;
    }
  }
  // ---- inclusive prefix scan along the row (cumsum / cumprod over the stride-1 axis) -----------
  // Row order: vector i of thread t is vector i * TEAM + t of the row.  Per round i every
  // thread scans its own vector, the vector totals are scanned over the team in thread order
  // (shuffles inside a warp, one slot per warp across warps), and the total of the rounds
  // before is carried along.  Op is SumOp or ProdOp; fp32 accumulation, as the reference's sums.
  template <class Op, class A> __device__ __forceinline__ vf<kE> scan(const A& val) {
    vf<kE> out;
    float carry = Op::identity();
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      float run = Op::identity();
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j) {
        run = Op::combine(run, inside(i, j) ? Cast<float>::from(at(val, i * Base::kVec + j)) : Op::identity());
        out.v[i * Base::kVec + j] = run;
      }
      // inclusive scan of `run` over the lanes of this thread's warp (or lane group), and the
      // exclusive one beside it (the operator need not have an inverse)
      float incl = run, before = Op::identity();
      const int wl = this->lane & (kGroup - 1);
#pragma unroll
      for (int off = 1; off < kGroup; off <<= 1) {
        const float up_i = __shfl_up_sync(kFull, incl, off, kGroup);
        if (wl >= off) incl = Op::combine(up_i, incl);
      }
      if constexpr (std::is_same<Op, SumOp>::value) {
        before = incl - run;              // sums have an inverse: no second shuffle
      } else {
        const float up = __shfl_up_sync(kFull, incl, 1, kGroup);
        if (wl >= 1) before = up;
      }
      float total = __shfl_sync(kFull, incl, kGroup - 1, kGroup);  // the warp's (group's) total
      if constexpr (TEAM > 32) {
        float* slot = slot_base();
        const int w = this->lane >> 5;
        if ((this->lane & 31) == 31) slot[w * 4] = incl;
        team_barrier(this->team + 1, TEAM);
        float ahead = Op::identity(), all = Op::identity();
#pragma unroll
        for (int k = 0; k < kW; ++k) {
          const float tk = slot[k * 4];
          if (k < w) ahead = Op::combine(ahead, tk);
          all = Op::combine(all, tk);
        }
        before = Op::combine(ahead, before);
        total = all;
        this->phase ^= 1;
      }
      const float base = Op::combine(carry, before);
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j) out.v[i * Base::kVec + j] = Op::combine(base, out.v[i * Base::kVec + j]);
      carry = Op::combine(carry, total);
    }
    return out;
  }
  // the same scan with exact 64-bit integers (cumsum / cumprod of integer, index or boolean rows)
  template <class IOp, class A> __device__ __forceinline__ vi<kE> scan_int(const A& val) {
    vi<kE> out;
    long long carry = IOp::id();
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      long long run = IOp::id();
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j) {
        run = IOp::f(run, inside(i, j) ? Cast<long long>::from(at(val, i * Base::kVec + j)) : IOp::id());
        out.v[i * Base::kVec + j] = run;
      }
      long long incl = run, before = IOp::id();
      const int wl = this->lane & (kGroup - 1);
#pragma unroll
      for (int off = 1; off < kGroup; off <<= 1) {
        const long long up_i = __shfl_up_sync(kFull, incl, off, kGroup);
        if (wl >= off) incl = IOp::f(up_i, incl);
      }
      if constexpr (std::is_same<IOp, ISum>::value) {
        before = incl - run;
      } else {
        const long long up = __shfl_up_sync(kFull, incl, 1, kGroup);
        if (wl >= 1) before = up;
      }
      long long total = __shfl_sync(kFull, incl, kGroup - 1, kGroup);
      if constexpr (TEAM > 32) {
        long long* slot = reinterpret_cast<long long*>(slot_base());
        const int w = this->lane >> 5;
        if ((this->lane & 31) == 31) slot[w * 2] = incl;
        team_barrier(this->team + 1, TEAM);
        long long ahead = IOp::id(), all = IOp::id();
#pragma unroll
        for (int k = 0; k < kW; ++k) {
          const long long tk = slot[k * 2];
          if (k < w) ahead = IOp::f(ahead, tk);
          all = IOp::f(all, tk);
        }
        before = IOp::f(ahead, before);
        total = all;
        this->phase ^= 1;
      }
      const long long base = IOp::f(carry, before);
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j) out.v[i * Base::kVec + j] = IOp::f(base, out.v[i * Base::kVec + j]);
      carry = IOp::f(carry, total);
    }
    return out;
  }

  // ---- thread-local folds -------------------------------------------------------------------
  // sum over pairs of elements (pair p = elements 2p, 2p + 1) in independent chains: step(p, acc) is
  // the accumulator with pair p added; only the vectors that may reach past the end of the row are
  // tested, and what lies there leaves the accumulator as it was
  template <class F> __device__ __forceinline__ float fold_pairs(const F& step) const {
    float2 acc[kChains];
#pragma unroll
    for (int c = 0; c < kChains; ++c) acc[c] = make_float2(0.f, 0.f);
#pragma unroll
    for (int p = 0; p < kE / 2; ++p) {
      float2& a = acc[p % kChains];
      const float2 v = step(p, a);
      if (inside((2 * p) / Base::kVec, (2 * p) % Base::kVec)) a.x = v.x;
      if (inside((2 * p + 1) / Base::kVec, (2 * p + 1) % Base::kVec)) a.y = v.y;
    }
#pragma unroll
    for (int c = 1; c < kChains; ++c) acc[0] = add2(acc[0], acc[c]);
    return acc[0].x + acc[0].y;
  }
  // ZEROS: what lies past the end of the row is zero in `val`
  template <bool ZEROS = false, class A> __device__ __forceinline__ float local_sum(const A& val) const {
    if constexpr ((FULL || (ZEROS && COLS > 0)) && op::is_fvec<A>::value) {
      // kChains independent chains of packed adds: a single chain would serialise on the
      // add latency with only a few warps resident
      float2 acc[kChains];
#pragma unroll
      for (int c = 0; c < kChains; ++c) acc[c] = op::pr(val, c);
#pragma unroll
      for (int p = kChains; p < kE / 2; ++p) acc[p % kChains] = add2(acc[p % kChains], op::pr(val, p));
#pragma unroll
      for (int c = 1; c < kChains; ++c) acc[0] = add2(acc[0], acc[c]);
      return acc[0].x + acc[0].y;
    } else if constexpr (COLS > 0 && op::is_fvec<A>::value) {
      return fold_pairs([&](int p, const float2& acc) { return add2(acc, op::pr(val, p)); });
    } else {
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < VPT; ++i)
#pragma unroll
        for (int j = 0; j < Base::kVec; ++j)
          if (inside(i, j)) acc += Cast<float>::from(at(val, i * Base::kVec + j));
      return acc;
    }
  }
  // sum of a[e] * b[e]
  template <class A, class B> __device__ __forceinline__ float local_dot(const A& a, const B& b) const {
    if constexpr (FULL && op::packable2<A, B>::value) {
      float2 acc[kChains];
#pragma unroll
      for (int c = 0; c < kChains; ++c) acc[c] = mul2(op::pr(a, c), op::pr(b, c));
#pragma unroll
      for (int p = kChains; p < kE / 2; ++p) acc[p % kChains] = fma2(op::pr(a, p), op::pr(b, p), acc[p % kChains]);
#pragma unroll
      for (int c = 1; c < kChains; ++c) acc[0] = add2(acc[0], acc[c]);
      return acc[0].x + acc[0].y;
    } else if constexpr (COLS > 0 && op::packable2<A, B>::value) {
      return fold_pairs([&](int p, const float2& acc) { return fma2(op::pr(a, p), op::pr(b, p), acc); });
    } else {
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < VPT; ++i)
#pragma unroll
        for (int j = 0; j < Base::kVec; ++j)
          if (inside(i, j))
            acc = fmaf(Cast<float>::from(at(a, i * Base::kVec + j)), Cast<float>::from(at(b, i * Base::kVec + j)), acc);
      return acc;
    }
  }
  template <class Op, class A> __device__ __forceinline__ float local_fold(const A& val) const {
    if constexpr (std::is_same<Op, SumOp>::value) {
      return local_sum(val);
    } else {
      float acc = Op::identity();
#pragma unroll
      for (int i = 0; i < VPT; ++i)
#pragma unroll
        for (int j = 0; j < Base::kVec; ++j)
          if (inside(i, j)) acc = Op::combine(acc, Cast<float>::from(at(val, i * Base::kVec + j)));
      return acc;
    }
  }

  // reductions over the valid elements of the row
  template <class Op, class A> __device__ __forceinline__ float reduce(const A& val) {
    return xreduce<Op>(local_fold<Op>(val));
  }
  // sum of an element-wise product (the multiply rides in the accumulating fma)
  template <class A, class B> __device__ __forceinline__ float reduce_dot(const A& a, const B& b) {
    return xreduce<SumOp>(local_dot(a, b));
  }
  // Exact integer reductions: 64-bit accumulators, shuffled as two halves, exchanged
  // through the same slots (a slot holds two 64-bit values).
  using ISum = ::ixb::gen::ISum;
  using IProd = ::ixb::gen::IProd;
  using IMax = ::ixb::gen::IMax;
  using IMin = ::ixb::gen::IMin;
  template <class IOp, class A> __device__ __forceinline__ long long local_fold_int(const A& val) const {
    long long acc = IOp::id();
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j)
        if (inside(i, j)) acc = IOp::f(acc, Cast<long long>::from(at(val, i * Base::kVec + j)));
    return acc;
  }
  template <class IOp> __device__ __forceinline__ long long xreduce_int(long long acc) {
#pragma unroll
    for (int o = kGroup / 2; o > 0; o >>= 1) acc = IOp::f(acc, __shfl_xor_sync(kFull, acc, o));
    if constexpr (kW > 1) {
      long long* slot = reinterpret_cast<long long*>(slot_base());
      if ((this->lane & 31) == 0) slot[(this->lane >> 5) * 2] = acc;
      team_barrier(this->team + 1, TEAM);
      acc = slot[(this->lane & (kW - 1)) * 2];
#pragma unroll
      for (int o = kW / 2; o > 0; o >>= 1) acc = IOp::f(acc, __shfl_xor_sync(kFull, acc, o));
      this->phase ^= 1;
    }
    return acc;
  }
  template <class IOp, class A> __device__ __forceinline__ long long reduce_int(const A& val) {
    return xreduce_int<IOp>(local_fold_int<IOp>(val));
  }
  template <bool IS_MAX, class A> __device__ __forceinline__ ArgPair local_arg(const A& val) const {
    ArgPair best = ArgOp<IS_MAX>::identity();
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j)
        if (inside(i, j))
          best = ArgOp<IS_MAX>::combine(
              best, ArgPair{Cast<float>::from(at(val, i * Base::kVec + j)), (long long)(vec_col(i) + j)});
    return best;
  }
  template <bool IS_MAX> __device__ __forceinline__ long long xreduce_arg(ArgPair best) {
    if constexpr (TEAM < 32) {
#pragma unroll
      for (int o = TEAM / 2; o > 0; o >>= 1) {
        ArgPair q;
        q.v = __shfl_xor_sync(kFull, best.v, o);
        q.i = __shfl_xor_sync(kFull, best.i, o);
        best = ArgOp<IS_MAX>::combine(best, q);
      }
      return best.i;
    } else {
      return Base::template reduce_arg<IS_MAX>(best).i;
    }
  }
  template <bool IS_MAX, class A> __device__ __forceinline__ long long reduce_arg(const A& val) {
    return xreduce_arg<IS_MAX>(local_arg<IS_MAX>(val));
  }

  // arg-reductions of 32- and 64-bit integers: compared as integers (as floats, neighbours
  // beyond 2^24 would tie and the smaller index would win); same tie rule, no NaN to consider
  struct ArgPairI {
    long long v, i;
  };
  template <bool IS_MAX> static __device__ __forceinline__ ArgPairI arg_identity_int() {
    return ArgPairI{IS_MAX ? (-0x7fffffffffffffffLL - 1) : 0x7fffffffffffffffLL, 0x7fffffffffffffffLL};
  }
  template <bool IS_MAX> static __device__ __forceinline__ ArgPairI arg_better(ArgPairI a, ArgPairI b) {
    const bool take_b = (a.v == b.v) ? (b.i < a.i) : (IS_MAX ? (b.v > a.v) : (b.v < a.v));
    return take_b ? b : a;
  }
  template <bool IS_MAX, class A> __device__ __forceinline__ ArgPairI local_arg_int(const A& val) const {
    ArgPairI best = arg_identity_int<IS_MAX>();
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j)
        if (inside(i, j))
          best = arg_better<IS_MAX>(
              best, ArgPairI{Cast<long long>::from(at(val, i * Base::kVec + j)), (long long)(vec_col(i) + j)});
    return best;
  }
  template <bool IS_MAX> __device__ __forceinline__ long long xreduce_arg_int(ArgPairI best) {
#pragma unroll
    for (int o = kGroup / 2; o > 0; o >>= 1) {
      ArgPairI q;
      q.v = __shfl_xor_sync(kFull, best.v, o);
      q.i = __shfl_xor_sync(kFull, best.i, o);
      best = arg_better<IS_MAX>(best, q);
    }
    if constexpr (kW > 1) {
      long long* slot = reinterpret_cast<long long*>(slot_base());   // a slot holds the pair
      if ((this->lane & 31) == 0) {
        slot[(this->lane >> 5) * 2] = best.v;
        slot[(this->lane >> 5) * 2 + 1] = best.i;
      }
      team_barrier(this->team + 1, TEAM);
      best.v = slot[(this->lane & (kW - 1)) * 2];
      best.i = slot[(this->lane & (kW - 1)) * 2 + 1];
#pragma unroll
      for (int o = kW / 2; o > 0; o >>= 1) {
        ArgPairI q;
        q.v = __shfl_xor_sync(kFull, best.v, o);
        q.i = __shfl_xor_sync(kFull, best.i, o);
        best = arg_better<IS_MAX>(best, q);
      }
      this->phase ^= 1;
    }
    return best.i;
  }
  template <bool IS_MAX, class A> __device__ __forceinline__ long long reduce_arg_int(const A& val) {
    return xreduce_arg_int<IS_MAX>(local_arg_int<IS_MAX>(val));
  }

  // ---- online softmax ------------------------------------------------------------------------
  // One exchange yields the row maximum, the sum of exp(value - maximum) and up to three
  // further row sums ("riders") that the emitter found it could form before the maximum is
  // known: NS of them are sums of exp(value - maximum) * w for a vector w (they are
  // accumulated relative to each thread's own maximum and rescaled as partial results are
  // folded, like the sum itself), NP are ordinary sums.  The thread keeps its exponentials
  // relative to its own maximum in `e` and the factor `r` that brings them to the row
  // maximum, so that exp(value - maximum) costs one multiply afterwards instead of a second
  // pass over the exponential unit.
  template <int NS, int NP> struct Online {
    float max, sum, r;
    vf<kE> e;
    float scaled[NS > 0 ? NS : 1], plain[NP > 0 ? NP : 1];
  };
  // COMPUTED: some w is not a plain operand, which is zero past the end of the row, but computed from
  // such zeros, and may be infinite or NaN there; no zero exponential removes that, so it is masked.
  // PLAIN: the same of the vectors of the plain sums; operands' sums need no test.
  template <int NS, int NP, bool COMPUTED = false, bool PLAIN = false, class A>
  __device__ __forceinline__ Online<NS, NP> online_softmax(const A& val, const VecRefs<kE, NS>& w,
                                                            const VecRefs<kE, NP>& pl) {
    static_assert(NS + NP <= 2, "a slot holds the maximum, the sum and two riders");
    Online<NS, NP> o;
    float mc[kChains];
#pragma unroll
    for (int c = 0; c < kChains; ++c) mc[c] = -INFINITY;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; j += 2) {
        const int e0 = i * Base::kVec + j;
        const float a = inside(i, j) ? Cast<float>::from(at(val, e0)) : -INFINITY;
        const float b = inside(i, j + 1) ? Cast<float>::from(at(val, e0 + 1)) : -INFINITY;
        mc[(e0 / 2) % kChains] = max3(mc[(e0 / 2) % kChains], a, b);
      }
    float m = mc[0];
#pragma unroll
    for (int c = 1; c < kChains; ++c) m = fmaxf(m, mc[c]);
    // v[0] = sum of exponentials, v[1..NS] scaled riders, then the plain riders
    float v[1 + NS + NP];
#pragma unroll
    for (int k = 0; k < 1 + NS + NP; ++k) v[k] = 0.f;
    const op::ExpScale ks(m == -INFINITY ? 0.f : m);
    float2 acc[1 + NS][kChains];
#pragma unroll
    for (int k = 0; k < 1 + NS; ++k)
#pragma unroll
      for (int c = 0; c < kChains; ++c) acc[k][c] = make_float2(0.f, 0.f);
#pragma unroll
    for (int p = 0; p < kE / 2; ++p) {
      const float2 x = make_float2(Cast<float>::from(at(val, 2 * p)), Cast<float>::from(at(val, 2 * p + 1)));
      const float2 t = fma2(x, make_float2(ks.scale, ks.scale), make_float2(ks.shift, ks.shift));
      float2 ex = make_float2(fast_exp2(t.x), fast_exp2(t.y));
      const bool in0 = inside((2 * p) / Base::kVec, (2 * p) % Base::kVec);
      const bool in1 = inside((2 * p + 1) / Base::kVec, (2 * p + 1) % Base::kVec);
      if (!in0) ex.x = 0.f;
      if (!in1) ex.y = 0.f;
      o.e.v[2 * p] = ex.x;
      o.e.v[2 * p + 1] = ex.y;
      acc[0][p % kChains] = add2(acc[0][p % kChains], ex);
#pragma unroll
      for (int k = 0; k < NS; ++k) {
        float2 weight = op::pr(*w.p[k], p);
        if (COMPUTED && !in0) weight.x = 0.f;
        if (COMPUTED && !in1) weight.y = 0.f;
        acc[1 + k][p % kChains] = fma2(ex, weight, acc[1 + k][p % kChains]);
      }
    }
#pragma unroll
    for (int k = 0; k < 1 + NS; ++k) {
#pragma unroll
      for (int c = 1; c < kChains; ++c) acc[k][0] = add2(acc[k][0], acc[k][c]);
      v[k] = acc[k][0].x + acc[k][0].y;
    }
#pragma unroll
    for (int k = 0; k < NP; ++k) v[1 + NS + k] = local_sum<!PLAIN>(*pl.p[k]);

    // warp stage: agree on the warp's maximum, rescale, sum
    float r;
    if constexpr (TEAM < 32) {
      const float mw = lane_group_reduce<FastMaxOp, TEAM>(m);
      r = (m == -INFINITY) ? 0.f : fast_exp2((m - mw) * kLog2e);
#pragma unroll
      for (int k = 0; k < 1 + NS; ++k) v[k] *= r;
#pragma unroll
      for (int k = 0; k < 1 + NS + NP; ++k) v[k] = lane_group_reduce<SumOp, TEAM>(v[k]);
      m = mw;
    } else {
      const float mw = warp_max_fast(m);
      r = (m == -INFINITY) ? 0.f : fast_exp2((m - mw) * kLog2e);
#pragma unroll
      for (int k = 0; k < 1 + NS; ++k) v[k] *= r;
      m = mw;
      if constexpr (kW == 1) {
        warp_sum<1 + NS + NP>(v);
      } else if constexpr (kW == 4) {
        float* slot = slot_base() + (this->lane >> 5) * 4;
        if constexpr (1 + NS + NP == 1) {
          warp_sum<1>(v);
          if ((this->lane & 31) == 0) *reinterpret_cast<float2*>(slot) = make_float2(mw, v[0]);
        } else {
          // lane 8 k holds sum k
          const float t = warp_sum_split(v[0], v[1], 1 + NS + NP > 2 ? v[NS + NP] : 0.f);
          if ((this->lane & 7) == 0) slot[((this->lane >> 3) + 1) & 3] = (this->lane & 31) == 24 ? mw : t;
        }
        team_barrier(this->team + 1, TEAM);
        float4 part[kW];
#pragma unroll
        for (int w = 0; w < kW; ++w) part[w] = *reinterpret_cast<const float4*>(slot_base() + w * 4);
        const float mm = max3(fmaxf(part[0].x, part[1].x), part[2].x, part[3].x);
        const float base = mm == -INFINITY ? 0.f : mm;
        v[0] = 0.f;
        if constexpr (NS + NP > 0) v[1] = 0.f;
        if constexpr (NS + NP > 1) v[2] = 0.f;
#pragma unroll
        for (int w = 0; w < kW; ++w) {
          const float f = fast_exp2((part[w].x - base) * kLog2e);
          const float pv[3] = {part[w].y, part[w].z, part[w].w};
#pragma unroll
          for (int k = 0; k < 1 + NS + NP; ++k) v[k] = k < 1 + NS ? fmaf(pv[k], f, v[k]) : v[k] + pv[k];
        }
        r *= fast_exp2((mw - base) * kLog2e);
        m = mm;
        this->phase ^= 1;
      } else {
        warp_sum<1 + NS + NP>(v);
        float* slot = slot_base();
        if ((this->lane & 31) == 0) {
          float4 s4 = make_float4(mw, v[0], 0.f, 0.f);
          if constexpr (1 + NS + NP > 1) s4.z = v[1];
          if constexpr (1 + NS + NP > 2) s4.w = v[2];
          *reinterpret_cast<float4*>(slot + (this->lane >> 5) * 4) = s4;
        }
        team_barrier(this->team + 1, TEAM);
        const float4 part = *reinterpret_cast<const float4*>(slot + (this->lane & (kW - 1)) * 4);
        const float mm = lane_group_reduce<FastMaxOp, kW>(part.x);
        const float f = (part.x == -INFINITY) ? 0.f : fast_exp2((part.x - mm) * kLog2e);
        const float pv[3] = {part.y, part.z, part.w};
#pragma unroll
        for (int k = 0; k < 1 + NS + NP; ++k)
          v[k] = lane_group_reduce<SumOp, kW>(k < 1 + NS ? pv[k] * f : pv[k]);
        r *= (mw == -INFINITY) ? 0.f : fast_exp2((mw - mm) * kLog2e);
        m = mm;
        this->phase ^= 1;
      }
    }
    o.max = m;
    o.sum = v[0];
    o.r = r;
#pragma unroll
    for (int k = 0; k < NS; ++k) o.scaled[k] = v[1 + k];
#pragma unroll
    for (int k = 0; k < NP; ++k) o.plain[k] = v[1 + NS + k];
    return o;
  }
  // (mean, sum of squared deviations, count) of the row with a single exchange: each
  // thread forms the statistics of its own elements and partial statistics are merged
  // pairwise (Chan et al.), which stays accurate when the mean is large against the spread
  struct Welford {
    float mean, m2, weight;
  };
  static __device__ __forceinline__ Welford merge(const Welford& a, const Welford& b) {
    const float n = a.weight + b.weight;
    const float w = n > 0.f ? __fdividef(b.weight, n) : 0.f;
    const float d = b.mean - a.mean;
    return Welford{fmaf(d, w, a.mean), a.m2 + b.m2 + d * d * a.weight * w, n};
  }
  // statistics of this thread's elements (two passes over registers: mean, then deviations)
  template <class A> __device__ __forceinline__ Welford local_welford(const A& val) const {
    float n = 0.f, sum = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j)
        if (inside(i, j)) {
          n += 1.f;
          sum += Cast<float>::from(at(val, i * Base::kVec + j));
        }
    Welford w{n > 0.f ? sum / n : 0.f, 0.f, n};
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j)
        if (inside(i, j)) {
          const float d = Cast<float>::from(at(val, i * Base::kVec + j)) - w.mean;
          w.m2 = fmaf(d, d, w.m2);
        }
    return w;
  }
  // merge the threads' statistics over the team; every thread gets the row's
  __device__ __forceinline__ Welford xwelford(Welford w) {
#pragma unroll
    for (int off = kGroup / 2; off > 0; off >>= 1) {
      Welford o{__shfl_xor_sync(0xffffffffu, w.mean, off), __shfl_xor_sync(0xffffffffu, w.m2, off),
                __shfl_xor_sync(0xffffffffu, w.weight, off)};
      // both lanes of a pair must fold in the same order to agree bit for bit
      w = (this->lane & off) ? merge(o, w) : merge(w, o);
    }
    if constexpr (TEAM > 32) {
      float* slot = this->red + this->phase * Base::kWarpsPerTeam * 4;
      if ((this->lane & 31) == 0)
        *reinterpret_cast<float4*>(slot + (this->lane >> 5) * 4) = make_float4(w.mean, w.m2, w.weight, 0.f);
      team_barrier(this->team + 1, TEAM);
      const float4 first = *reinterpret_cast<const float4*>(slot);
      w = Welford{first.x, first.y, first.z};
#pragma unroll
      for (int k = 1; k < Base::kWarpsPerTeam; ++k) {
        const float4 part = *reinterpret_cast<const float4*>(slot + k * 4);
        w = merge(w, Welford{part.x, part.y, part.z});
      }
      this->phase ^= 1;
    }
    return w;
  }
  template <class A> __device__ __forceinline__ Welford welford(const A& val) { return xwelford(local_welford(val)); }
  // Online softmax of a row walked in chunks: the running (maximum, sum of exponentials
  // relative to it) of this thread absorbs one chunk; the team exchange follows the loop.
  struct MaxSum {
    float max, sum;
  };
  template <class A> __device__ __forceinline__ void online_chunk(MaxSum& acc, const A& val) const {
    float m = acc.max;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j)
        if (inside(i, j)) m = fmaxf(m, Cast<float>::from(at(val, i * Base::kVec + j)));
    if (m == -INFINITY) return;      // nothing but -inf so far
    float s = acc.sum * fast_exp2((acc.max - m) * kLog2e);   // exp2(-inf) == 0 covers the first chunk
    const op::ExpScale ks(m);
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < Base::kVec; ++j)
        if (inside(i, j)) s += fast_exp2(fmaf(Cast<float>::from(at(val, i * Base::kVec + j)), ks.scale, ks.shift));
    acc.max = m;
    acc.sum = s;
  }
  __device__ __forceinline__ MaxSum online_finish(MaxSum acc) {
    float m = acc.max, s[1] = {acc.sum}, none[1] = {0.f};
    if constexpr (TEAM < 32) {
      const float mw = lane_group_reduce<FastMaxOp, TEAM>(m);
      const float r = (m == -INFINITY) ? 0.f : fast_exp2((m - mw) * kLog2e);
      return MaxSum{mw, lane_group_reduce<SumOp, TEAM>(s[0] * r)};
    } else {
      Base::template reduce_rescaled<1, 0>(m, s, none, kLog2e);
      return MaxSum{m, s[0]};
    }
  }
  template <class A> __device__ __forceinline__ bool reduce_any(const A& val) {
    return reduce<MaxOp>(op::where(val, 1.f, 0.f)) != 0.f;
  }
};

// Per-column operand J of a generated body: the first KREGS operands (the most used ones) are
// registers of the thread, the others are read from the shared-memory table when needed.
template <int J, int KREGS, class Ctx, class U, int E>
__device__ __forceinline__ void kinit(Ctx& c, vf<E>& reg, const U* rowp) {
  if constexpr (J < KREGS) reg = c.template load_row<false>(rowp);
  else c.template fill_sconst<J - KREGS>(rowp);
}
template <int J, int KREGS, class Ctx, int E>
__device__ __forceinline__ vf<E> kget(const Ctx& c, const vf<E>& reg) {
  if constexpr (J < KREGS) return reg;
  else return c.template sconst<J - KREGS>();
}

// Order in which a row kernel with short rows walks its kept index.  The kept space is
// [A][LC][LB] with LB fastest (the order of the output), while the rows that are adjacent in
// memory are the ones that differ in the LC digit.  Walking it in TB x TC tiles - TC consecutive
// LC digits fastest, then TB consecutive LB digits - makes a warp read adjacent rows (one
// contiguous span) and lets the one-element-per-row results of a tile fill whole sectors, the
// job the reference gives its transposed tile (inductor_x/codegen/triton.py:856-888).
// B_FIRST: inside a tile the output digit runs fastest, so the rows a warp works on at once
// store one contiguous run (a full 32-byte sector for sixteen 16-bit results); chosen when a
// row is at least one 128-byte line, i.e. when reading rows that are far apart wastes nothing.
// At the ends of the digits the tiles are smaller (a stripe of TC or what is left LC digits is walked tile
// after tile, the last of them narrower); the divisors are constants in each of the four kinds.
template <int LB, int TB, int TC, int B, int C, bool B_FIRST>  // a tile of B x C, the first LC digit of its stripe
__device__ __forceinline__ unsigned in_tile(unsigned b_hi, unsigned in, unsigned c0) {
  const unsigned c_lo = B_FIRST ? in / B : in % C, b_lo = B_FIRST ? in % B : in / C;
  return (c0 + c_lo) * LB + b_hi * TB + b_lo;
}
template <int LB, int TB, int TC, int C, bool B_FIRST>         // a stripe of C digits
__device__ __forceinline__ unsigned in_stripe(unsigned rem, unsigned c0) {
  const unsigned b_hi = rem / (C * TB), in = rem - b_hi * (C * TB);
  if constexpr (LB % TB != 0) {
    if (b_hi >= LB / TB) return in_tile<LB, TB, TC, LB % TB, C, B_FIRST>(b_hi, in, c0);
  }
  return in_tile<LB, TB, TC, TB, C, B_FIRST>(b_hi, in, c0);
}
template <int LB, int LC, int TB, int TC, bool B_FIRST = false, class I>
__device__ __forceinline__ long long tile_order(I slot) {
  constexpr I kPlane = (I)LB * LC;
  const I a = slot / kPlane;
  const unsigned rem = (unsigned)(slot - a * kPlane);
  const unsigned c_hi = rem / (TC * LB), in = rem - c_hi * (TC * LB);
  if constexpr (LC % TC != 0) {
    if (c_hi >= LC / TC) return (long long)(a * kPlane + in_stripe<LB, TB, TC, LC % TC, B_FIRST>(in, c_hi * TC));
  }
  return (long long)(a * kPlane + in_stripe<LB, TB, TC, TC, B_FIRST>(in, c_hi * TC));
}

// CTAs of a row kernel that fit on one SM, cached per device (the attribute is a property of
// the device the calling thread has current; several host threads may ask at once)
template <class K> inline int row_resident(K kern, int threads, size_t smem = 0) {
  static std::atomic<int> cache[64];
  int dev = 0;
  cudaGetDevice(&dev);
  const int slot = dev & 63;
  int n = cache[slot].load(std::memory_order_acquire);
  if (n == 0) {
    // static + dynamic shared memory beyond 48 KiB needs the opt-in, once per device
    if (smem > 32 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return -1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem) != cudaSuccess || n < 1) return -1;
    cache[slot].store(n, std::memory_order_release);
  }
  return n;
}

// Sums over the rows beside the row's own work (the gradient of a norm's weight beside that of its input):
// every thread sums its columns over the rows of its team in fp32, a block folds its teams and stores one
// row of partial sums, and finish_columns adds those.  A kernel of its own reads both operands a second
// time: 32768 x 4096 bf16, gradient of the input 121 us and of the weight 88,
// both together 123.
__host__ __device__ constexpr long long partial_pitch(long long cols) { return (cols + 3) / 4 * 4; }
// 32 columns a block, a warp for every 32nd partial row: there are few of them to go round (eight warps
// a block took 4 us longer on 1024 columns)
constexpr int kFinishSlices = 32;
template <class U>
__global__ void __launch_bounds__(32 * kFinishSlices) finish_columns_kernel(const float* partial, int rows, int cols, U* out) {
  __shared__ float fold[kFinishSlices][33];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int col = (int)blockIdx.x * 32 + lane;
  pdl_launch_dependents();
  pdl_wait();
  float s[2] = {0.f, 0.f};
  if (col < cols) {
    const float* p = partial + col;
    const long long pitch = partial_pitch(cols);
    int r = slice;
#pragma unroll 2
    for (; r + kFinishSlices < rows; r += 2 * kFinishSlices) {
      s[0] += p[r * pitch];
      s[1] += p[(r + kFinishSlices) * pitch];
    }
    if (r < rows) s[0] += p[r * pitch];
  }
  fold[slice][lane] = s[0] + s[1];
  __syncthreads();
  // a warp for each column
  const float t = warp_reduce<SumOp>(fold[lane][slice]);
  const int mine = (int)blockIdx.x * 32 + slice;
  if (lane == 0 && mine < cols) Mem<U>::st(out + mine, t);
}
template <class U> int finish_columns(const float* partial, long long rows, int cols, U* out, void* stream) {
  return (int)launch_pdl(finish_columns_kernel<U>, (unsigned)((cols + 31) / 32), 32 * kFinishSlices, 0, (cudaStream_t)stream, partial,
                         (int)rows, cols, out);
}

// Sub-warp teams whose threads load nothing once for all rows get a block for every batch of four rows a
// team (see stream_grid) where there are more than the resident blocks would see in three batches and they move
// more than stays in L2: the permuted sum of 64 x 128 x 256 x 64 fp16 48.9 -> 45.4 us, softmax of 2^24 fp32
// in rows of 16 24.7 -> 22.0, LayerNorm in rows of 32 24.2 -> 22.0.  Below that nothing drifts apart in DRAM and the
// blocks' starts are what is left: of 2^22 6.0 -> 6.9, 5.8 -> 6.1, softmax of 65536 x 64 bf16 4.1 -> 4.7.
template <class Body, int TEAM, bool STAGED> constexpr bool kStreamRows = TEAM < 32 && STAGED && Body::kStream > 0 && Body::kConsts == 0;
// the L2 of a B200; what a kernel moves beyond it comes from and goes to DRAM
constexpr long long kL2Bytes = 126ll << 20;

template <class Body, typename T, int TEAM, int TEAMS, int VPT, int MIN_CTAS, int PF, int COLS, bool STAGED>
__global__ void __launch_bounds__(TEAM* TEAMS, MIN_CTAS)
    row_gen_kernel(const Body body, const long long rows, const int cols, const bool a_batch_each) {
  // Rows off a 16-byte boundary repeat their offset every kShiftPeriod rows.  Block b works on rows b,
  // b + period, ... only: its offset stays what it is, and the row is worked on in the aligned
  // vectors of memory as if it began there (`off` elements that are masked), per-column operands
  // shifted once to match - nothing is shifted per row.
  static_assert(Body::kColumns == 0 || (TEAM >= 32 && !Body::kLooped), "sums over the rows want whole warps to a row, and the row on chip");
  constexpr int kPeriod = STAGED && TEAM >= 32 ? Body::kShiftPeriod : 0;
  using Ctx = GenRowCtx<T, TEAM, TEAMS, VPT, COLS, (kPeriod > 0)>;
  constexpr int kSlots = TEAM > 32 ? 2 * (TEAM / 32) * 4 : 1;  // exchange floats per team
  __shared__ __align__(16) float exchange[TEAMS * kSlots];
  extern __shared__ __align__(16) unsigned char operand_table[];   // Body::kSmemConsts slots
  Ctx c;
  c.lane = threadIdx.x % TEAM;
  c.team = threadIdx.x / TEAM;
  c.cols = cols;
  c.phase = 0;
  c.red = exchange + c.team * kSlots;
  c.ktab = reinterpret_cast<const float4*>(operand_table);
  // the next launch of the stream may place its CTAs as ours retire; no global access
  // happens before the launch ahead of us has completed
  pdl_launch_dependents();
  pdl_wait();
  const long long stride = (long long)gridDim.x * TEAMS;
  long long row0 = (long long)blockIdx.x * TEAMS + c.team;
  if constexpr (kPeriod > 0) {
    const int cls = (int)(blockIdx.x % kPeriod);
    row0 = cls + kPeriod * ((long long)(blockIdx.x / kPeriod) * TEAMS + c.team);
    c.off = body.row_offset(cls);
  }
  // the first row's vectors are requested before the per-column operands are loaded and
  // widened, so that both latencies overlap (it matters for kernels of a few microseconds)
  typename Body::Raw nxt;
  if constexpr (TEAM >= 32 && STAGED) {
    if (row0 < rows) body.fetch(c, row0, nxt);
  }
  typename Body::Cols sums;
  body.clear(sums);
  typename Body::Consts k;
  body.init(c, k);
  if constexpr (Body::kSmemConsts > 0) __syncthreads();   // the operand table is complete
  if constexpr (TEAM < 32) {
    // The teams of a warp run the same number of rows (full-mask shuffles inside).  Rows this
    // short give a thread one vector each, so kBatch rows are fetched before the first is
    // worked on: kBatch independent loads in flight per thread instead of one.
    constexpr int kBatch = STAGED ? 4 : 1;
    typename Body::Raw raw[kBatch];
    // Rows walked in tiles (tile_order), with enough of them to go round: the rows of a batch
    // follow each other, so that a CTA reads a whole 16 x 16 tile at a time - 2 KB from each of 16
    // places instead of 512 bytes - and DRAM pages are used up while they are open (sum over the
    // last axis of a permuted 64 x 128 x 256 x 64 fp16: 54.6 -> 52.4 us).  Rows in memory order
    // gain nothing from it (43.3 against 44.8 us) and keep the strided batches.
    // Where a block is started for every batch (launch_row_gen) the batches in flight follow each other
    // through memory, and so do the rows of a batch.
    const bool blocked = a_batch_each || (Body::kTiled && rows >= stride * kBatch);
    const long long ustep = blocked ? TEAMS : stride;
    for (long long base = (long long)blockIdx.x * TEAMS * (blocked ? kBatch : 1); base < rows; base += stride * kBatch) {
      if constexpr (STAGED) {
        // Rows the batch does not have are not fetched: the last row in their place, as every team of every CTA asked
        // for it, is one line of L2 that answers one request at a time.  Rows enough for half a batch a CTA,
        // with that row and without: cumsum of 74898 x 56 bf16 9.3 and 3.5 us, LayerNorm of 131072 x 32 fp32 9.1 and
        // 6.0, sum of 16384 x 64 fp16 (permuted) 4.1 and 1.7.
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const long long r = base + u * ustep + c.team;
          if (u == 0 || base + u * ustep < rows) body.fetch(c, r < rows ? r : rows - 1, raw[u]);   // (uniform over the CTA)
        }
      }
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const long long b = base + u * ustep;
        if (b >= rows) break;            // uniform over the CTA
        const long long r = b + c.team;
        c.live = r < rows;
        body.template row<STAGED>(c, k, c.live ? r : rows - 1, raw[u], sums);
      }
    }
    return;
  } else {
    long long r = row0;
    while (r < rows) {
      const typename Body::Raw cur = nxt;
      const long long rn = r + stride;
      if constexpr (STAGED) {
        if (rn < rows) body.fetch(c, rn, nxt);
      }
      // PF rows beyond the fetched one are on their way from DRAM to L2
      if constexpr (PF > 0) {
        const long long ahead = r + (PF + (STAGED ? 1 : 0)) * stride;
        if (ahead < rows) body.prefetch(c, ahead);
      }
      body.template row<STAGED>(c, k, r, cur, sums);
      r = rn;
    }
    if constexpr (Body::kColumns > 0) {
      __syncthreads();    // the operand table is done with
      body.flush(c, sums, reinterpret_cast<float4*>(operand_table));
    }
  }
}
template <class Body, typename T, int TEAM, int TEAMS, int VPT, int MIN_CTAS = 1, int PF = 0, int COLS = 0>
int launch_row_gen(const Body& body, long long rows, int cols, void* stream, bool aligned = false,
                   long long* blocks = nullptr) {
  if (rows <= 0) return 0;
  if (COLS > 0 && cols != COLS) return (int)cudaErrorInvalidValue;
  // a row longer than the team can hold (a run-time extent beyond the compiled capacity);
  // looped bodies walk any length in chunks
  if (cols < 0 || (!Body::kLooped && cols > TEAM * VPT * Elem<T>::kVec)) return (int)cudaErrorInvalidValue;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long groups = (rows + TEAMS - 1) / TEAMS;
  using Ctx = GenRowCtx<T, TEAM, TEAMS, VPT, COLS>;
  // (the table also takes one column sum of the block's teams)
  constexpr int kSlots = Body::kSmemConsts > 0 ? Body::kSmemConsts : (Body::kColumns > 0 && TEAMS > 1 ? 1 : 0);
  const size_t smem = (size_t)kSlots * Ctx::kQuads * Ctx::kTabVecs * sizeof(float4);
  constexpr int kPeriod = TEAM >= 32 ? Body::kShiftPeriod : 0;
  // (a row in the vectors of memory may need one vector more than its own length)
  if (kPeriod > 0 && cols + Elem<T>::kVec - 1 > TEAM * VPT * Elem<T>::kVec) aligned = false;
  if (aligned) {
    auto kern = row_gen_kernel<Body, T, TEAM, TEAMS, VPT, MIN_CTAS, PF, COLS, true>;
    const int resident = row_resident(kern, TEAM * TEAMS, smem);
    if (resident < 1) return (int)cudaErrorInvalidConfiguration;
    long long grid = (long long)sms * resident;
    if (Body::kColumns > 0 && grid > Body::kPartials) grid = Body::kPartials;
    if constexpr (kPeriod > 0) {      // as many blocks for each offset
      const long long most = grid < kPeriod ? kPeriod : grid / kPeriod * kPeriod;
      grid = (groups + kPeriod - 1) / kPeriod * kPeriod;
      if (grid > most) grid = most;
    } else if (grid > groups) {
      grid = groups;
    }
    bool a_batch_each = false;
    if (kStreamRows<Body, TEAM, true> && groups > 3 * (long long)sms * resident &&
        rows * (cols * (long long)sizeof(T) * Body::kStream) > kL2Bytes) {
      grid = (groups + 3) / 4;
      a_batch_each = true;
    }
    if (blocks != nullptr) *blocks = grid;
    return (int)launch_pdl(kern, (unsigned)grid, TEAM * TEAMS, smem, (cudaStream_t)stream, body, rows, cols, a_batch_each);
  }
  auto kern = row_gen_kernel<Body, T, TEAM, TEAMS, VPT, MIN_CTAS, PF, COLS, false>;
  const int resident = row_resident(kern, TEAM * TEAMS, smem);
  if (resident < 1) return (int)cudaErrorInvalidConfiguration;
  long long grid = (long long)sms * resident;
  if (Body::kColumns > 0 && grid > Body::kPartials) grid = Body::kPartials;
  if (grid > groups) grid = groups;
  if (blocks != nullptr) *blocks = grid;
  return (int)launch_pdl(kern, (unsigned)grid, TEAM * TEAMS, smem, (cudaStream_t)stream, body, rows, cols, false);
}

// ---- outer reduction family -----------------------------------------------------------------
// The kept (x) axis is stride-1 in memory and the reduced axis is not.  Threads form a
// TX x TY grid: TX threads cover the contiguous run of the kept axis (kVec elements each;
// TX is chosen by the generator so that TX * kVec elements are adjacent in memory) and the
// TY thread rows split the reduced axis.  With a short run a warp therefore reads 32 / TX
// consecutive reduced indices, which are adjacent spans when the reduced stride equals the
// run.  Partial vectors are folded by shuffles inside a warp and through shared memory
// across warps.  The generated body carries the loop over the reduced index itself:
//   Body::tile<FAST>(ctx, xbase, nvalid)  - for (r = ctx.ty; r < rnumel; r += kTY) {...},
//                                           then ctx.combine<Op>(acc), epilogue, stores by
//                                           the thread row ty == 0.
template <int V, int TX, int TY> struct OuterCtx {
  static constexpr int kTY = TY;
  static constexpr int kWarps = TX * TY / 32;
  static constexpr int kRowsPerWarp = 32 / TX;   // thread rows that share a warp
  static_assert(TX <= 32 && 32 % TX == 0 && (TX * TY) % 32 == 0, "thread grid must tile warps");
  int tx, ty;
  float* part;  // [kWarps][TX * V]
  // the reduced indices this thread row walks, and who stores the result of a tile
  __device__ __forceinline__ long long rbegin() const { return ty; }
  __device__ __forceinline__ long long rstep() const { return TY; }
  __device__ __forceinline__ bool writer() const { return ty == 0; }

  template <int N> static __device__ __forceinline__ vf<N> splat(float v) {
    vf<N> r;
#pragma unroll
    for (int i = 0; i < N; ++i) r.v[i] = v;
    return r;
  }
  using ISum = ::ixb::gen::ISum;
  using IProd = ::ixb::gen::IProd;
  using IMax = ::ixb::gen::IMax;
  using IMin = ::ixb::gen::IMin;
  template <int N> static __device__ __forceinline__ vi<N> splat_int(long long v) {
    vi<N> r;
#pragma unroll
    for (int i = 0; i < N; ++i) r.v[i] = v;
    return r;
  }
  // exact integer fold: the shared scratch is sized for floats, so the 64-bit partials of
  // the warps cross it in two rounds (low and high halves would not fold; values do)
  template <class IOp> __device__ __forceinline__ vi<V> combine_int(const vi<V>& acc) {
    vi<V> r = acc;
#pragma unroll
    for (int off = TX; off < 32; off <<= 1)
#pragma unroll
      for (int i = 0; i < V; ++i) r.v[i] = IOp::f(r.v[i], __shfl_xor_sync(kFull, r.v[i], off));
    if constexpr (kWarps > 1) {
      const int warp = (ty * TX + tx) >> 5;
      long long* ipart = reinterpret_cast<long long*>(part);
      // the scratch holds kWarps * TX * V floats = half as many 64-bit values: fold the
      // vector in two halves
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        constexpr int HV = (V + 1) / 2;
        if (ty % kRowsPerWarp == 0) {
#pragma unroll
          for (int i = 0; i < HV; ++i)
            if (h * HV + i < V) ipart[(warp * TX + tx) * HV + i] = r.v[h * HV + i];
        }
        __syncthreads();
        if (writer()) {
#pragma unroll
          for (int i = 0; i < HV; ++i) {
            if (h * HV + i < V) {
              long long a = ipart[tx * HV + i];
#pragma unroll
              for (int w = 1; w < kWarps; ++w) a = IOp::f(a, ipart[(w * TX + tx) * HV + i]);
              r.v[h * HV + i] = a;
            }
          }
        }
        __syncthreads();
      }
    }
    return r;
  }
  // fold the TY partial vectors; the writer row receives the result
  template <class Op> __device__ __forceinline__ vf<V> combine(const vf<V>& acc) {
    vf<V> r = acc;
#pragma unroll
    for (int off = TX; off < 32; off <<= 1)
#pragma unroll
      for (int i = 0; i < V; ++i) r.v[i] = Op::combine(r.v[i], __shfl_xor_sync(kFull, r.v[i], off));
    if constexpr (kWarps > 1) {
      const int warp = (ty * TX + tx) >> 5;
      if (ty % kRowsPerWarp == 0) {
#pragma unroll
        for (int i = 0; i < V; ++i) part[(warp * TX + tx) * V + i] = r.v[i];
      }
      __syncthreads();
      // only the thread row that stores the tile needs the folded vector (a generated outer
      // kernel has one reduction and nothing after it but the store): the other rows skip
      // the kWarps x V shared-memory reads
      if (writer()) {
#pragma unroll
        for (int i = 0; i < V; ++i) {
          float a = part[tx * V + i];
#pragma unroll
          for (int w = 1; w < kWarps; ++w) a = Op::combine(a, part[(w * TX + tx) * V + i]);
          r.v[i] = a;
        }
      }
      __syncthreads();
    }
    return r;
  }
};

// GROUPS tiles a CTA: more than one where a tile is the work of one warp, whose fold is shuffles alone.
template <class Body, int TX, int TY, int GROUPS, bool ALIGNED>
__global__ void __launch_bounds__(TX* TY* GROUPS) outer_gen_kernel(const Body body, const long long xnumel) {
  static_assert(GROUPS == 1 || TX * TY == 32, "several tiles a CTA: a warp each");
  constexpr int V = Body::kVec;
  __shared__ __align__(16) float part[(TX * TY / 32) * TX * V];
  OuterCtx<V, TX, TY> c;
  c.tx = threadIdx.x % TX;
  c.ty = threadIdx.x / TX % TY;
  c.part = part;
  const long long per_cta = (long long)TX * V;
  const long long ntiles = (xnumel + per_cta - 1) / per_cta;
  for (long long t = (long long)blockIdx.x * GROUPS + threadIdx.x / (TX * TY); t < ntiles; t += (long long)gridDim.x * GROUPS) {
    const long long xbase = t * per_cta + (long long)c.tx * V;
    const long long left = xnumel - xbase;
    // the choice is uniform per tile (the fold synchronises all that work on it)
    if (ALIGNED && xnumel - t * per_cta >= per_cta) body.template tile<true>(c, xbase, V);
    else body.template tile<false>(c, xbase, left >= V ? V : (left > 0 ? (int)left : 0));
  }
}
// ---- outer reduction split over a thread-block cluster -----------------------------------------
// When the kept extent gives fewer tiles than the GPU has SMs and the reduced axis is long, a
// cluster of CS CTAs shares one tile: rank k walks the reduced indices k * TY + ty, + TY * CS, ...
// and the partial vectors meet in the shared memory of rank 0 (distributed shared memory):
// every other rank stores its vector there (st.shared::cluster to the address mapa gives) and
// arrives on rank 0's mbarrier with cluster-scope release; rank 0 waits on it with a bounded
// acquire wait, folds and stores.  This is the reference's outer split
// (inductor_x/codegen/split_tiling.py:159-165), which combines with atomic adds in global
// memory; here nothing leaves the chip.  One tile per cluster, so the inbox is used once.
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
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// bounded wait with cluster-scope acquire (the data was written by other CTAs of the cluster)
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, 1000000;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > kWaitCycles) {
      atomicAdd(&g_wait_timeouts, 1u);
      return false;
    }
  }
}

template <int V, int TX, int TY, int CS> struct OuterSplitCtx : OuterCtx<V, TX, TY> {
  using Base = OuterCtx<V, TX, TY>;
  int rank = 0;      // CTA rank inside the cluster
  float* inbox;      // [CS - 1][TX * V]; only rank 0's copy is written to
  uint64_t* bar;     // arrivals of the other ranks; only rank 0's copy is used
  bool ok = true;    // false after rank 0's wait gave up: the tile is not stored
  __device__ __forceinline__ long long rbegin() const { return (long long)rank * TY + this->ty; }
  __device__ __forceinline__ long long rstep() const { return (long long)TY * CS; }
  __device__ __forceinline__ bool writer() const { return this->ty == 0 && rank == 0 && ok; }
  template <class Op> __device__ __forceinline__ vf<V> combine(const vf<V>& acc) {
    vf<V> r = Base::template combine<Op>(acc);   // the CTA's own partial, in every thread row
    if (this->ty != 0) return r;
    if (rank != 0) {
      const uint32_t dst = map_to_rank(inbox + ((rank - 1) * TX + this->tx) * V, 0);
#pragma unroll
      for (int i = 0; i < V; ++i) st_cluster_f32(dst + 4 * i, r.v[i]);
      mbar_arrive_remote(map_to_rank(bar, 0));
    } else {
      ok = mbar_wait_cluster(bar, 0);
      if (ok) {
#pragma unroll
        for (int k = 0; k < CS - 1; ++k)
#pragma unroll
          for (int i = 0; i < V; ++i) r.v[i] = Op::combine(r.v[i], inbox[(k * TX + this->tx) * V + i]);
      }
    }
    return r;
  }
};

template <class Body, int TX, int TY, int CS, bool ALIGNED>
__global__ void __launch_bounds__(TX* TY) outer_split_gen_kernel(const Body body, const long long xnumel) {
  constexpr int V = Body::kVec;
  __shared__ __align__(16) float part[(TX * TY / 32) * TX * V];
  __shared__ __align__(16) float inbox[(CS - 1) * TX * V];
  __shared__ __align__(8) uint64_t bar;
  OuterSplitCtx<V, TX, TY, CS> c;
  c.tx = threadIdx.x % TX;
  c.ty = threadIdx.x / TX;
  c.part = part;
  c.inbox = inbox;
  c.bar = &bar;
  c.rank = (int)cluster_rank();
  if (c.rank == 0 && threadIdx.x == 0) {
    mbar_init(&bar, (CS - 1) * TX);
    mbar_init_fence();
  }
  // every CTA of the cluster is resident and rank 0's barrier is initialised before anyone pushes
  cluster_sync_all();
  const long long per_cta = (long long)TX * V;
  const long long t = blockIdx.x / CS;   // one tile per cluster
  const long long xbase = t * per_cta + (long long)c.tx * V;
  const long long left = xnumel - xbase;
  if (ALIGNED && xnumel - t * per_cta >= per_cta) body.template tile<true>(c, xbase, V);
  else body.template tile<false>(c, xbase, left >= V ? V : (left > 0 ? (int)left : 0));
}
template <class Body, int TX, int CS>
int launch_outer_split_gen(const Body& body, long long xnumel, void* stream, bool aligned = false) {
  if (xnumel <= 0) return 0;
  constexpr int TY = 256 / TX;
  const long long per_cta = (long long)TX * Body::kVec;
  const long long tiles = (xnumel + per_cta - 1) / per_cta;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * CS));
  cfg.blockDim = dim3(TX * TY);
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (aligned) return (int)cudaLaunchKernelEx(&cfg, outer_split_gen_kernel<Body, TX, TY, CS, true>, body, xnumel);
  return (int)cudaLaunchKernelEx(&cfg, outer_split_gen_kernel<Body, TX, TY, CS, false>, body, xnumel);
}

// Short reduced axes: with 256 threads to a tile each would add one or two vectors and then wait for two
// barriers of the CTA.  A warp a tile has eight times as many steps a thread and folds by shuffles.
// Bound: HBM.  Maximum over the 26 of 6163 x 26 x 22 x 32 bf16 (memory order): see _outer_warp.
template <class Body, int TX>
int launch_outer_warps_gen(const Body& body, long long xnumel, void* stream, bool aligned = false) {
  if (xnumel <= 0) return 0;
  constexpr int TY = 32 / TX, GROUPS = 8;
  const long long tiles = (xnumel + (long long)TX * Body::kVec - 1) / ((long long)TX * Body::kVec);
  long long grid = (tiles + GROUPS - 1) / GROUPS;
  if (grid > 0x7fffffffLL) grid = 0x7fffffffLL;
  if (aligned) outer_gen_kernel<Body, TX, TY, GROUPS, true><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(body, xnumel);
  else outer_gen_kernel<Body, TX, TY, GROUPS, false><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(body, xnumel);
  return (int)cudaGetLastError();
}

template <class Body, int TX = 32>
int launch_outer_gen(const Body& body, long long xnumel, void* stream, bool aligned = false) {
  if (xnumel <= 0) return 0;
  constexpr int TY = 256 / TX;
  static const long long cap_a = resident_ctas(outer_gen_kernel<Body, TX, TY, 1, true>, TX * TY);
  static const long long cap_u = resident_ctas(outer_gen_kernel<Body, TX, TY, 1, false>, TX * TY);
  const long long per_cta = (long long)TX * Body::kVec;
  long long grid = (xnumel + per_cta - 1) / per_cta;
  // A tile ends with a CTA-wide fold during which the CTA has no loads in flight, so the grid
  // holds several waves of CTAs (the hardware starts the next CTA's loads while another folds)
  // instead of exactly the resident set.  IXB_OUTER_WAVES overrides the default.
  static const long long waves = [] {
    const char* v = getenv("IXB_OUTER_WAVES");
    const long long w = v != nullptr ? atoll(v) : 2;
    return w < 1 ? 1 : w;
  }();
  const long long cap = (aligned ? cap_a : cap_u) * waves;
  if (grid > cap) grid = cap;
  if (aligned) outer_gen_kernel<Body, TX, TY, 1, true><<<(unsigned)grid, TX * TY, 0, (cudaStream_t)stream>>>(body, xnumel);
  else outer_gen_kernel<Body, TX, TY, 1, false><<<(unsigned)grid, TX * TY, 0, (cudaStream_t)stream>>>(body, xnumel);
  return (int)cudaGetLastError();
}

}  // namespace gen
}  // namespace ixb
