// C-ABI entry points of the fused ROW-family graphs (persistent row template).
#include "host.h"
#include "ixb/row_bodies.cuh"

namespace {

using ixb_host::aligned16;

// Resolve the launch configuration: the caller's, or the chooser's.
int resolve_cfg(const ixb_cfg* user, int64_t cols, int elsize, int max_vpt, ixb_cfg* cfg) {
  if (user != nullptr && user->team > 0 && user->vpt > 0) {
    *cfg = *user;
    const int64_t vec = 16 / elsize;
    if ((int64_t)cfg->team * cfg->vpt * vec < cols) return IXB_ERR_SHAPE;
    return IXB_OK;
  }
  ixb_cfg c = {};
  if (!ixb_host::choose_row(cols, elsize, max_vpt, &c)) return IXB_ERR_SHAPE;
  if (user != nullptr) c.grid = user->grid;
  *cfg = c;
  return IXB_OK;
}

template <typename T>
int softmax_layernorm_t(const void* x, const void* g, const void* gamma, const void* beta, void* y,
                        int64_t rows, int64_t cols, float eps, const ixb_cfg* user,
                        ixb_stream stream) {
  using Body = ixb::SoftmaxLayerNorm<T>;
  const ixb_devinfo* dev = ixb_host::current_device();
  if (dev == nullptr) return IXB_ERR_CUDA;
  ixb_cfg cfg;
  if (int st = resolve_cfg(user, cols, sizeof(T), 4, &cfg)) return st;
  typename Body::Params p{(const T*)x, (const T*)g, (const T*)gamma, (const T*)beta, (T*)y, eps};
  const bool al = cols % Body::kVec == 0 && aligned16(x) && aligned16(g) && aligned16(gamma) &&
                  aligned16(beta) && aligned16(y);
  if (al) {
    IXB_ROW_DISPATCH(Body, true)
  } else {
    IXB_ROW_DISPATCH(Body, false)
  }
  return IXB_ERR_UNSUPPORTED;
}

// Vectors of memory that a row may touch, wherever it begins.
int64_t vectors_touched(int64_t cols, int vec) { return (cols + vec - 1 + vec - 1) / vec; }

// Launch shape of a row worked on in the vectors of memory: the least of the dispatched capacities that
// holds the vectors it may touch.
bool choose_shift(int64_t cols, int vec, ixb_cfg* cfg) {
  const int64_t touched = vectors_touched(cols, vec);
  for (int team = 32; team <= 1024; team *= 2)
    for (int vpt = team == 32 ? 1 : 3; vpt <= 4; ++vpt)
      if ((int64_t)team * vpt >= touched) {
        cfg->team = team;
        cfg->vpt = vpt;
        return true;
      }
  return false;
}

template <typename T, bool RES>
int rmsnorm_t(const void* x, const void* res, const void* w, void* y, void* h_out, int64_t rows,
              int64_t cols, float eps, const ixb_cfg* user, ixb_stream stream) {
  using Body = ixb::RmsNorm<T, RES>;
  const ixb_devinfo* dev = ixb_host::current_device();
  if (dev == nullptr) return IXB_ERR_CUDA;
  ixb_cfg cfg;
  if (int st = resolve_cfg(user, cols, sizeof(T), 4, &cfg)) return st;
  typename Body::Params p{(const T*)x, (const T*)res, (const T*)w, (T*)y, (T*)h_out, eps};
  const bool al = cols % Body::kVec == 0 && aligned16(x) && aligned16(res) && aligned16(w) &&
                  aligned16(y) && aligned16(h_out);
  // Rows off a boundary whose operands all have the same offset from it (bases alike modulo 16 bytes and
  // a multiple of the element) are worked on in the vectors of memory: one load a vector, requested a row
  // ahead, in place of two that are shifted on the spot.  Measured, covering words -> this: fp32 7847 x 2077
  // 58.8 -> 21.0 us, with residual 100 -> 47.8; fp16 1094 x 9460 21.7 -> 10.1; bf16 40000 x 1537 with
  // residual 185 -> 97; 100000 x 67 36.8 -> 25.1; fp32 1094 x 9460, the nearest, 15.7 -> 14.9.
  // Short rows of 16 bits, so few of them that hardly one is asked for ahead of another, keep the covering words:
  // the words at their ends, cut element by element, are most of the work.  Covering words and this, fp16:
  // 250 x 77 2.0 and 2.3 us, 250 x 333 2.1 and 2.4, 1000 x 131 2.3 and 2.4, with residual 2000 x 131 3.1 and 3.5; from
  // 50000 vectors on, 4000 x 131 3.4 and 3.3, 2000 x 333 3.1 and 3.0, 8000 x 77 4.1 and 3.6.
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) & 15u;
  auto alike = [at](const void* q) { return q == nullptr || (reinterpret_cast<uintptr_t>(q) & 15u) == at; };
  ixb_cfg shift = {};
  if (!al && at % sizeof(T) == 0 && alike(res) && alike(y) && alike(h_out) && (user == nullptr || user->team <= 0 || user->vpt <= 0) &&
      choose_shift(cols, Body::kVec, &shift) &&
      !(sizeof(T) == 2 && shift.team == 32 && shift.vpt <= (RES ? 1 : 2) && rows * vectors_touched(cols, Body::kVec) < 50000)) {
    shift.grid = cfg.grid;
    cfg = shift;
    int period = Body::kVec;
    while (period > 1 && cols * (period / 2) % Body::kVec == 0) period /= 2;
    IXB_ROW_SHIFT_DISPATCH(Body)
  }
  if (al) {
    IXB_ROW_DISPATCH(Body, true)
  } else {
    IXB_ROW_DISPATCH(Body, false)
  }
  return IXB_ERR_UNSUPPORTED;
}

}  // namespace

extern "C" {

int ixb_affine_gelu_rowsum_f32(const float* x, const float* w, const float* b, float* out,
                               int64_t rows, int64_t cols, const ixb_cfg* user,
                               ixb_stream stream) {
  using Body = ixb::AffineGeluRowSum;
  if (rows < 0 || cols <= 0) return IXB_ERR_ARG;
  if (rows == 0) return IXB_OK;
  if (x == nullptr || w == nullptr || b == nullptr || out == nullptr) return IXB_ERR_ARG;
  const ixb_devinfo* dev = ixb_host::current_device();
  if (dev == nullptr) return IXB_ERR_CUDA;
  ixb_cfg cfg;
  // two vectors per thread keep w and b in registers (measured 9.1 us vs 11.6 us at four
  // vectors per thread on 8192 x 1024); longer rows fall back to the general choice
  if (resolve_cfg(user, cols, 4, 2, &cfg) != IXB_OK) {
    if (int st = resolve_cfg(user, cols, 4, 8, &cfg)) return st;
  }
  Body::Params p{x, w, b, out};
  const bool al = cols % 4 == 0 && aligned16(x) && aligned16(w) && aligned16(b);
  if (al) {
    IXB_ROW_DISPATCH(Body, true)
  } else {
    IXB_ROW_DISPATCH(Body, false)
  }
  return IXB_ERR_UNSUPPORTED;
}

int ixb_softmax_layernorm(int dtype, const void* x, const void* g, const void* gamma,
                          const void* beta, void* y, int64_t rows, int64_t cols, float eps,
                          const ixb_cfg* cfg, ixb_stream stream) {
  if (rows < 0 || cols <= 0) return IXB_ERR_ARG;
  if (rows == 0) return IXB_OK;
  if (!x || !g || !gamma || !beta || !y) return IXB_ERR_ARG;
  switch (dtype) {
    case IXB_BF16:
      return softmax_layernorm_t<ixb::bf16>(x, g, gamma, beta, y, rows, cols, eps, cfg, stream);
    case IXB_F16:
      return softmax_layernorm_t<ixb::f16>(x, g, gamma, beta, y, rows, cols, eps, cfg, stream);
    case IXB_F32:
      return softmax_layernorm_t<float>(x, g, gamma, beta, y, rows, cols, eps, cfg, stream);
    default:
      return IXB_ERR_DTYPE;
  }
}

int ixb_rmsnorm(int dtype, const void* x, const void* res, const void* w, void* y, void* h_out,
                int64_t rows, int64_t cols, float eps, const ixb_cfg* cfg, ixb_stream stream) {
  if (rows < 0 || cols <= 0) return IXB_ERR_ARG;
  if (rows == 0) return IXB_OK;
  if (!x || !w || !y) return IXB_ERR_ARG;
  if (res == nullptr && h_out != nullptr) return IXB_ERR_ARG;
  switch (dtype) {
    case IXB_BF16:
      return res ? rmsnorm_t<ixb::bf16, true>(x, res, w, y, h_out, rows, cols, eps, cfg, stream)
                 : rmsnorm_t<ixb::bf16, false>(x, res, w, y, h_out, rows, cols, eps, cfg, stream);
    case IXB_F16:
      return res ? rmsnorm_t<ixb::f16, true>(x, res, w, y, h_out, rows, cols, eps, cfg, stream)
                 : rmsnorm_t<ixb::f16, false>(x, res, w, y, h_out, rows, cols, eps, cfg, stream);
    case IXB_F32:
      return res ? rmsnorm_t<float, true>(x, res, w, y, h_out, rows, cols, eps, cfg, stream)
                 : rmsnorm_t<float, false>(x, res, w, y, h_out, rows, cols, eps, cfg, stream);
    default:
      return IXB_ERR_DTYPE;
  }
}

}  // extern "C"
