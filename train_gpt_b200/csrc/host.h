// What the host path's translation units share: the C ABI by address, checks and allocation, and quantised operands as raw
// memory (Arena, Form) with the calls that fill and contract them.
#ifndef TRAIN_GPT_B200_HOST_H_
#define TRAIN_GPT_B200_HOST_H_

#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <array>
#include <atomic>
#include <optional>
#include <sstream>
#include <string>
#include <utility>
#include <vector>

#include "../../include/train_gpt_b200.h"
#include "host_api.h"

namespace tgh {

namespace py = pybind11;
using at::Tensor;
using Pair = std::pair<Tensor, Tensor>;

constexpr int64_t kTile = 128;
constexpr auto kF8 = at::kFloat8_e4m3fn;

// ---- the C ABI, by address ------------------------------------------------------------------------------------

#define TG_API(X)                                                                                                  \
  X(tg_last_cuda_error) X(tg_quantize_rowwise) X(tg_quantize_colwise) X(tg_quantize_rowcol) X(tg_quantize_rowcol_ld) \
  X(tg_act_quantize_rowcol) X(tg_quantize_block128) X(tg_rmsnorm_fwd) X(tg_rmsnorm_quant_fwd)                       \
  X(tg_add_rmsnorm_quant_fwd) X(tg_rmsnorm_bwd_scratch_bytes) X(tg_rmsnorm_bwd) X(tg_rmsnorm_bwd_add) X(tgh_rmsnorm_bwd_parts) X(tgh_dgamma_reduce) \
  X(tg_softcap_ce_fwd) X(tg_softcap_ce_bwd) X(tg_sumsq_scratch_bytes) X(tg_sumsq_bf16) X(tg_adamw_bf16)             \
  X(tg_gemm_workspace_bytes) X(tg_gemm_fp8_blockscaled) X(tgh_gemm_two) X(tgh_quantize_jobs) X(tgh_softcap_ce_fits) X(tgh_softcap_ce) X(tgh_mean) \
  X(tgh_global_norm_scratch_bytes) X(tgh_global_norm) X(tgh_adamw) X(tgh_embed) X(tgh_embed_bwd_cleared)

struct Api {
#define X(name) decltype(&::name) name = nullptr;
  TG_API(X)
#undef X
};
extern Api api;

// a launcher's status as an exception: ValueError for sizes the kernel cannot take, RuntimeError for the rest
inline void check(int rc, const char* what) {
  if (rc == TG_OK) return;
  const char* name = rc == TG_ERR_SHAPE ? "TG_ERR_SHAPE" : rc == TG_ERR_ALIGN ? "TG_ERR_ALIGN" : rc == TG_ERR_ARCH ? "TG_ERR_ARCH"
                     : rc == TG_ERR_CUDA ? "TG_ERR_CUDA" : rc == TG_ERR_TOO_LARGE ? "TG_ERR_TOO_LARGE" : "unknown status";
  const std::string msg = std::string(what) + ": " + name;
  if (rc == TG_ERR_SHAPE || rc == TG_ERR_TOO_LARGE || rc == TG_ERR_ALIGN) throw py::value_error(msg);
  throw std::runtime_error(rc == TG_ERR_CUDA ? msg + " " + api.tg_last_cuda_error() : msg);
}

// ---- small helpers -----------------------------------------------------------------------------------------------

template <typename... A>
inline std::string cat(const A&... a) {
  std::ostringstream o;
  (o << ... << a);
  return o.str();
}

inline std::string dtype_name(at::ScalarType t) {
  switch (t) {
    case at::kBFloat16: return "torch.bfloat16";
    case at::kFloat: return "torch.float32";
    case at::kHalf: return "torch.float16";
    case at::kDouble: return "torch.float64";
    default: return c10::toString(t);
  }
}

inline Tensor need(const Tensor& t, at::ScalarType dt, const char* name) {
  if (!t.is_cuda()) throw std::runtime_error(cat(name, " must be a CUDA tensor (there is no CPU path)"));
  if (t.scalar_type() != dt) throw py::type_error(cat(name, " must be ", dtype_name(dt), ", got ", dtype_name(t.scalar_type())));
  return t.is_contiguous() ? t : t.contiguous();
}

inline int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

// New CUDA memory straight from the allocator: at::empty is the same behind a dispatcher call.  With it, and with the conversions that
// change nothing also going through the dispatcher, the two calls of a decode step took the host 10.7 us instead of 9.7.
inline Tensor empty(at::IntArrayRef shape, at::ScalarType dt, const Tensor& like) {
  return at::detail::empty_cuda(shape, dt, like.device(), std::nullopt);
}
inline Tensor empty_as(const Tensor& contiguous) { return empty(contiguous.sizes(), contiguous.scalar_type(), contiguous); }

// t in another type or shape; no dispatcher call where it has them
inline Tensor to(const Tensor& t, at::ScalarType dt) { return t.scalar_type() == dt ? t : t.to(dt); }
inline Tensor as_rows(const Tensor& t, int64_t rows, int64_t cols) { return t.dim() == 2 ? t : t.reshape({rows, cols}); }

inline void* cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

inline float* fptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

inline std::vector<int64_t> with_last(const Tensor& x, int64_t last) {
  std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
  s.back() = last;
  return s;
}

// losses.py:12: the mean of the tokens' values
inline Tensor mean_of(const Tensor& nll) {
  if (nll.numel() > 65536) return nll.mean();
  const Tensor m = empty({}, at::kFloat, nll);
  check(api.tgh_mean(fptr(nll), nll.numel(), fptr(m), cur_stream()), "tgh_mean");
  return m;
}

// The word a GEMM reports an expired device wait in, one per device (-1: the current one), made once.
Tensor status_word(int64_t device);

// kernels the most recent GEMM launched (1, or 2 with the reduce of a cut contraction)
extern std::atomic<int> last_gemm_launches;

struct Strides {
  int64_t row, kb;
};

// Device memory for several temporaries of one call, or for what a node keeps, as ONE allocation: a caching-allocator
// round trip costs about as much host time as a third of a launch, and a linear has up to ten such buffers.
class Arena {
 public:
  size_t add(int64_t bytes) {
    const size_t at = size_;
    size_ += (size_t(bytes) + 255) / 256 * 256;
    return at;
  }
  void make(const Tensor& like) {
    if (size_ > 0) memory_ = empty({int64_t(size_)}, at::kByte, like);
    base_ = size_ > 0 ? static_cast<uint8_t*>(memory_.data_ptr()) : nullptr;
  }
  void* at(size_t offset) const { return base_ + offset; }
  const Tensor& memory() const { return memory_; }

 private:
  size_t size_ = 0;
  uint8_t* base_ = nullptr;
  Tensor memory_;
};

// One quantised matrix: e4m3 bytes and float32 scales
struct Form {
  void* q = nullptr;
  float* s = nullptr;
  explicit operator bool() const { return q != nullptr; }
};
struct FormAt {
  size_t q = 0, s = 0;
  Form in(const Arena& m) const { return {m.at(q), static_cast<float*>(m.at(s))}; }
};
inline FormAt add_row(Arena& m, int64_t rows, int64_t cols) { return {m.add(rows * cols), m.add(rows * (cols / kTile) * 4)}; }
inline FormAt add_col(Arena& m, int64_t rows, int64_t cols) { return {m.add(rows * cols), m.add(cdiv(rows, kTile) * cols * 4)}; }
inline FormAt add_block(Arena& m, int64_t rows, int64_t cols) { return {m.add(rows * cols), m.add(cdiv(rows, kTile) * (cols / kTile) * 4)}; }

// A 2-D bf16 matrix the quantisers can read as it lies: unit stride along a row and, unless it is only wanted by column,
// rows at 16-byte boundaries.  Anything else is copied.
inline Tensor readable(const Tensor& t, bool any_alignment) {
  if (t.stride(1) == 1 && (t.size(0) <= 1 || t.stride(0) >= t.size(1)) &&
      (any_alignment || ((t.size(0) <= 1 || t.stride(0) % 8 == 0) && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0)))
    return t;
  return t.contiguous();
}
inline int64_t pitch(const Tensor& t) { return t.size(0) > 1 ? t.stride(0) : t.size(1); }

inline tgh_quantize_job job_of(const Tensor& x) {
  tgh_quantize_job j = {};
  j.x = x.data_ptr();
  j.rows = x.size(0);
  j.cols = x.size(1);
  j.ld = pitch(x);
  return j;
}
inline void want_row(tgh_quantize_job& j, const Form& f) {
  j.q_row = f.q; j.s_row = f.s; j.q_row_ld = j.cols; j.s_row_ld = j.cols / kTile;
}
inline void want_col(tgh_quantize_job& j, const Form& f, int64_t ld) {
  j.form = TGH_FORM_COLUMNS; j.q = f.q; j.s = f.s; j.q_ld = j.s_ld = ld;
}
inline void want_block(tgh_quantize_job& j, const Form& f) {
  j.form = TGH_FORM_BLOCKS; j.q = f.q; j.s = f.s; j.q_ld = j.cols; j.s_ld = j.cols / kTile;
}

// A GEMM of forms.  (rows of A, columns of B and their contraction; see gemm_fwd / gemm_dgrad / gemm_wgrad for the layouts)
inline tg_gemm_args gemm_args(int64_t m, int64_t n, int64_t k, int64_t lda, int a_major, Strides sa, int64_t ldb, int b_major, Strides sb,
                       bool per_column, int64_t ldd, bool f32, unsigned* status) {
  tg_gemm_args g = {};
  g.lda = lda; g.ldb = ldb; g.a_major = a_major; g.b_major = b_major;
  g.sa_stride_m = sa.row; g.sa_stride_kb = sa.kb; g.sb_stride_n = sb.row; g.sb_stride_kb = sb.kb;
  g.sb_gran_n = per_column ? 1 : int(kTile);
  g.ldd = ldd; g.out_dtype = f32 ? TG_OUT_F32 : TG_OUT_BF16;
  g.M = m; g.N = n; g.K = k;
  g.status = status;
  return g;
}
inline void set_operands(tg_gemm_args& g, const Form& a, const Form& b, void* d, void* workspace, int64_t workspace_bytes) {
  g.a = a.q; g.sa = a.s; g.b = b.q; g.sb = b.s;
  g.d = d;
  g.workspace = workspace_bytes > 0 ? workspace : nullptr;
  g.workspace_bytes = workspace_bytes;
}
inline void run_gemm(tg_gemm_args& g, const Form& a, const Form& b, void* d, void* workspace, int64_t workspace_bytes) {
  set_operands(g, a, b, d, workspace, workspace_bytes);
  check(api.tg_gemm_fp8_blockscaled(&g, cur_stream()), "tg_gemm_fp8_blockscaled");
  last_gemm_launches.store(workspace_bytes > 0 ? 2 : 1, std::memory_order_relaxed);
}
inline unsigned* status_of(const Tensor& like) { return static_cast<unsigned*>(ptr(status_word(like.get_device()))); }

void register_step(py::module_& m);      // step.cpp

}  // namespace tgh

#endif
