// The host path of the torch-facing API, native: argument checks, output allocation, the C-ABI calls of
// include/train_gpt_b200.h and the autograd nodes of the public functions.
//
// Most calls of this library are short -- a decode step's GEMM runs for 8 us -- and the Python that used to
// prepare them (ctypes structures, shape arithmetic, torch.empty, torch.autograd.Function) took 10 to 15 us per
// kernel and held the GPU back in every call below about 100 us.  Here a launch costs 3 to 4 us of host time and
// the backward pass runs on the autograd engine's own thread without the interpreter lock.
//
// The kernels stay behind the C ABI: bind() takes the addresses of the one loaded library (the same image ctypes
// uses), so a build named by TRAIN_GPT_B200_LIB serves both.
#include "host.h"

#include <dlfcn.h>
#include <torch/csrc/autograd/engine.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <functional>
#include <memory>
#include <mutex>
#include <tuple>

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace tgh {

Api api;
std::atomic<int> last_gemm_launches{0};

// The word a GEMM reports an expired device wait in, one per device, made once (so that a captured CUDA graph
// keeps pointing at it) and never freed: the CUDA context may be gone by the time static objects are.
Tensor status_word(int64_t device) {
  static std::mutex mu;
  static auto* words = new std::array<Tensor, 64>();
  if (device < 0) device = c10::cuda::current_device();
  std::lock_guard<std::mutex> lock(mu);
  Tensor& w = words->at(size_t(device));
  if (!w.defined()) w = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, c10::DeviceIndex(device)));
  return w;
}

}  // namespace tgh

namespace {

using namespace tgh;

constexpr int64_t kAddNormMaxCols = 2048;   // rows the fused add + norm kernels take

void bind(const std::string& path) {
  void* lib = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (lib == nullptr) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
#define X(name)                                                                       \
  api.name = reinterpret_cast<decltype(api.name)>(dlsym(lib, #name));                 \
  if (api.name == nullptr) throw std::runtime_error(path + " does not export " #name);
  TG_API(X)
#undef X
}

void need_2d(const Tensor& t, const char* what) {
  if (t.dim() != 2) throw py::value_error(cat(what, " takes a 2-D tensor"));
}

// ---- quantisers -----------------------------------------------------------------------------------------------

void need_tiles(int64_t k) {
  if (k % kTile) throw py::value_error(cat("K=", k, " not divisible by block_k=", kTile));
}

Pair quantize_rowwise(const Tensor& x_) {
  const Tensor x = need(x_, at::kBFloat16, "x");
  const int64_t k = x.size(-1);
  need_tiles(k);
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor q = empty(x.sizes(), kF8, x), s = empty(with_last(x, k / kTile), at::kFloat, x);
  check(api.tg_quantize_rowwise(ptr(x), ptr(q), fptr(s), k ? x.numel() / k : 0, k, cur_stream()), "tg_quantize_rowwise");
  return {q, s};
}

Pair quantize_colwise(const Tensor& x_) {
  const Tensor x = need(x_, at::kBFloat16, "x");
  need_2d(x, "quantize_colwise");
  const int64_t r = x.size(0), c = x.size(1);
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor q = empty({r, c}, kF8, x), s = empty({cdiv(r, kTile), c}, at::kFloat, x);
  check(api.tg_quantize_colwise(ptr(x), ptr(q), fptr(s), r, c, cur_stream()), "tg_quantize_colwise");
  return {q, s};
}

Pair quantize_block128(const Tensor& x_) {
  const Tensor x = need(x_, at::kBFloat16, "x");
  need_2d(x, "quantize_block128");
  const int64_t r = x.size(0), c = x.size(1);
  if (c % kTile) throw py::value_error(cat("C=", c, " not divisible by ", kTile));
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor q = empty({r, c}, kF8, x), s = empty({cdiv(r, kTile), c / kTile}, at::kFloat, x);
  check(api.tg_quantize_block128(ptr(x), ptr(q), fptr(s), r, c, cur_stream()), "tg_quantize_block128");
  return {q, s};
}

struct RowCol {
  Tensor q_row, s_row, q_col, s_col;
  py::tuple tuple() const { return py::make_tuple(q_row, s_row, q_col, s_col); }
};

RowCol rowcol_like(const Tensor& x) {
  const int64_t r = x.size(0), c = x.size(1);
  return {empty({r, c}, kF8, x), empty({r, c / kTile}, at::kFloat, x), empty({r, c}, kF8, x), empty({cdiv(r, kTile), c}, at::kFloat, x)};
}

RowCol quantize_rowcol(const Tensor& x_) {
  const Tensor x = need(x_, at::kBFloat16, "x");
  need_2d(x, "quantize_rowcol");
  need_tiles(x.size(1));
  const c10::cuda::CUDAGuard guard(x.device());
  RowCol o = rowcol_like(x);
  check(api.tg_quantize_rowcol(ptr(x), ptr(o.q_row), fptr(o.s_row), ptr(o.q_col), fptr(o.s_col), x.size(0), x.size(1), cur_stream()),
        "tg_quantize_rowcol");
  return o;
}

// either form into column slices of wider matrices (see ops.quantize_rowcol)
RowCol quantize_rowcol_into(const Tensor& x_, const std::optional<Pair>& row_out, const std::optional<Pair>& col_out) {
  const Tensor x = need(x_, at::kBFloat16, "x");
  need_2d(x, "quantize_rowcol");
  const int64_t r = x.size(0), c = x.size(1);
  need_tiles(c);
  const c10::cuda::CUDAGuard guard(x.device());
  auto form = [&](const std::optional<Pair>& out, int64_t s_rows, int64_t s_cols, const char* what) -> Pair {
    if (!out) return {empty({r, c}, kF8, x), empty({s_rows, s_cols}, at::kFloat, x)};
    const Tensor &q = out->first, &s = out->second;
    if (q.scalar_type() != kF8 || s.scalar_type() != at::kFloat || !q.is_cuda() || !s.is_cuda() ||
        q.sizes() != at::IntArrayRef({r, c}) || s.sizes() != at::IntArrayRef({s_rows, s_cols}))
      throw py::type_error(cat(what, " must be an e4m3 (", r, ", ", c, ") and a float32 (", s_rows, ", ", s_cols, ") CUDA tensor"));
    if (q.stride(1) != 1 || s.stride(1) != 1) throw py::value_error(cat(what, " tensors must have unit stride along a row"));
    return *out;
  };
  const Pair row = form(row_out, r, c / kTile, "row_out"), col = form(col_out, cdiv(r, kTile), c, "col_out");
  auto ld = [](const Tensor& t, int64_t least) {      // a one-row tensor's row stride is arbitrary
    return t.size(0) > 1 ? std::max(t.stride(0), least) : least;
  };
  check(api.tg_quantize_rowcol_ld(ptr(x), ptr(row.first), ld(row.first, std::max<int64_t>(c, 16)), fptr(row.second),
                                  ld(row.second, c / kTile), ptr(col.first), ld(col.first, std::max<int64_t>(c, 16)),
                                  fptr(col.second), ld(col.second, c), r, c, cur_stream()),
        "tg_quantize_rowcol_ld");
  return {row.first, row.second, col.first, col.second};
}

RowCol act_quantize_rowcol(const Tensor& x_, int act, const std::string& act_name, const std::optional<Tensor>& gate_) {
  const Tensor x = need(x_, at::kBFloat16, "x");
  need_2d(x, "act_quantize_rowcol");
  Tensor gate;
  const bool bwd = act == TG_ACT_RELU2_BWD || act == TG_ACT_GELU_BWD;
  if (bwd) {
    if (!gate_) throw py::value_error(act_name + " needs the upstream gradient `gate`");
    gate = need(*gate_, at::kBFloat16, "gate");
    if (gate.sizes() != x.sizes()) throw py::value_error(cat("gate shape ", gate.sizes(), " != x shape ", x.sizes()));
  }
  need_tiles(x.size(1));
  const c10::cuda::CUDAGuard guard(x.device());
  RowCol o = rowcol_like(x);
  check(api.tg_act_quantize_rowcol(ptr(x), ptr(gate), act, ptr(o.q_row), fptr(o.s_row), ptr(o.q_col), fptr(o.s_col), x.size(0),
                                   x.size(1), cur_stream()),
        "tg_act_quantize_rowcol");
  return o;
}

// ---- norms --------------------------------------------------------------------------------------------------------

void need_gamma(const Tensor& gamma, int64_t d) {
  if (gamma.dim() != 1 || gamma.size(0) != d)
    throw py::value_error(cat("scale shape ", gamma.sizes(), " does not match last dim ", d));
}

Pair rmsnorm_fwd(const Tensor& x_, const Tensor& gamma_, double eps, bool pure, bool want_rnorm) {
  const Tensor x = need(x_, at::kBFloat16, "x"), gamma = need(gamma_, at::kBFloat16, "gamma");
  const int64_t d = x.size(-1);
  need_gamma(gamma, d);
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = empty_as(x), rn;
  if (want_rnorm) rn = empty(x.sizes().slice(0, x.dim() - 1), at::kFloat, x);
  check(api.tg_rmsnorm_fwd(ptr(x), ptr(gamma), float(eps), ptr(y), fptr(rn), x.numel() / d, d, pure ? TG_NORM_PURE : TG_NORM_FUSED,
                           cur_stream()),
        "tg_rmsnorm_fwd");
  return {y, rn};
}

struct NormQuant {
  Tensor q, s, y, rn;
};

NormQuant rmsnorm_quant_fwd(const Tensor& x_, const Tensor& gamma_, double eps, bool pure, bool want_y, bool want_rnorm) {
  const Tensor x = need(x_, at::kBFloat16, "x"), gamma = need(gamma_, at::kBFloat16, "gamma");
  const int64_t d = x.size(-1);
  need_gamma(gamma, d);
  need_tiles(d);
  const c10::cuda::CUDAGuard guard(x.device());
  NormQuant o;
  o.q = empty(x.sizes(), kF8, x);
  o.s = empty(with_last(x, d / kTile), at::kFloat, x);
  if (want_y) o.y = empty_as(x);
  if (want_rnorm) o.rn = empty(x.sizes().slice(0, x.dim() - 1), at::kFloat, x);
  check(api.tg_rmsnorm_quant_fwd(ptr(x), ptr(gamma), float(eps), ptr(o.q), fptr(o.s), ptr(o.y), fptr(o.rn), x.numel() / d, d,
                                 pure ? TG_NORM_PURE : TG_NORM_FUSED, cur_stream()),
        "tg_rmsnorm_quant_fwd");
  return o;
}

struct AddNorm {
  Tensor sum, q, s, y;
};

AddNorm add_rmsnorm_quant_fwd(const Tensor& x_, const Tensor& res_, const Tensor& gamma_, double eps, bool pure, bool want_q,
                              bool want_y) {
  const Tensor x = need(x_, at::kBFloat16, "x"), res = need(res_, at::kBFloat16, "res"), gamma = need(gamma_, at::kBFloat16, "gamma");
  const int64_t d = x.size(-1);
  if (res.sizes() != x.sizes()) throw py::value_error("x and res shapes differ");
  need_gamma(gamma, d);
  if (d % kTile || d > kAddNormMaxCols)
    throw py::value_error(cat("K=", d, " must be a multiple of ", kTile, " and at most ", kAddNormMaxCols));
  if (!want_q && !want_y) throw py::value_error("nothing to compute: neither the quantised nor the bf16 output is wanted");
  const c10::cuda::CUDAGuard guard(x.device());
  AddNorm o;
  o.sum = empty_as(x);
  if (want_q) {
    o.q = empty(x.sizes(), kF8, x);
    o.s = empty(with_last(x, d / kTile), at::kFloat, x);
  }
  if (want_y) o.y = empty_as(x);
  check(api.tg_add_rmsnorm_quant_fwd(ptr(x), ptr(res), ptr(gamma), float(eps), ptr(o.sum), ptr(o.q), fptr(o.s), ptr(o.y), nullptr,
                                     x.numel() / d, d, pure ? TG_NORM_PURE : TG_NORM_FUSED, cur_stream()),
        "tg_add_rmsnorm_quant_fwd");
  return o;
}

Pair rmsnorm_bwd(const Tensor& x_, const Tensor& gamma_, const Tensor& g_, double eps, const std::optional<Tensor>& addend_) {
  const Tensor x = need(x_, at::kBFloat16, "x"), gamma = need(gamma_, at::kBFloat16, "gamma"), g = need(g_, at::kBFloat16, "g");
  if (g.sizes() != x.sizes()) throw py::value_error("g and x shapes differ");
  const int64_t d = x.size(-1), rows = x.numel() / d;
  Tensor addend;
  if (addend_) {
    addend = need(*addend_, at::kBFloat16, "addend");
    if (addend.sizes() != x.sizes()) throw py::value_error("addend and x shapes differ");
    if (d > kAddNormMaxCols) throw py::value_error(cat("the fused add takes rows of at most ", kAddNormMaxCols));
  }
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor dx = empty_as(x), dgamma = empty({d}, at::kBFloat16, x);
  const int64_t bytes = std::max<int64_t>(api.tg_rmsnorm_bwd_scratch_bytes(rows, d), 16);
  Tensor scratch = empty({bytes}, at::kByte, x);
  if (addend.defined())
    check(api.tg_rmsnorm_bwd_add(ptr(x), ptr(gamma), ptr(g), ptr(addend), float(eps), ptr(dx), ptr(dgamma), ptr(scratch), rows, d,
                                 cur_stream()),
          "tg_rmsnorm_bwd_add");
  else
    check(api.tg_rmsnorm_bwd(ptr(x), ptr(gamma), ptr(g), float(eps), ptr(dx), ptr(dgamma), ptr(scratch), rows, d, cur_stream()),
          "tg_rmsnorm_bwd");
  return {dx, dgamma};
}

// ---- loss ---------------------------------------------------------------------------------------------------------

std::tuple<Tensor, Tensor, Tensor> softcap_ce_fwd(const Tensor& logits_, const Tensor& targets, double cap, bool want_tanh) {
  Tensor logits = need(logits_, at::kBFloat16, "logits");
  if (logits.dim() != 2) throw py::value_error("logits must be 2-D (rows, vocab)");
  if (targets.scalar_type() != at::kInt || !targets.is_cuda() || !targets.is_contiguous())
    throw py::type_error("targets must be a contiguous int32 CUDA tensor");
  const int64_t rows = logits.size(0), vocab = logits.size(1), pitch = cdiv(vocab, 8) * 8;
  if (targets.numel() != rows) throw py::value_error("one target per row");
  const c10::cuda::CUDAGuard guard(logits.device());
  if (pitch != vocab) {
    // a vocabulary that is not a multiple of 8 (train-gpt's default 50257, config.py:8): the kernels want a
    // 16-byte row pitch, so the rows move to a padded buffer; the pad columns are never used
    Tensor padded = empty({rows, pitch}, at::kBFloat16, logits);
    padded.narrow(1, 0, vocab).copy_(logits);
    logits = padded;
  }
  Tensor nll = empty({rows}, at::kFloat, logits), lse = empty({rows}, at::kFloat, logits), th;
  if (want_tanh) th = empty({rows, pitch}, at::kBFloat16, logits);
  check(api.tg_softcap_ce_fwd(ptr(logits), static_cast<const int32_t*>(ptr(targets)), float(cap), ptr(th), fptr(lse), fptr(nll), rows,
                              vocab, pitch, pitch, cur_stream()),
        "tg_softcap_ce_fwd");
  if (th.defined() && pitch != vocab) th = th.narrow(1, 0, vocab);     // a view: the row pitch stays `pitch`
  return {nll, lse, th};
}

Tensor softcap_ce_bwd(const Tensor& th, const Tensor& targets, const Tensor& lse, const std::optional<Tensor>& gscale_, double cap,
                      bool in_place) {
  if (!th.is_cuda() || th.scalar_type() != at::kBFloat16 || th.dim() != 2 || th.stride(1) != 1)
    throw py::type_error("tanh must be a 2-D bf16 CUDA tensor with unit inner stride (as softcap_ce_fwd returns it)");
  const c10::cuda::CUDAGuard guard(th.device());
  const int64_t rows = th.size(0), vocab = th.size(1), pitch = th.stride(0);
  Tensor d = th;
  int64_t d_pitch = pitch;
  if (!in_place) {
    d_pitch = cdiv(vocab, 8) * 8;
    d = empty({rows, d_pitch}, at::kBFloat16, th).narrow(1, 0, vocab);
  }
  Tensor gscale;
  if (gscale_) gscale = need(gscale_->reshape({1}), at::kFloat, "gscale");
  check(api.tg_softcap_ce_bwd(ptr(th), static_cast<const int32_t*>(ptr(targets)), fptr(lse), fptr(gscale), float(cap), ptr(d), rows,
                              vocab, pitch, d_pitch, cur_stream()),
        "tg_softcap_ce_bwd");
  return d;
}

// ---- optimiser ----------------------------------------------------------------------------------------------------

Tensor sumsq(const Tensor& x_, const std::optional<Tensor>& out_, const std::optional<Tensor>& scratch_) {
  const Tensor x = need(x_, at::kBFloat16, "x");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor out = out_ ? *out_ : empty({1}, at::kFloat, x);
  Tensor scratch = scratch_ ? *scratch_ : empty({api.tg_sumsq_scratch_bytes()}, at::kByte, x);
  check(api.tg_sumsq_bf16(ptr(x), x.numel(), fptr(out), ptr(scratch), cur_stream()), "tg_sumsq_bf16");
  return out;
}

void adamw_step(const Tensor& p, const Tensor& g, const Tensor& m, const Tensor& v, const Tensor& step, double lr, double b1, double b2,
                double eps, double weight_decay, const std::optional<Tensor>& gscale) {
  const std::pair<const Tensor*, const char*> all[] = {{&p, "p"}, {&g, "g"}, {&m, "m"}, {&v, "v"}};
  for (const auto& [t, n] : all)
    if (!t->is_cuda() || t->scalar_type() != at::kBFloat16 || !t->is_contiguous())
      throw py::type_error(cat(n, " must be a contiguous bf16 CUDA tensor"));
  if (p.numel() != g.numel() || p.numel() != m.numel() || p.numel() != v.numel()) throw py::value_error("p, g, m, v sizes differ");
  if (step.scalar_type() != at::kInt || !step.is_cuda()) throw py::type_error("step must be an int32 CUDA scalar");
  const c10::cuda::CUDAGuard guard(p.device());
  check(api.tg_adamw_bf16(ptr(p), ptr(g), ptr(m), ptr(v), p.numel(), float(lr), float(b1), float(b2), float(eps), float(weight_decay),
                          static_cast<const int32_t*>(ptr(step)), gscale ? fptr(*gscale) : nullptr, cur_stream()),
        "tg_adamw_bf16");
}

void need_flat_bf16(const Tensor& t, const char* n) {
  if (!t.is_cuda() || t.scalar_type() != at::kBFloat16 || !t.is_contiguous())
    throw py::type_error(cat(n, " must be a contiguous bf16 CUDA tensor"));
}

// sqrt of the sum of squares over all of `grads`; scratch from global_norm_scratch
Tensor global_norm(const std::vector<Tensor>& grads, const Tensor& scratch) {
  if (grads.empty()) throw py::value_error("no gradients");
  std::vector<tgh_span> spans(grads.size());
  for (size_t i = 0; i < grads.size(); ++i) {
    need_flat_bf16(grads[i], "g");
    spans[i] = {nullptr, grads[i].data_ptr(), nullptr, nullptr, grads[i].numel()};
  }
  const c10::cuda::CUDAGuard guard(grads[0].device());
  Tensor norm = empty({}, at::kFloat, grads[0]);
  check(api.tgh_global_norm(spans.data(), int(spans.size()), ptr(scratch), fptr(norm), nullptr, nullptr, nullptr, cur_stream()),
        "tgh_global_norm");
  return norm;
}
Tensor global_norm_scratch(const Tensor& like, int n) {
  return at::zeros({api.tgh_global_norm_scratch_bytes(n)}, at::TensorOptions().dtype(at::kByte).device(like.device()));
}

// clip by `norm` and AdamW on all tensors; step: int32 (2,), the step count and a zero
void clipped_adamw(const std::vector<Tensor>& p, const std::vector<Tensor>& g, const std::vector<Tensor>& m, const std::vector<Tensor>& v,
                   const Tensor& step, const Tensor& norm, double clip, double lr, double b1, double b2, double eps, double weight_decay) {
  if (p.empty()) return;
  if (p.size() != g.size() || p.size() != m.size() || p.size() != v.size()) throw py::value_error("p, g, m, v differ in number");
  std::vector<tgh_span> spans(p.size());
  for (size_t i = 0; i < p.size(); ++i) {
    need_flat_bf16(p[i], "p"); need_flat_bf16(g[i], "g"); need_flat_bf16(m[i], "m"); need_flat_bf16(v[i], "v");
    if (p[i].numel() != g[i].numel() || p[i].numel() != m[i].numel() || p[i].numel() != v[i].numel())
      throw py::value_error("p, g, m, v sizes differ");
    spans[i] = {p[i].data_ptr(), g[i].data_ptr(), m[i].data_ptr(), v[i].data_ptr(), p[i].numel()};
  }
  const c10::cuda::CUDAGuard guard(p[0].device());
  const Tensor n = to(norm, at::kFloat);
  check(api.tgh_adamw(spans.data(), int(spans.size()), float(lr), float(b1), float(b2), float(eps), float(weight_decay), fptr(n),
                      float(clip), static_cast<int32_t*>(ptr(step)), cur_stream()),
        "tgh_adamw");
}

// ---- GEMM ---------------------------------------------------------------------------------------------------------

Tensor gemm(const Tensor& a, const Tensor& b, const Tensor& sa, const Tensor& sb, int64_t m, int64_t n, int64_t k, int a_major,
            int b_major, Strides sa_st, Strides sb_st, int sb_gran_n, at::ScalarType out_dtype, const Tensor& status_, Tensor out,
            bool split) {
  const std::pair<const Tensor*, const char*> operands[] = {{&a, "a"}, {&b, "b"}};
  for (const auto& [t, name] : operands)
    if (t->scalar_type() != kF8 || t->dim() != 2 || t->stride(1) != 1)
      throw py::type_error(cat(name, " must be a 2-D e4m3 tensor with unit inner stride"));
  const c10::cuda::CUDAGuard guard(a.device());
  if (!out.defined()) out = empty({m, n}, out_dtype, a);
  const Tensor status = status_.defined() ? status_ : status_word(a.get_device());   // an expired wait must leave a trace
  tg_gemm_args args = {};
  args.a = ptr(a); args.b = ptr(b); args.lda = a.stride(0); args.ldb = b.stride(0);
  args.a_major = a_major; args.b_major = b_major;
  args.sa = fptr(sa); args.sa_stride_m = sa_st.row; args.sa_stride_kb = sa_st.kb;
  args.sb = fptr(sb); args.sb_stride_n = sb_st.row; args.sb_stride_kb = sb_st.kb; args.sb_gran_n = sb_gran_n;
  args.d = ptr(out); args.ldd = out.stride(0);
  args.out_dtype = out.scalar_type() == at::kFloat ? TG_OUT_F32 : TG_OUT_BF16;
  args.M = m; args.N = n; args.K = k;
  args.status = static_cast<unsigned*>(ptr(status));
  Tensor ws;
  if (split) {
    const int64_t bytes = api.tg_gemm_workspace_bytes(&args);
    if (bytes > 0) {
      ws = empty({bytes}, at::kByte, a);
      args.workspace = ptr(ws);
      args.workspace_bytes = bytes;
    }
  }
  check(api.tg_gemm_fp8_blockscaled(&args, cur_stream()), "tg_gemm_fp8_blockscaled");
  last_gemm_launches.store(ws.defined() ? 2 : 1, std::memory_order_relaxed);
  return out;
}

// y = x W: x (M, K) in 1x128 tiles, W (K, N) in 128x1 or 128x128 tiles
Tensor gemm_fwd(const Tensor& x_q, const Tensor& x_s, const Tensor& w_q, const Tensor& w_s, bool w_cols, at::ScalarType out_dtype,
                const Tensor& status) {
  const int64_t n = w_q.size(1);
  return gemm(x_q, w_q, x_s, w_s, x_q.size(0), n, x_q.size(1), TG_MAJOR_K, TG_MAJOR_MN, {x_s.size(1), 1},
              {1, w_cols ? n : w_s.size(1)}, w_cols ? 1 : int(kTile), out_dtype, status, Tensor(), true);
}

// dx = g W^T (contracts N): g (M, N) in 1x128 tiles, W (K, N) in 1x128 tiles along N or in 128x128 tiles
Tensor gemm_dgrad(const Tensor& g_q, const Tensor& g_s, const Tensor& w_q, const Tensor& w_s, bool w_cols, at::ScalarType out_dtype,
                  const Tensor& status) {
  return gemm(g_q, w_q, g_s, w_s, g_q.size(0), w_q.size(0), g_q.size(1), TG_MAJOR_K, TG_MAJOR_K, {g_s.size(1), 1}, {w_s.size(1), 1},
              w_cols ? 1 : int(kTile), out_dtype, status, Tensor(), true);
}

// dW = x^T g (contracts the tokens): x (T, K) in 128x1 tiles, g (T, N) in 128x1 or 128x128 tiles
Tensor gemm_wgrad(const Tensor& x_q, const Tensor& x_s, const Tensor& g_q, const Tensor& g_s, bool g_cols, at::ScalarType out_dtype,
                  const Tensor& status, const Tensor& out) {
  const int64_t k = x_q.size(1), n = g_q.size(1);
  if (out.defined() && (out.sizes() != at::IntArrayRef({k, n}) || out.stride(1) != 1 || !out.is_cuda() ||
                        (out.scalar_type() != at::kBFloat16 && out.scalar_type() != at::kFloat)))
    throw py::value_error(cat("out must be a (", k, ", ", n, ") bf16 or float32 CUDA tensor with unit inner stride"));
  return gemm(x_q, g_q, x_s, g_s, k, n, x_q.size(0), TG_MAJOR_MN, TG_MAJOR_MN, {1, k}, {1, g_cols ? n : g_s.size(1)},
              g_cols ? 1 : int(kTile), out_dtype, status, out, true);
}

// ---- the block-scaled linear: forward, backward, autograd -----------------------------------------------------------

// bf16 view of an operand; a wider tensor is taken only if narrowing it is exact (see fp8._as_bf16)
Tensor as_bf16(const Tensor& t, const char* name) {
  if (t.scalar_type() == at::kBFloat16) return t;
  if (!t.is_floating_point()) throw py::type_error(cat(name, " must be a floating-point tensor, got ", dtype_name(t.scalar_type())));
  Tensor n = t.to(at::kBFloat16);
  if (!n.to(t.scalar_type()).eq(t).all().item<bool>())
    throw py::type_error(cat(name, " is ", dtype_name(t.scalar_type()),
                             " with values bf16 cannot hold: the sm_100a kernels quantise bf16 operands "
                             "(as the reference's model does); cast explicitly if that rounding is intended"));
  return n;
}

enum Mode { kSte = 0, kFp8 = 1, kFp8BlockGrad = 2 };

struct Linear {
  int64_t k, n;
};

Linear validate(const Tensor& a, const Tensor& b, int64_t block_k) {
  const int64_t k = a.size(-1);
  if (b.dim() != 2) throw py::value_error(cat("b must be 2-D, got ", b.dim(), " dimensions"));
  if (k != b.size(0)) throw py::value_error(cat("contracted-dim mismatch: a K=", k, ", b K=", b.size(0)));       // fp8.py:53-54
  if (k % block_k) throw py::value_error(cat("K=", k, " not divisible by block_k=", block_k));                   // fp8.py:55-56
  if (block_k != kTile)
    throw py::value_error(cat("block_k=", block_k, " is not supported by the sm_100a kernels (only ", kTile, ")"));
  return {k, b.size(1)};
}

int64_t rows_of(const Tensor& a) {
  int64_t m = 1;
  for (int64_t i = 0; i + 1 < a.dim(); ++i) m *= a.size(i);
  return m;
}

// the 1x128 form of an activation as its caller has it
Pair row_form(const Tensor& q, const Tensor& s, int64_t k) {
  if (!q.defined()) return {};
  if (q.scalar_type() != kF8 || s.scalar_type() != at::kFloat)
    throw py::type_error(cat("a_quantized must be an e4m3 and a float32 tensor, got ", dtype_name(q.scalar_type()), " and ", dtype_name(s.scalar_type())));
  return {q.reshape({-1, k}).contiguous(), s.reshape({-1, k / kTile}).contiguous()};
}

struct ForwardOut {
  Tensor y;                 // (..., N)
  Tensor kept;              // memory of the two below
  Form w;                   // the weight in 128x128 tiles: dgrad reads it too
  Form x_col;               // the activation's column form, which the weight gradient contracts
};

// fp8.py:50-78.  row_q / row_s: the activation's row form made earlier.  keep_x / keep_w: what the backward pass will want
// of the activation (its column form, from the same read) and of the weight outlives the call.  weight: receives the quantised weight.
ForwardOut fp8_forward(const Tensor& a, const Tensor& b_, bool w_cols, const Tensor& row_q, const Tensor& row_s, bool keep_x, bool keep_w,
                       Pair* weight = nullptr) {
  ForwardOut o;
  const int64_t k = a.size(-1), n = b_.size(1), m = rows_of(a);
  Tensor x;
  if (!row_q.defined()) {
    x = as_rows(as_bf16(a, "a"), m, k);
    if (!x.is_cuda()) need(x, at::kBFloat16, "x");
    x = readable(x, false);
  }
  Tensor b = as_bf16(b_, "b");
  if (!b.is_cuda()) need(b, at::kBFloat16, "x");
  if (!w_cols && n % kTile) throw py::value_error(cat("C=", n, " not divisible by ", kTile));
  b = readable(b, w_cols);
  const c10::cuda::CUDAGuard guard(b.device());
  // the TMA row pitch of the (K, N) weight must be a multiple of 16 bytes: its quantised form is widened with zero
  // columns and the result's extra columns are dropped
  const int64_t np = w_cols ? cdiv(n, 16) * 16 : n;
  o.y = empty(with_last(a, np), at::kBFloat16, b);
  tg_gemm_args g = gemm_args(m, np, k, k, TG_MAJOR_K, {k / kTile, 1}, np, TG_MAJOR_MN, {1, w_cols ? np : n / kTile}, w_cols, np, false,
                             status_of(b));
  const int64_t ws_bytes = api.tg_gemm_workspace_bytes(&g);
  Arena kept, temp;
  FormAt x_row_at, x_col_at, w_at;
  if (x.defined()) {
    x_row_at = add_row(temp, m, k);
    if (keep_x) x_col_at = add_col(kept, m, k);
  }
  if (weight == nullptr) w_at = w_cols ? add_col(temp, k, np) : add_block(keep_w ? kept : temp, k, n);
  const size_t ws_at = temp.add(ws_bytes);
  kept.make(b);
  temp.make(b);
  tgh_quantize_job jobs[2];
  int n_jobs = 0;
  Form x_row = {ptr(row_q), fptr(row_s)};
  if (x.defined()) {
    tgh_quantize_job& j = jobs[n_jobs++] = job_of(x);
    want_row(j, x_row = x_row_at.in(temp));
    if (keep_x) want_col(j, o.x_col = x_col_at.in(kept), k);
  }
  tgh_quantize_job& j = jobs[n_jobs++] = job_of(b);
  Form w;
  if (weight != nullptr) {
    *weight = {empty({k, np}, kF8, b), empty({k / kTile, w_cols ? np : n / kTile}, at::kFloat, b)};
    w = {ptr(weight->first), fptr(weight->second)};
  } else {
    w = w_at.in(!w_cols && keep_w ? kept : temp);
  }
  if (w_cols) want_col(j, w, np);
  else want_block(j, w);
  check(api.tgh_quantize_jobs(jobs, n_jobs, cur_stream()), "tgh_quantize_jobs");
  run_gemm(g, x_row, w, ptr(o.y), temp.at(ws_at), ws_bytes);
  if (np != n) {
    o.y = o.y.narrow(-1, 0, n);
    if (o.y.dim() != 2) o.y = o.y.contiguous();
  }
  o.kept = kept.memory();
  if (!w_cols && keep_w) o.w = w;
  return o;
}

struct BackwardIn {
  bool w_cols;
  Mode mode;
  Form w;                                            // the forward's 128x128 weight tiles, reused by dgrad
  Form x_col;                                        // the activation's column form
  std::function<Tensor()> slot_take;                 // where the weight gradient goes instead of a new tensor ...
  std::function<void()> slot_ready;                  // ... and whom to tell that it is there
  bool want_a = true, want_b = true;
};

// fp8.py:85-98 (mode kSte), or the same two GEMMs in block-scaled e4m3
Pair fp8_backward(const Tensor& a, const Tensor& b, const Tensor& g_, at::IntArrayRef a_shape, at::ScalarType a_dtype,
                  at::ScalarType b_dtype, int64_t k, int64_t n, const BackwardIn& in) {
  Tensor da, db;
  if (in.mode == kSte) {
    // (the engine's thread may not have touched the device yet, and cuBLAS wants a context when it makes its handle)
    const c10::cuda::CUDAGuard guard(g_.device());
    cudaFree(nullptr);
    const Tensor g2 = to(g_.dim() == 2 ? g_ : g_.reshape({-1, n}), at::kBFloat16);
    if (in.want_a) da = at::mm(g2, to(b, at::kBFloat16).t());                                 // fp8.py:96 (cuBLAS bf16)
    if (in.want_b) db = at::mm(to(a.dim() == 2 ? a : a.reshape({-1, k}), at::kBFloat16).t(), g2);                // fp8.py:97
    if (da.defined()) da = to(a_shape.size() == 2 ? da : da.reshape(a_shape), a_dtype);
    if (db.defined()) db = to(db, b_dtype);
    return {da, db};
  }
  TORCH_CHECK_VALUE(n % kTile == 0, "N=", n, " not divisible by block_k=", kTile, " (needed by the FP8 dgrad)");
  if (!in.want_a && !in.want_b) return {da, db};
  int64_t m = 1;
  for (size_t i = 0; i + 1 < a_shape.size(); ++i) m *= a_shape[i];
  const Tensor g = readable(to(as_rows(g_, m, n), at::kBFloat16), false);
  const c10::cuda::CUDAGuard guard(g.device());
  const bool g_cols = in.mode == kFp8;               // the weight gradient's upstream operand: columns, or 128x128 tiles
  unsigned* status = status_of(g);
  tg_gemm_args dgrad, wgrad;
  Tensor db_slot;
  int64_t ws_bytes[2] = {0, 0};
  if (in.want_a) {
    da = empty(a_shape, at::kBFloat16, g);
    dgrad = gemm_args(m, k, n, n, TG_MAJOR_K, {n / kTile, 1}, n, TG_MAJOR_K, {n / kTile, 1}, in.w_cols, k, false, status);
    ws_bytes[0] = api.tg_gemm_workspace_bytes(&dgrad);
  }
  if (in.want_b) {
    if (in.slot_take) db_slot = in.slot_take();
    else db = empty({k, n}, at::kBFloat16, g);
    const Tensor& out = in.slot_take ? db_slot : db;
    if (out.sizes() != at::IntArrayRef({k, n}) || out.stride(1) != 1 || !out.is_cuda() ||
        (out.scalar_type() != at::kBFloat16 && out.scalar_type() != at::kFloat))
      throw py::value_error(cat("out must be a (", k, ", ", n, ") bf16 or float32 CUDA tensor with unit inner stride"));
    wgrad = gemm_args(k, n, m, k, TG_MAJOR_MN, {1, k}, n, TG_MAJOR_MN, {1, g_cols ? n : n / kTile}, g_cols, pitch(out),
                      out.scalar_type() == at::kFloat, status);
    ws_bytes[1] = api.tg_gemm_workspace_bytes(&wgrad);
  }
  // everything that is still to be quantised, in one launch: g once for both contractions, the weight along N, the activation
  Arena temp;
  FormAt g_row_at, g_col_at, w_at, x_at;
  const bool make_w = in.want_a && (in.w_cols || !in.w), make_x = in.want_b && !in.x_col;
  if (in.want_a) g_row_at = add_row(temp, m, n);
  if (in.want_b) g_col_at = g_cols ? add_col(temp, m, n) : add_block(temp, m, n);
  if (make_w) w_at = in.w_cols ? add_row(temp, k, n) : add_block(temp, k, n);
  if (make_x) x_at = add_col(temp, m, k);
  const size_t ws_at = temp.add(std::max(ws_bytes[0], ws_bytes[1]));
  temp.make(g);
  tgh_quantize_job jobs[3];
  int n_jobs = 0;
  Form g_row, g_col, w = in.w, x = in.x_col;
  {
    tgh_quantize_job& j = jobs[n_jobs++] = job_of(g);
    if (in.want_a) want_row(j, g_row = g_row_at.in(temp));
    if (in.want_b) {
      g_col = g_col_at.in(temp);
      if (g_cols) want_col(j, g_col, n);
      else want_block(j, g_col);
    }
  }
  Tensor b2, a2;
  if (make_w) {
    b2 = readable(to(b, at::kBFloat16), false);
    tgh_quantize_job& j = jobs[n_jobs++] = job_of(b2);
    w = w_at.in(temp);
    if (in.w_cols) want_row(j, w);
    else want_block(j, w);
  }
  if (make_x) {
    a2 = readable(to(as_rows(a, m, k), at::kBFloat16), false);
    tgh_quantize_job& j = jobs[n_jobs++] = job_of(a2);
    want_col(j, x = x_at.in(temp), k);
  }
  check(api.tgh_quantize_jobs(jobs, n_jobs, cur_stream()), "tgh_quantize_jobs");
  if (in.want_a) set_operands(dgrad, g_row, w, ptr(da), temp.at(ws_at), ws_bytes[0]);
  if (in.want_b) set_operands(wgrad, x, g_col, ptr(db.defined() ? db : db_slot), temp.at(ws_at), ws_bytes[1]);
  if (in.want_a && in.want_b) check(api.tgh_gemm_two(&dgrad, &wgrad, cur_stream()), "tgh_gemm_two");
  else check(api.tg_gemm_fp8_blockscaled(in.want_a ? &dgrad : &wgrad, cur_stream()), "tg_gemm_fp8_blockscaled");
  last_gemm_launches.store(ws_bytes[in.want_b ? 1 : 0] > 0 ? 2 : 1, std::memory_order_relaxed);
  if (in.want_a) da = to(da, a_dtype);
  if (in.want_b) {
    if (in.slot_take) in.slot_ready();
    else db = to(db, b_dtype);
  }
  return {da, db};
}

// A Python object owned by an autograd node, which may die on a thread that does not hold the interpreter lock.
class PyHandle {
 public:
  explicit PyHandle(py::object o) : o_(std::move(o)) {}
  PyHandle(const PyHandle&) = delete;
  PyHandle& operator=(const PyHandle&) = delete;
  ~PyHandle() {
    if (!Py_IsInitialized()) {
      o_.release();
      return;
    }
    py::gil_scoped_acquire gil;
    o_ = py::object();
  }
  const py::object& get() const { return o_; }

 private:
  py::object o_;
};

std::shared_ptr<PyHandle> hold(const py::object& o) { return o.is_none() ? nullptr : std::make_shared<PyHandle>(o); }

[[noreturn]] void backward_twice() {
  throw std::runtime_error(
      "Trying to backward through the graph a second time (or directly access saved tensors after they have already been freed). "
      "Saved intermediate values of the graph are freed when you call .backward() or autograd.grad(). Specify retain_graph=True if "
      "you need to backward through the graph a second time or if you need to access saved tensors after calling backward.");
}

// The custom VJP of fp8.py:30,101.
struct BlockScaledMatmulBackward : public Node {
  SavedVariable a, b;                        // the unquantised residuals (fp8.py:81-82) that the mode needs
  bool has_a = false, has_b = false, released = false;
  Tensor kept;                               // memory of `w` and `x_col`
  Form w, x_col;
  std::shared_ptr<PyHandle> activation, slot;
  std::vector<int64_t> a_shape;
  at::ScalarType a_dtype, b_dtype;
  int64_t k, n;
  bool w_cols;
  Mode mode;

  std::string name() const override { return "BlockScaledMatmulBackward"; }

  void release_variables() override {
    a.reset_data();
    b.reset_data();
    kept = Tensor();
    activation.reset();
    slot.reset();
    released = true;
  }

  variable_list apply(variable_list&& grads) override {
    variable_list out(2);
    if (!grads[0].defined()) return out;
    if (released) backward_twice();
    std::optional<at::AutoDispatchBelowADInplaceOrView> below;      // (under create_graph the straight-through GEMMs are recorded)
    if (!at::GradMode::is_enabled()) below.emplace();
    BackwardIn in;
    in.w_cols = w_cols;
    in.mode = mode;
    in.want_a = task_should_compute_output(0);
    in.want_b = task_should_compute_output(1);
    in.w = w;
    in.x_col = x_col;
    Pair shared;                             // the activation's own column form, made on first use and kept by it
    if (activation && !x_col && in.want_b && mode != kSte) {
      py::gil_scoped_acquire gil;
      shared = activation->get().attr("colwise")().cast<Pair>();
      in.x_col = {ptr(shared.first), fptr(shared.second)};
    }
    if (slot) {
      in.slot_take = [this] {
        py::gil_scoped_acquire gil;
        return slot->get().attr("take")().cast<Tensor>();
      };
      in.slot_ready = [this] {
        py::gil_scoped_acquire gil;
        slot->get().attr("ready")();
      };
    }
    const Tensor av = has_a ? a.unpack() : Tensor(), bv = has_b ? b.unpack() : Tensor();
    std::tie(out[0], out[1]) = fp8_backward(av, bv, grads[0], a_shape, a_dtype, b_dtype, k, n, in);
    return out;
  }
};

Tensor block_scaled_matmul(const Tensor& a, const Tensor& b, int64_t block_k, bool w_cols, int mode_, const py::object& activation,
                           const Tensor& row_q, const Tensor& row_s, const py::object& slot) {
  const Linear d = validate(a, b, block_k);
  const Mode mode = Mode(mode_);
  const bool track = at::GradMode::is_enabled() && (a.requires_grad() || b.requires_grad());
  const auto [rq, rs] = row_form(row_q, row_s, d.k);
  const bool keep = track && mode != kSte, keep_x = keep && b.requires_grad() && activation.is_none() && !rq.defined();
  ForwardOut f;
  {
    at::AutoDispatchBelowADInplaceOrView below;     // none of what happens here is recorded: the node below is the derivative
    f = fp8_forward(a, b, w_cols, rq, rs, keep_x, keep);
  }
  if (!track) return f.y;
  std::shared_ptr<BlockScaledMatmulBackward> node(new BlockScaledMatmulBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(a, b));
  node->k = d.k;
  node->n = d.n;
  node->a_shape.assign(a.sizes().begin(), a.sizes().end());
  node->a_dtype = a.scalar_type();
  node->b_dtype = b.scalar_type();
  node->w_cols = w_cols;
  node->mode = mode;
  node->has_a = mode == kSte || (!f.x_col && activation.is_none());
  node->has_b = mode == kSte || w_cols;
  if (node->has_a) node->a = SavedVariable(a, false);
  if (node->has_b) node->b = SavedVariable(b, false);
  node->kept = f.kept;
  node->w = f.w;
  node->x_col = f.x_col;
  node->activation = hold(activation);
  node->slot = hold(slot);
  torch::autograd::set_history(f.y, node);
  return f.y;
}

// ---- the norm's and the loss's autograd -----------------------------------------------------------------------------

struct RmsNormBackward : public Node {
  SavedVariable x, gamma;                    // kernels.py:101-102
  double eps = 0;
  std::string name() const override { return "RmsNormBackward"; }
  void release_variables() override {
    x.reset_data();
    gamma.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(2);
    if (!grads[0].defined()) return out;
    std::tie(out[0], out[1]) = rmsnorm_bwd(x.unpack(), gamma.unpack(), to(grads[0], at::kBFloat16), eps, std::nullopt);   // kernels.py:104-118
    return out;
  }
};

Tensor rms_norm(const Tensor& x, const Tensor& gamma, double eps, bool pure) {
  const bool track = at::GradMode::is_enabled() && (x.requires_grad() || gamma.requires_grad());
  Tensor y;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    y = rmsnorm_fwd(x, gamma, eps, pure, false).first;
  }
  if (!track) return y;
  std::shared_ptr<RmsNormBackward> node(new RmsNormBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(x, gamma));
  node->x = SavedVariable(x, false);
  node->gamma = SavedVariable(gamma, false);
  node->eps = eps;
  torch::autograd::set_history(y, node);
  return y;
}

// The loss of rows the one-pass kernel takes: forward makes the gradient too, for an upstream gradient of 1 -- what
// `loss.backward()` brings.  Another one is seen on the device (no synchronisation) and the gradient is made again
// from the logits with it, so that it is rounded once all the same.  (Logits that were overwritten in between are no
// error, as they never were for this function: the gradient at hand is then scaled.)
struct CappedCEBackward : public Node {
  Tensor logits, targets, d;
  uint32_t version = 0;
  double cap = 0;
  bool given = false;                        // `d` has been handed out: it is no longer this node's own
  std::string name() const override { return "CappedCEBackward"; }
  void release_variables() override {
    logits = targets = d = Tensor();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined()) return out;
    if (!targets.defined()) backward_twice();
    const Tensor& x = logits;
    if (x._version() != version) {
      out[0] = (d * grads[0].to(at::kFloat)).to(at::kBFloat16);
      return out;
    }
    const int64_t vocab = x.size(-1), rows = x.numel() / vocab;
    const Tensor g = grads[0].to(at::kFloat).contiguous();
    const bool again = given;
    if (again) d = empty_as(d);
    const c10::cuda::CUDAGuard guard(x.device());
    check(api.tgh_softcap_ce(ptr(x), ptr(targets), targets.scalar_type() == at::kLong, float(cap), ptr(d), fptr(g), !again, nullptr,
                             rows, vocab, vocab, cur_stream()),
          "tgh_softcap_ce");
    given = true;
    out[0] = d;
    return out;
  }
};

// ... and of any others: the tanh values go from the forward kernel to the backward one through memory
struct SoftcapCEBackward : public Node {
  Tensor th, targets, lse;
  std::vector<int64_t> shape;
  double cap = 0;
  std::string name() const override { return "SoftcapCEBackward"; }
  void release_variables() override { th = targets = lse = Tensor(); }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined()) return out;
    if (!th.defined()) backward_twice();
    // the tanh buffer is this node's own: the gradient replaces it in place, unless it will be wanted again
    const bool last = !torch::autograd::get_current_graph_task_keep_graph();
    out[0] = softcap_ce_bwd(th, targets, lse, grads[0].to(at::kFloat), cap, last).reshape(shape);
    return out;
  }
};

Tensor capped_cross_entropy(const Tensor& logits_, const Tensor& target_ids, double cap) {
  if (logits_.dim() == 0 || logits_.sizes().slice(0, logits_.dim() - 1) != target_ids.sizes())
    throw py::value_error(cat("logits ", logits_.sizes(), " and target_ids ", target_ids.sizes(), " do not match"));
  const bool track = at::GradMode::is_enabled() && logits_.requires_grad();
  const int64_t vocab = logits_.size(-1), rows = target_ids.numel();
  Tensor logits = need(logits_, at::kBFloat16, "logits"), t = target_ids.contiguous(), loss;
  if (t.scalar_type() != at::kLong) t = t.to(at::kInt);
  const c10::cuda::CUDAGuard guard(logits.device());
  if (rows > 0 && t.is_cuda() && api.tgh_softcap_ce_fits(float(cap), rows, vocab)) {
    Tensor d;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      if (reinterpret_cast<uintptr_t>(ptr(logits)) & 15u) logits = logits.clone();
      if (track) d = empty_as(logits);
      Tensor nll = empty({rows}, at::kFloat, logits);
      check(api.tgh_softcap_ce(ptr(logits), ptr(t), t.scalar_type() == at::kLong, float(cap), ptr(d), nullptr, 0, fptr(nll), rows, vocab,
                               vocab, cur_stream()),
            "tgh_softcap_ce");
      loss = mean_of(nll);
    }
    if (!track) return loss;
    std::shared_ptr<CappedCEBackward> node(new CappedCEBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(logits_));
    node->logits = logits.detach();
    node->version = logits._version();
    node->targets = t;
    node->d = d;
    node->cap = cap;
    torch::autograd::set_history(loss, node);
    return loss;
  }
  Tensor th, lse, nll;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    t = t.reshape({-1}).to(at::kInt);
    std::tie(nll, lse, th) = softcap_ce_fwd(logits.reshape({-1, vocab}), t, cap, true);
    loss = nll.mean();                                                               // losses.py:12
  }
  if (!track) return loss;
  std::shared_ptr<SoftcapCEBackward> node(new SoftcapCEBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(logits_));
  node->th = th;
  node->targets = t;
  node->lse = lse;
  node->cap = cap;
  node->shape.assign(logits_.sizes().begin(), logits_.sizes().end());
  torch::autograd::set_history(loss, node);
  return loss;
}

// ---- bindings -------------------------------------------------------------------------------------------------------

Tensor or_none(const std::optional<Tensor>& t) { return t ? *t : Tensor(); }

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("bind", &bind);
  m.def("quantize_rowwise", &quantize_rowwise);
  m.def("quantize_colwise", &quantize_colwise);
  m.def("quantize_block128", &quantize_block128);
  m.def("quantize_rowcol", [](const Tensor& x) { return quantize_rowcol(x).tuple(); });
  m.def("quantize_rowcol_into", [](const Tensor& x, const std::optional<Pair>& row_out, const std::optional<Pair>& col_out) {
    return quantize_rowcol_into(x, row_out, col_out).tuple();
  });
  m.def("act_quantize_rowcol", [](const Tensor& x, int act, const std::string& name, const std::optional<Tensor>& gate) {
    return act_quantize_rowcol(x, act, name, gate).tuple();
  });
  m.def("rmsnorm_fwd", [](const Tensor& x, const Tensor& gamma, double eps, bool pure, bool want_rnorm) -> py::object {
    const Pair o = rmsnorm_fwd(x, gamma, eps, pure, want_rnorm);
    return want_rnorm ? py::object(py::make_tuple(o.first, o.second)) : py::cast(o.first);
  });
  m.def("rmsnorm_quant_fwd", [](const Tensor& x, const Tensor& gamma, double eps, bool pure, bool want_y, bool want_rnorm) {
    const NormQuant o = rmsnorm_quant_fwd(x, gamma, eps, pure, want_y, want_rnorm);
    return py::make_tuple(o.q, o.s, o.y, o.rn);
  });
  m.def("add_rmsnorm_quant_fwd",
        [](const Tensor& x, const Tensor& res, const Tensor& gamma, double eps, bool pure, bool want_q, bool want_y) {
          const AddNorm o = add_rmsnorm_quant_fwd(x, res, gamma, eps, pure, want_q, want_y);
          return py::make_tuple(o.sum, o.q, o.s, o.y);
        });
  m.def("rmsnorm_bwd", &rmsnorm_bwd);
  m.def("softcap_ce_fwd", &softcap_ce_fwd);
  m.def("softcap_ce_bwd", &softcap_ce_bwd);
  m.def("sumsq", &sumsq);
  m.def("adamw_step", &adamw_step);
  m.def("global_norm", &global_norm);
  m.def("global_norm_scratch", &global_norm_scratch);
  m.def("clipped_adamw", &clipped_adamw);
  m.def("status_word", &status_word);
  m.def("last_gemm_launches", [] { return last_gemm_launches.load(std::memory_order_relaxed); });
  m.def("gemm", [](const Tensor& a, const Tensor& b, const Tensor& sa, const Tensor& sb, int64_t M, int64_t N, int64_t K, int a_major,
                   int b_major, std::pair<int64_t, int64_t> sa_st, std::pair<int64_t, int64_t> sb_st, int gran, bool out_f32,
                   const std::optional<Tensor>& status, const std::optional<Tensor>& out, bool split) {
    return gemm(a, b, sa, sb, M, N, K, a_major, b_major, {sa_st.first, sa_st.second}, {sb_st.first, sb_st.second}, gran,
                out_f32 ? at::kFloat : at::kBFloat16, or_none(status), or_none(out), split);
  });
  m.def("gemm_fwd", [](const Tensor& xq, const Tensor& xs, const Tensor& wq, const Tensor& ws, bool w_cols, bool f32,
                       const std::optional<Tensor>& status) {
    return gemm_fwd(xq, xs, wq, ws, w_cols, f32 ? at::kFloat : at::kBFloat16, or_none(status));
  });
  m.def("gemm_dgrad", [](const Tensor& gq, const Tensor& gs, const Tensor& wq, const Tensor& ws, bool w_cols, bool f32,
                         const std::optional<Tensor>& status) {
    return gemm_dgrad(gq, gs, wq, ws, w_cols, f32 ? at::kFloat : at::kBFloat16, or_none(status));
  });
  m.def("gemm_wgrad", [](const Tensor& xq, const Tensor& xs, const Tensor& gq, const Tensor& gs, bool g_cols, bool f32,
                         const std::optional<Tensor>& status, const std::optional<Tensor>& out) {
    return gemm_wgrad(xq, xs, gq, gs, g_cols, f32 ? at::kFloat : at::kBFloat16, or_none(status), or_none(out));
  });
  m.def("fp8_forward", [](const Tensor& a, const Tensor& b, int64_t block_k, bool w_cols, const std::optional<Tensor>& row_q,
                          const std::optional<Tensor>& row_s, bool return_weight) -> py::object {
    const Linear d = validate(a, b, block_k);
    const auto [rq, rs] = row_form(or_none(row_q), or_none(row_s), d.k);
    Pair weight;
    const Tensor y = fp8_forward(a, b, w_cols, rq, rs, false, false, return_weight ? &weight : nullptr).y;
    return return_weight ? py::object(py::make_tuple(y, weight)) : py::cast(y);
  });
  m.def("fp8_backward", [](const Tensor& a, const Tensor& b, const Tensor& g, bool w_cols, int mode, const py::object& activation,
                           const std::optional<Tensor>& w_q, const std::optional<Tensor>& w_s, const py::object& slot) {
    BackwardIn in;
    in.w_cols = w_cols;
    in.mode = Mode(mode);
    in.w = {ptr(or_none(w_q)), fptr(or_none(w_s))};
    Pair shared;
    if (!activation.is_none() && in.mode != kSte) {
      shared = activation.attr("colwise")().cast<Pair>();
      in.x_col = {ptr(shared.first), fptr(shared.second)};
    }
    if (!slot.is_none()) {
      in.slot_take = [&] { return slot.attr("take")().cast<Tensor>(); };
      in.slot_ready = [&] { slot.attr("ready")(); };
    }
    return fp8_backward(a, b, g, a.sizes(), a.scalar_type(), b.scalar_type(), a.size(-1), b.size(1), in);
  });
  m.def("block_scaled_matmul", [](const Tensor& a, const Tensor& b, int64_t block_k, bool w_cols, int mode, const py::object& activation,
                                  const std::optional<Tensor>& row_q, const std::optional<Tensor>& row_s, const py::object& slot) {
    return block_scaled_matmul(a, b, block_k, w_cols, mode, activation, or_none(row_q), or_none(row_s), slot);
  });
  m.def("rms_norm", &rms_norm);
  m.def("capped_cross_entropy", &capped_cross_entropy);
  register_step(m);
}
