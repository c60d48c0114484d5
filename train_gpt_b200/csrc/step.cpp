// The training step of train_gpt_b200.step with the default switches -- FP8 linears with 128x128 weight tiles, fused norms,
// MLP and q/k/v, one-pass loss, flat parameters and gradients -- written out: forward, backward, global norm and AdamW as one
// native program instead of some 150 autograd nodes and tensor operations in Python.
//
// It launches the same kernels on the same operands in the same order as the model does through autograd, so its results
// are bit-identical to that path's (tests/test_gpu_step.py compares the two, and a trajectory recorded with the step launched
// operation by operation).  What it saves is what autograd cannot see:
//   * host time: a launch costs 2-4 us here, 15-25 us through Python -- train-gpt's small model spent 3.4 ms per step on
//     0.45 ms of kernels;
//   * launches: every weight of the model is quantised in one, a backward step's quantisers (upstream gradients and the
//     column form of the activation) in one per linear, norm-weight and unembedding gradients are written where they belong
//     instead of added into zeros, norm, clip factor, step count and update are two launches.
//
// Memory: what a layer keeps for its backward pass is one allocation; operands that live only between a quantiser and its
// GEMM share scratch that every layer reuses (one stream orders them).
#include "host.h"

#include <ATen/ops/_fused_sdp_choice.h>
#include <ATen/ops/_scaled_dot_product_cudnn_attention.h>
#include <ATen/ops/_scaled_dot_product_cudnn_attention_backward.h>
#include <ATen/ops/_scaled_dot_product_flash_attention.h>
#include <ATen/ops/_scaled_dot_product_flash_attention_backward.h>
#include <ATen/ops/scaled_dot_product_attention.h>
#include <torch/csrc/autograd/autograd.h>

#include <algorithm>

namespace {

using namespace tgh;

enum SdpBackend { kMath = 0, kFlash = 1, kCudnn = 3 };     // what at::_fused_sdp_choice answers

// Causal attention and what its backward pass needs.
struct Attention {
  int64_t backend = -1;
  Tensor q, k, v, out, lse, cum_q, cum_k, seed, offset;
  c10::SymInt max_q, max_k;

  static int64_t choose(const Tensor& q, const Tensor& k, const Tensor& v) {
    return at::_fused_sdp_choice(q.detach().set_requires_grad(true), k, v, {}, 0.0, true);
  }
  // q, k, v: (B, H, T, D); choice: what choose() says of them
  void forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, int64_t choice) {
    q = q_; k = k_; v = v_;
    Tensor debug;
    backend = choice;
    if (backend == kCudnn) {
      std::tie(out, lse, cum_q, cum_k, max_q, max_k, seed, offset, debug) =
          at::_scaled_dot_product_cudnn_attention(q, k, v, {}, true, 0.0, true, false, std::nullopt);
    } else if (backend == kFlash && q.size(-1) % 8 == 0) {
      std::tie(out, lse, cum_q, cum_k, max_q, max_k, seed, offset, debug) =
          at::_scaled_dot_product_flash_attention(q, k, v, 0.0, true, false, std::nullopt);
    } else {                                    // another backend: through autograd
      backend = kMath;
      at::AutoGradMode on(true);
      q = q.detach().set_requires_grad(true);
      k = k.detach().set_requires_grad(true);
      v = v.detach().set_requires_grad(true);
      out = at::scaled_dot_product_attention(q, k, v, {}, 0.0, true);
    }
  }
  std::array<Tensor, 3> backward(const Tensor& g) {
    std::array<Tensor, 3> d;
    if (backend == kCudnn) {
      std::tie(d[0], d[1], d[2]) = at::_scaled_dot_product_cudnn_attention_backward_symint(
          g, q, k, v, out, lse, seed, offset, Tensor(), cum_q, cum_k, max_q, max_k, 0.0, true, std::nullopt);
    } else if (backend == kFlash) {
      std::tie(d[0], d[1], d[2]) = at::_scaled_dot_product_flash_attention_backward_symint(
          g, q, k, v, out, lse, cum_q, cum_k, max_q, max_k, 0.0, true, seed, offset, std::nullopt);
    } else {
      const auto r = torch::autograd::grad({out}, {q, k, v}, {g});
      d = {r[0], r[1], r[2]};
    }
    q = k = v = out = lse = cum_q = cum_k = seed = offset = Tensor();
    return d;
  }
};

struct LayerTensors {
  Tensor norm1, wqkv, wo, norm2, w_up, w_down;
};

struct Config {
  int64_t heads, head_dim;
  double eps, cap;
  int act, act_bwd;
};
struct Hyper {
  double lr, b1, b2, eps, weight_decay, clip;
};

class StepProgram {
 public:
  // Parameters and, in the same structure, the slices of the flat gradient tensors; `flat`: per bucket the flat parameters,
  // gradients and moments; params: all parameters, as autograd knows them; count: int32 (2,), see tgh_adamw.  on_bucket(i) / on_attention() / on_end(), or None: a bucket's
  // gradients are complete / an attention backward is about to be launched / the backward pass is over.
  StepProgram(Config c, Tensor embed, Tensor pos, Tensor final_norm, Tensor unembed, std::vector<std::vector<Tensor>> layers,
              Tensor g_embed, Tensor g_pos, Tensor g_final_norm, Tensor g_unembed, std::vector<std::vector<Tensor>> g_layers,
              std::vector<std::vector<Tensor>> flat, std::vector<Tensor> params, Tensor count, py::object on_bucket, py::object on_attention, py::object on_end)
      : c_(c), embed_(embed), pos_(pos), final_norm_(final_norm), unembed_(unembed), g_embed_(g_embed), g_pos_(g_pos),
        g_final_norm_(g_final_norm), g_unembed_(g_unembed), count_(count), params_(std::move(params)), on_bucket_(on_bucket), on_attention_(on_attention),
        on_end_(on_end) {
    auto layer = [](const std::vector<Tensor>& t) { return LayerTensors{t.at(0), t.at(1), t.at(2), t.at(3), t.at(4), t.at(5)}; };
    for (const auto& t : layers) layers_.push_back(layer(t));
    for (const auto& t : g_layers) grads_.push_back(layer(t));
    for (const auto& f : flat) {
      for (const Tensor& t : f) need_flat(t);
      flat_.push_back(f);
    }
    d_ = embed.size(1);
    vocab_ = embed.size(0);
    hd_ = c.heads * c.head_dim;
    ff_ = layers_.empty() ? 0 : layers_[0].w_up.size(1);
    norm_scratch_ = at::zeros({api.tgh_global_norm_scratch_bytes(int(flat_.size()))}, embed.options().dtype(at::kByte));
  }

  // Whether this step may run here: every gradient is computed and none handed to autograd, so only while every parameter wants one and
  // none has a hook that expects to see it.
  bool applies() const {
    for (const Tensor& p : params_)
      if (!p.requires_grad() || !torch::autograd::impl::hooks(p).empty()) return false;
    return true;
  }

  // (loss, global gradient norm); the loss is NaN if a GEMM gave up on a device wait.  The hyper-parameters come with every step: a
  // schedule changes them between steps.
  Pair step(const Tensor& ids_, const Tensor& targets_, const Hyper& h) {
    const at::NoGradGuard no_grad;
    const c10::cuda::CUDAGuard guard(embed_.device());
    Tensor ids = ids_.to(embed_.device(), at::kLong).contiguous(), targets = targets_.contiguous();
    if (ids.dim() != 2 || targets.sizes() != ids.sizes() || !targets.is_cuda())
      throw py::value_error("ids and targets are (batch, tokens) tensors of one shape, targets on the GPU");
    if (targets.scalar_type() != at::kLong) targets = targets.to(at::kInt);
    b_ = ids.size(0);
    t_ = ids.size(1);
    m_ = b_ * t_;
    if (t_ > pos_.size(0)) throw py::value_error(cat("sequence of ", t_, " tokens, positions for ", pos_.size(0)));
    status_ = static_cast<unsigned*>(ptr(status_word(embed_.get_device())));
    norms_.clear();
    plan();
    quantize_weights();

    const int64_t n_layers = int64_t(layers_.size());
    // one attention backend for the step, as all its layers have one shape; the library ones need none of autograd's dispatch
    attention_ = -1;
    std::optional<at::AutoDispatchBelowADInplaceOrView> below;
    if (n_layers > 0) {
      const Tensor qkv = act(3 * hd_);
      attention_ = Attention::choose(heads(qkv, 0), heads(qkv, 1), heads(qkv, 2));
      if (attention_ == kCudnn || (attention_ == kFlash && c_.head_dim % 8 == 0)) below.emplace();
    }
    std::vector<Kept> kept(n_layers);
    Tensor x = act(d_), branch;
    check(api.tgh_embed(ids.data_ptr<int64_t>(), ptr(embed_), ptr(pos_), ptr(x), b_, t_, d_, vocab_, status_, token_table_, ptr(g_embed_), cur_stream()),
          "tgh_embed");
    for (int64_t l = 0; l < n_layers; ++l) forward_layer(l, kept[l], x, branch);
    // the head: x + branch, norm, logits, loss and the logits' gradient
    Tensor xs = x, hf = act(d_);
    if (branch.defined()) {
      xs = act(d_);
      check(api.tg_add_rmsnorm_quant_fwd(ptr(x), ptr(branch), ptr(final_norm_), float(c_.eps), ptr(xs), nullptr, nullptr, ptr(hf), nullptr,
                                         m_, d_, TG_NORM_FUSED, cur_stream()),
            "tg_add_rmsnorm_quant_fwd");
    } else {
      check(api.tg_rmsnorm_fwd(ptr(x), ptr(final_norm_), float(c_.eps), ptr(hf), nullptr, m_, d_, TG_NORM_FUSED, cur_stream()),
            "tg_rmsnorm_fwd");
    }
    x = branch = Tensor();
    Tensor logits = at::mm(hf, unembed_);                      // stays bf16 (bench_fp8_norm.py:86)
    Tensor dlogits = empty_as(logits), nll = empty({m_}, at::kFloat, embed_);
    check(api.tgh_softcap_ce(ptr(logits), ptr(targets), targets.scalar_type() == at::kLong, float(c_.cap), ptr(dlogits), nullptr, 0,
                             fptr(nll), m_, vocab_, vocab_, cur_stream()),
          "tgh_softcap_ce");
    const Tensor loss = mean_of(nll);
    logits = Tensor();
    // ---- backward
    at::mm_out(g_unembed_, hf.t(), dlogits);
    Tensor dh = at::mm(dlogits, unembed_.t());
    dlogits = hf = Tensor();
    Tensor d = act(d_);
    norm_bwd(xs, final_norm_, dh, Tensor(), d, g_final_norm_);
    xs = dh = Tensor();
    bucket_done(0);
    for (int64_t l = n_layers - 1; l >= 0; --l) {
      d = backward_layer(l, kept[l], d);
      kept[l] = Kept();
      bucket_done(int(n_layers - l));
    }
    // pos: the sum over the batch; embed: summed by token
    Tensor g_seq = g_pos_.narrow(0, 0, t_);
    at::sum_out(g_seq, d.view({b_, t_, d_}), at::IntArrayRef({0}));
    if (t_ < g_pos_.size(0)) g_pos_.narrow(0, t_, g_pos_.size(0) - t_).zero_();
    check(api.tgh_embed_bwd_cleared(ids.data_ptr<int64_t>(), ptr(d), ptr(g_embed_), token_table_, m_, d_, vocab_, cur_stream()), "tgh_embed_bwd");
    bucket_done(int(n_layers + 1));
    finish_norms();
    if (!on_end_.is_none()) on_end_();
    scratch_ = weights_memory_ = Tensor();
    // ---- optimiser
    std::vector<tgh_span> spans;
    for (const auto& f : flat_) spans.push_back({f[0].data_ptr(), f[1].data_ptr(), f[2].data_ptr(), f[3].data_ptr(), f[0].numel()});
    Tensor norm = empty({}, at::kFloat, embed_), loss_out = empty({}, at::kFloat, embed_);
    check(api.tgh_global_norm(spans.data(), int(spans.size()), ptr(norm_scratch_), fptr(norm), fptr(loss), status_, fptr(loss_out),
                              cur_stream()),
          "tgh_global_norm");
    check(api.tgh_adamw(spans.data(), int(spans.size()), float(h.lr), float(h.b1), float(h.b2), float(h.eps), float(h.weight_decay),
                        fptr(norm), float(h.clip), static_cast<int32_t*>(ptr(count_)), cur_stream()),
          "tgh_adamw");
    return {loss_out, norm};
  }

 private:
  // what a layer's backward pass reads
  struct Kept {
    Tensor memory;
    Tensor x1, h1, x2, h2, u;                    // the norms' inputs and outputs, the pre-activation
    Form o_col, a_col;                           // column forms of the attention output and of the activation
    Attention attention;
  };
  struct Weights {
    Form qkv, o, up, down;
  };

  static void need_flat(const Tensor& t) {
    if (!t.is_cuda() || t.scalar_type() != at::kBFloat16 || !t.is_contiguous()) throw py::type_error("flat tensors must be contiguous bf16 CUDA tensors");
  }
  Tensor act(int64_t cols) const { return empty({m_, cols}, at::kBFloat16, embed_); }

  // GEMMs of this step's size
  tg_gemm_args fwd(int64_t k, int64_t n) const {
    return gemm_args(m_, n, k, k, TG_MAJOR_K, {k / kTile, 1}, n, TG_MAJOR_MN, {1, n / kTile}, false, n, false, status_);
  }
  tg_gemm_args dgrad(int64_t k, int64_t n) const {
    return gemm_args(m_, k, n, n, TG_MAJOR_K, {n / kTile, 1}, n, TG_MAJOR_K, {n / kTile, 1}, false, k, false, status_);
  }
  tg_gemm_args wgrad(int64_t k, int64_t n) const {
    return gemm_args(k, n, m_, k, TG_MAJOR_MN, {1, k}, n, TG_MAJOR_MN, {1, n}, true, n, false, status_);
  }
  void run(tg_gemm_args g, const Form& a, const Form& b, void* d) {
    run_gemm(g, a, b, d, workspace_, api.tg_gemm_workspace_bytes(&g));
  }

  // the data gradient of a (k, n) linear into dx and its weight gradient into dw, from the gradient's two forms in row_ and col_
  void run_backward(int64_t k, int64_t n, const Form& w, void* dx, const Form& x_col, void* dw) {
    tg_gemm_args a = dgrad(k, n), b = wgrad(k, n);
    set_operands(a, row_, w, dx, workspace_, api.tg_gemm_workspace_bytes(&a));
    set_operands(b, x_col, col_, dw, workspace_, api.tg_gemm_workspace_bytes(&b));
    check(api.tgh_gemm_two(&a, &b, cur_stream()), "tgh_gemm_two");
  }

  // Scratch for the widest of every use: a row form, a column form beside it, a third one, the norm backward's partial
  // sums, the GEMMs' workspace.
  void plan() {
    const int64_t wide = std::max({d_, hd_, ff_, 3 * hd_});
    int64_t ws = 0;
    const std::pair<int64_t, int64_t> shapes[] = {{d_, 3 * hd_}, {hd_, d_}, {d_, ff_}, {ff_, d_}};
    for (const auto& [k, n] : shapes)
      for (tg_gemm_args g : {fwd(k, n), dgrad(k, n), wgrad(k, n)}) ws = std::max(ws, api.tg_gemm_workspace_bytes(&g));
    Arena a;
    const FormAt row = add_row(a, m_, wide), col = add_col(a, m_, wide), third = add_col(a, m_, d_);
    norm_bytes_ = (std::max<int64_t>(api.tg_rmsnorm_bwd_scratch_bytes(m_, d_), 16) + 255) / 256 * 256;
    // (where buckets are exchanged each finishes its own: the head's norm, or a layer's two)
    norms_at_once_ = std::min<int64_t>(on_bucket_.is_none() ? kNormsAtOnce : 2, 2 * int64_t(layers_.size()) + 1);
    const size_t norm = a.add(norm_bytes_ * norms_at_once_), gemm = a.add(ws), table = a.add(vocab_ * 8);
    a.make(embed_);
    scratch_ = a.memory();
    row_ = row.in(a);
    col_ = col.in(a);
    third_ = third.in(a);
    norm_partial_ = a.at(norm);
    workspace_ = a.at(gemm);
    token_table_ = a.at(table);
  }

  void quantize_weights() {
    Arena a;
    std::vector<std::array<FormAt, 4>> at(layers_.size());
    for (auto& w : at) w = {add_block(a, d_, 3 * hd_), add_block(a, hd_, d_), add_block(a, d_, ff_), add_block(a, ff_, d_)};
    a.make(embed_);
    weights_memory_ = a.memory();
    weights_.resize(layers_.size());
    std::vector<tgh_quantize_job> jobs;
    for (size_t l = 0; l < layers_.size(); ++l) {
      weights_[l] = {at[l][0].in(a), at[l][1].in(a), at[l][2].in(a), at[l][3].in(a)};
      const std::pair<const Tensor*, const Form*> each[] = {{&layers_[l].wqkv, &weights_[l].qkv}, {&layers_[l].wo, &weights_[l].o},
                                                            {&layers_[l].w_up, &weights_[l].up}, {&layers_[l].w_down, &weights_[l].down}};
      for (const auto& [t, f] : each) {
        jobs.push_back(job_of(*t));
        want_block(jobs.back(), *f);
      }
    }
    check(api.tgh_quantize_jobs(jobs.data(), int(jobs.size()), cur_stream()), "tgh_quantize_jobs");
  }

  // x + branch (branch undefined: x alone), norm and quantise: the sum replaces x
  Tensor norm_fwd(Tensor& x, const Tensor& branch, const Tensor& gamma, Tensor& h) {
    h = act(d_);
    if (!branch.defined()) {
      check(api.tg_rmsnorm_quant_fwd(ptr(x), ptr(gamma), float(c_.eps), row_.q, row_.s, ptr(h), nullptr, m_, d_, TG_NORM_FUSED, cur_stream()),
            "tg_rmsnorm_quant_fwd");
      return x;
    }
    Tensor sum = act(d_);
    check(api.tg_add_rmsnorm_quant_fwd(ptr(x), ptr(branch), ptr(gamma), float(c_.eps), ptr(sum), row_.q, row_.s, ptr(h), nullptr, m_, d_,
                                       TG_NORM_FUSED, cur_stream()),
          "tg_add_rmsnorm_quant_fwd");
    return x = sum;
  }
  void norm_bwd(const Tensor& x, const Tensor& gamma, const Tensor& g, const Tensor& addend, const Tensor& dx, const Tensor& dgamma) {
    if (int64_t(norms_.size()) == norms_at_once_) finish_norms();
    void* partial = static_cast<char*>(norm_partial_) + norms_.size() * norm_bytes_;
    check(api.tgh_rmsnorm_bwd_parts(ptr(x), ptr(gamma), ptr(g), addend.defined() ? ptr(addend) : nullptr, float(c_.eps), ptr(dx), partial, m_, d_,
                                    cur_stream()),
          "tgh_rmsnorm_bwd_parts");
    norms_.push_back({partial, ptr(dgamma)});
  }
  // the weight gradients of the norms whose backward kernels ran since the last call, in one launch
  void finish_norms() {
    if (norms_.empty()) return;
    check(api.tgh_dgamma_reduce(norms_.data(), int(norms_.size()), m_, d_, cur_stream()), "tgh_dgamma_reduce");
    norms_.clear();
  }
  void quantize(const tgh_quantize_job* jobs, int n) { check(api.tgh_quantize_jobs(jobs, n, cur_stream()), "tgh_quantize_jobs"); }
  Tensor heads(const Tensor& qkv, int64_t which) const {        // (B, H, T, D), a view
    return qkv.as_strided({b_, c_.heads, t_, c_.head_dim}, {t_ * 3 * hd_, c_.head_dim, 3 * hd_, 1}, which * hd_);
  }
  // a (B, H, T, D) tensor as (tokens, H D), without a copy where it lies that way
  Tensor tokens(const Tensor& o) const {
    if (o.stride(3) == 1 && o.stride(1) == c_.head_dim && o.stride(2) == hd_ && o.stride(0) == t_ * hd_)
      return o.as_strided({m_, hd_}, {hd_, 1});
    return o.transpose(1, 2).reshape({m_, hd_});
  }

  void forward_layer(int64_t l, Kept& k, Tensor& x, Tensor& branch) {
    const LayerTensors& p = layers_[l];
    const Weights& w = weights_[l];
    k.x1 = norm_fwd(x, branch, p.norm1, k.h1);                                  // model.py:72 of the layer before, :76
    Tensor qkv = act(3 * hd_);
    run(fwd(d_, 3 * hd_), row_, w.qkv, ptr(qkv));                               // model.py:63-65
    k.attention.forward(heads(qkv, 0), heads(qkv, 1), heads(qkv, 2), attention_);
    const Tensor o = readable(tokens(k.attention.out), false);
    Arena keep;
    const FormAt o_col = add_col(keep, m_, hd_), a_col = add_col(keep, m_, ff_);
    keep.make(embed_);
    k.memory = keep.memory();
    k.o_col = o_col.in(keep);
    k.a_col = a_col.in(keep);
    tgh_quantize_job j = job_of(o);
    want_row(j, row_);
    want_col(j, k.o_col, hd_);
    quantize(&j, 1);
    branch = act(d_);
    run(fwd(hd_, d_), row_, w.o, ptr(branch));
    k.x2 = norm_fwd(x, branch, p.norm2, k.h2);                                  // model.py:68, :77
    k.u = act(ff_);
    run(fwd(d_, ff_), row_, w.up, ptr(k.u));
    check(api.tg_act_quantize_rowcol(ptr(k.u), nullptr, c_.act, row_.q, row_.s, k.a_col.q, k.a_col.s, m_, ff_, cur_stream()),
          "tg_act_quantize_rowcol");                                            // model.py:72
    branch = act(d_);
    run(fwd(ff_, d_), row_, w.down, ptr(branch));
  }

  // d: the gradient of the layer's output; returns that of its input
  Tensor backward_layer(int64_t l, Kept& k, Tensor d) {
    const LayerTensors &p = layers_[l], &g = grads_[l];
    const Weights& w = weights_[l];
    Tensor dh = act(d_);
    {                                                                           // the MLP
      tgh_quantize_job j[2] = {job_of(d), job_of(k.h2)};
      want_row(j[0], row_);
      want_col(j[0], col_, d_);
      want_col(j[1], third_, d_);
      quantize(j, 2);
      Tensor da = act(ff_);
      run_backward(ff_, d_, w.down, ptr(da), k.a_col, ptr(g.w_down));
      check(api.tg_act_quantize_rowcol(ptr(k.u), ptr(da), c_.act_bwd, row_.q, row_.s, col_.q, col_.s, m_, ff_, cur_stream()),
            "tg_act_quantize_rowcol");
      run_backward(d_, ff_, w.up, ptr(dh), third_, ptr(g.w_up));
    }
    k.u = k.h2 = Tensor();
    Tensor d2 = act(d_);
    norm_bwd(k.x2, p.norm2, dh, d, d2, g.norm2);
    k.x2 = Tensor();
    Tensor dov = empty({b_, t_, c_.heads, c_.head_dim}, at::kBFloat16, embed_);
    {                                                                           // the attention output's projection
      tgh_quantize_job j = job_of(d2);
      want_row(j, row_);
      want_col(j, col_, d_);
      quantize(&j, 1);
      run_backward(hd_, d_, w.o, ptr(dov), k.o_col, ptr(g.wo));
    }
    if (!on_attention_.is_none()) on_attention_();
    std::array<Tensor, 3> dq = k.attention.backward(dov.transpose(1, 2));
    {                                                                           // q, k, v as one
      tgh_quantize_job j[4];
      Tensor parts[3];
      for (int i = 0; i < 3; ++i) {
        parts[i] = readable(tokens(dq[i]), false);
        j[i] = job_of(parts[i]);
        j[i].q_row = static_cast<uint8_t*>(row_.q) + i * hd_;
        j[i].s_row = row_.s + i * (hd_ / kTile);
        j[i].q_row_ld = 3 * hd_;
        j[i].s_row_ld = 3 * hd_ / kTile;
        j[i].form = TGH_FORM_COLUMNS;
        j[i].q = static_cast<uint8_t*>(col_.q) + i * hd_;
        j[i].s = col_.s + i * hd_;
        j[i].q_ld = j[i].s_ld = 3 * hd_;
      }
      j[3] = job_of(k.h1);
      want_col(j[3], third_, d_);
      quantize(j, 4);
      run_backward(d_, 3 * hd_, w.qkv, ptr(dh), third_, ptr(g.wqkv));
    }
    k.h1 = Tensor();
    if (l > 0) {
      norm_bwd(k.x1, p.norm1, dh, d2, d, g.norm1);
      return d;
    }
    norm_bwd(k.x1, p.norm1, dh, Tensor(), d, g.norm1);       // the first layer's input joins the two paths in bf16
    return d.add_(d2);
  }

  void bucket_done(int i) {
    if (on_bucket_.is_none()) return;
    finish_norms();                            // (a bucket that is exchanged holds a norm's weight gradient)
    on_bucket_(i);
  }

  Config c_;
  Tensor embed_, pos_, final_norm_, unembed_, g_embed_, g_pos_, g_final_norm_, g_unembed_, count_, norm_scratch_;
  std::vector<Tensor> params_;
  std::vector<LayerTensors> layers_, grads_;
  std::vector<std::vector<Tensor>> flat_;
  py::object on_bucket_, on_attention_, on_end_;
  int64_t d_, hd_, ff_, vocab_;
  // of the step under way
  int64_t b_ = 0, t_ = 0, m_ = 0;
  unsigned* status_ = nullptr;
  Tensor scratch_, weights_memory_;
  std::vector<Weights> weights_;
  Form row_, col_, third_;
  void *norm_partial_ = nullptr, *workspace_ = nullptr, *token_table_ = nullptr;
  int64_t attention_ = -1;
  static constexpr int64_t kNormsAtOnce = 16;  // partial sums of so many norms are kept (1.8 MB each at 8192 x 1024)
  int64_t norm_bytes_ = 0, norms_at_once_ = 0;
  std::vector<tgh_dgamma_job> norms_;
};

}  // namespace

void tgh::register_step(py::module_& m) {
  py::class_<StepProgram>(m, "StepProgram")
      .def(py::init([](std::tuple<int64_t, int64_t, double, double, int, int> c, Tensor embed, Tensor pos, Tensor final_norm, Tensor unembed, std::vector<std::vector<Tensor>> layers, Tensor g_embed,
                       Tensor g_pos, Tensor g_final_norm, Tensor g_unembed, std::vector<std::vector<Tensor>> g_layers,
                       std::vector<std::vector<Tensor>> flat, std::vector<Tensor> params, Tensor count, py::object on_bucket, py::object on_attention,
                       py::object on_end) {
        const auto [heads, head_dim, eps, cap, act, act_bwd] = c;
        return std::make_unique<StepProgram>(Config{heads, head_dim, eps, cap, act, act_bwd}, embed, pos,
                                             final_norm, unembed, layers, g_embed, g_pos, g_final_norm, g_unembed, g_layers, flat, params, count,
                                             on_bucket, on_attention, on_end);
      }))
      .def("step", [](StepProgram& p, const Tensor& ids, const Tensor& targets, double lr, double b1, double b2, double eps, double weight_decay,
                      double clip) { return p.applies() ? std::optional(p.step(ids, targets, Hyper{lr, b1, b2, eps, weight_decay, clip})) : std::nullopt; });
  m.def("softcap_ce_fits", [](double cap, int64_t rows, int64_t vocab) { return bool(api.tgh_softcap_ce_fits(float(cap), rows, vocab)); });
}
