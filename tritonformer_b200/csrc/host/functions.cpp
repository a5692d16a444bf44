// Autograd functions of the single operators.
#include "functions.h"

#include <ATen/FuncTorchTLS.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <torch/csrc/autograd/forward_grad.h>

namespace tfb_host {

// --------------------------------------------------------------------------------------------- gradient targets
bool grad_fits(const Tensor& param, at::ScalarType type) {
  if (!g_mode.accumulating.load(std::memory_order_relaxed) || !param.is_leaf()) return false;
  const Tensor& g = param.grad();
  return g.defined() && g.scalar_type() == type && g.is_contiguous() && g.sizes() == param.sizes();
}

GradTarget weight_target(const Tensor& w, at::ScalarType type) {
  GradTarget t;
  if (grad_fits(w, type)) {
    t.in_place = true;
    t.p = w.grad().data_ptr();
    t.ld = w.size(1);
    t.add = !g_mode.overwrite.load(std::memory_order_relaxed);
    if (!t.add) note_written(t.p);
    return t;
  }
  t.fresh = at::empty({w.size(0), w.size(1)}, w.options().dtype(type));
  t.p = t.fresh.data_ptr();
  t.ld = w.size(1);
  return t;
}

void weight_grad(const Mat& x, const Mat& dy, const GradTarget& g, int dtype, c10::Device device, cudaStream_t stream) {
  Epilogue e;
  if (g.add) {
    e.addend = g.p;
    e.ld_addend = g.ld;
  }
  gemm(x.t(), dy, g.p, g.ld, e, dtype, device, stream);
}

bool adjacent_columns(const Tensor* const* parts, int n, int64_t width) {
  const Tensor& first = *parts[0];
  if (!first.defined() || first.dim() != 2) return false;
  const char* base = static_cast<const char*>(first.data_ptr());
  const int64_t step = first.size(1) * first.element_size();
  for (int i = 0; i < n; ++i) {
    const Tensor& t = *parts[i];
    if (!t.defined() || t.scalar_type() != first.scalar_type() || t.sizes() != first.sizes() || t.stride(1) != 1 ||
        t.stride(0) != width || static_cast<const char*>(t.data_ptr()) != base + i * step)
      return false;
  }
  return true;
}

// A tensor that only stands for one (fake tensors, wrapper subclasses): a kernel would read from address zero.
static bool has_no_memory(const Tensor& t) {
  if (!t.unsafeGetTensorImpl()->is_python_dispatch() || t.numel() == 0) return false;
  return !t.has_storage() || t.storage().unsafeGetStorageImpl()->_mutable_data_ptr_no_checks().get() == nullptr;
}

bool needs_node(std::initializer_list<const Tensor*> inputs) {
  for (const Tensor* t : inputs)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !has_no_memory(*t),
                                "the operators of tritonformer_b200 run on tensors that hold data");
  if (const auto& functorch = at::functorch::functorchTLSAccessor()) functorch->checkSupportsCppAutogradFunction();
  if (torch::autograd::ForwardADLevel::try_get_by_idx(0))
    for (const Tensor* t : inputs)
      TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(0).defined(),
                                  "the operators of tritonformer_b200 have no forward-mode derivative");
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : inputs)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// -------------------------------------------------------------------------------------------------------- linear
static void check_linear(const Tensor& x, const Tensor& w, const Tensor& bias) {
  TFB_ASSERT(x.is_cuda() && w.is_cuda(), "Linear expects CUDA tensors");
  TFB_ASSERT(x.dim() >= 2 && w.dim() == 2, "Incorrect number of dimensions for LHS or RHS");
  if (x.size(-1) != w.size(0))
    throw ArgumentError("Dimension mismatch. Expected a.shape[2] (" + std::to_string(x.size(-1)) +
                        ") to be equal to b.shape[0] (" + std::to_string(w.size(0)) + ")");
  TFB_ASSERT((x.scalar_type() == at::kHalf || x.scalar_type() == at::kBFloat16) && w.scalar_type() == x.scalar_type(),
             "Linear expects matching fp16/bf16");
  if (bias.defined())
    TFB_ASSERT(bias.scalar_type() == x.scalar_type() && bias.numel() == w.size(1), "bias must be (out_features,)");
}

static std::vector<int64_t> with_last(const Tensor& x, int64_t n) {
  std::vector<int64_t> s = x.sizes().vec();
  s.back() = n;
  return s;
}

static Tensor linear_body(const Tensor& x, const Tensor& w, const Tensor& bias, bool relu, Mat* mx, Mat* mw) {
  check_linear(x, w, bias);
  const int dtype = dtype_code(x.scalar_type());
  *mx = tma_fit(as_rows(x), x, dtype);
  *mw = tma_fit(as_matrix(w), x, dtype);
  Tensor y = at::empty(with_last(x, mw->cols), x.options());
  Epilogue e;
  Tensor bc;
  if (bias.defined()) {
    bc = bias.contiguous();
    e.bias = bc.data_ptr();
  }
  e.relu = relu;
  gemm(*mx, *mw, y.data_ptr(), mw->cols, e, dtype, x.device(), current_stream(x));
  return y;
}

// A saved operand: the tensor itself, or the copy with aligned rows that forward made of it, by rows or by columns.  Which of
// the two forward says: a saved-tensor hook may have handed the plain tensor back with other strides.
static Mat saved_operand(const Mat& plain, const Tensor& packed, bool by_rows) {
  if (!packed.defined()) return plain;
  Mat m = plain;
  m.keep = packed;
  m.p = packed.data_ptr();
  m.s0 = by_rows ? packed.size(1) : 1;
  m.s1 = by_rows ? 1 : packed.size(1);
  return m;
}

struct LinearFn : torch::autograd::Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& w_, const OptTensor& bias_, bool relu) {
    Amp amp;
    BodyGuard guard;
    Tensor x = amp(x_), w = amp(w_);
    Mat mx, mw;
    Tensor y = linear_body(x, w, amp(val(bias_)), relu, &mx, &mw);
    ctx->saved_data["flags"] = int64_t(bias_.has_value() | (mx.s1 == 1) << 1 | (mw.s1 == 1) << 2);
    ctx->save_for_backward({x, w, relu ? y : Tensor(), mx.packed, mw.packed});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    BodyGuard guard;
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &act = saved[2];
    const at::ScalarType type = x.scalar_type();
    const int dtype = dtype_code(type);
    const int64_t flags = ctx->saved_data["flags"].toInt();
    const bool has_bias = flags & 1;
    const bool need_dx = ctx->needs_input_grad(0), need_dw = ctx->needs_input_grad(1);
    const bool need_db = has_bias && ctx->needs_input_grad(2);
    Tensor dx, dw, db;
    // dz: the incoming gradient masked by the ReLU, with rows the products can read, and its column sums
    const Tensor dy = grads[0].to(type);
    Mat dz = as_rows(dy);
    if (act.defined() || !tma_fits(dz)) {
      dz = grad_rows(dz, act, need_db ? &db : nullptr, x, dtype);
    } else if (need_db) {
      db = column_sum(dy);
    }
    const Mat mw = saved_operand(as_matrix(w), saved[4], flags & 4);
    GradTarget g;
    Mat mx;
    if (need_dx) dx = at::empty(x.sizes(), x.options());
    if (need_dw) {
      g = weight_target(w, type);
      mx = saved_operand(as_rows(x), saved[3], flags & 2);
    }
    const bool fork = need_dx && need_dw && g.in_place && g_mode.fork.load(std::memory_order_relaxed);
    SideWork side(x, fork);
    side.mark();
    if (need_dx) gemm(dz, mw.t(), dx.data_ptr(), mw.rows, Epilogue{}, dtype, x.device(), side.main());
    if (need_dw) {
      weight_grad(mx, dz, g, dtype, x.device(), side.stream());
      side.keep(mx.keep);
      side.keep(dz.keep);
      dw = g.fresh;
    }
    side.join(g_mode.defer.load(std::memory_order_relaxed));
    return {dx, dw, db, Tensor()};
  }
};

Tensor linear(const Tensor& x, const Tensor& w, const Tensor& bias, bool relu) {
  if (needs_node({&x, &w, &bias})) return LinearFn::apply(x, w, opt(bias), relu);
  Amp amp;
  BodyGuard guard;
  Mat mx, mw;
  return linear_body(amp(x), amp(w), amp(bias), relu, &mx, &mw);
}

// ----------------------------------------------------------------------------------------------------- LayerNorm
struct LayerNormFn : torch::autograd::Function<LayerNormFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& alpha_, const Tensor& beta_, double eps) {
    Amp amp;
    BodyGuard guard;
    Tensor x = amp(x_), alpha = amp(alpha_), beta = amp(beta_), y, stats;
    std::tie(y, stats) = layernorm_forward(x, alpha, beta, eps);
    ctx->save_for_backward({x, alpha, stats});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    BodyGuard guard;
    const variable_list s = ctx->get_saved_variables();
    const Tensor& x = s[0];
    Tensor da = at::empty(s[1].sizes(), x.options()), db = at::empty(s[1].sizes(), x.options());
    Tensor dx = layernorm_backward(grads[0].to(x.scalar_type()), x, s[1], s[2], Tensor(), da.data_ptr(), db.data_ptr(), false);
    return {dx, da, db, Tensor()};
  }
};

Tensor layernorm(const Tensor& x, const Tensor& alpha, const Tensor& beta, double eps) {
  if (needs_node({&x, &alpha, &beta})) return LayerNormFn::apply(x, alpha, beta, eps);
  Amp amp;
  BodyGuard guard;
  return std::get<0>(layernorm_forward(amp(x), amp(alpha), amp(beta), eps));
}

// ----------------------------------------------------------------------------------------------------- attention
static Tensor unit_inner(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
static Heads heads_of(const Tensor& t) {
  return {t.data_ptr(), {t.stride(0), t.stride(1), t.stride(2)}};
}

// q, k, v of shape (B, H, T, hd) are the views [.., 0:d], [.., d:2d], [.., 2d:3d] of one (B, T, 3 d) tensor.
static bool column_block_heads(const Tensor& q, const Tensor& k, const Tensor& v) {
  const int64_t h = q.size(1), t = q.size(2), hd = q.size(3), d = h * hd;
  const std::array<int64_t, 4> want{t * 3 * d, hd, 3 * d, 1};
  const at::IntArrayRef w(want);
  const char* p = static_cast<const char*>(q.data_ptr());
  const int64_t step = d * q.element_size();
  return q.strides() == w && k.strides() == w && v.strides() == w && static_cast<const char*>(k.data_ptr()) == p + step &&
         static_cast<const char*>(v.data_ptr()) == p + 2 * step;
}

static std::tuple<Tensor, Tensor> attention_body(Tensor& q, Tensor& k, Tensor& v, const Bias& bias) {
  TFB_ASSERT(q.is_cuda() && q.dim() == 4, "attention expects (B, H, T, head_dim) CUDA tensors");
  TFB_ASSERT(q.sizes() == k.sizes() && k.sizes() == v.sizes(), "q, k, v must have the same shape");
  TFB_ASSERT(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(),
             "attention expects matching fp16/bf16 inputs");
  const AttnShape s{q.size(0), q.size(1), q.size(2), q.size(3)};
  check_attention(s, q.scalar_type());
  q = unit_inner(q);
  k = unit_inner(k);
  v = unit_inner(v);
  Tensor out = at::empty_like(q);  // keeps q's (dense, permuted) strides
  if (out.stride(-1) != 1) out = at::empty(q.sizes(), q.options());
  Tensor lse = at::empty({s.b, s.h, s.t}, q.options().dtype(at::kFloat));
  attention_forward(heads_of(q), heads_of(k), heads_of(v), heads_of(out), static_cast<float*>(lse.data_ptr()), s, bias,
                    dtype_code(q.scalar_type()), current_stream(q));
  return {out, lse};
}

struct AttentionFn : torch::autograd::Function<AttentionFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_, const OptTensor& slopes,
                        int64_t rounded, const OptTensor& table, bool with_amp) {
    Amp amp;
    if (!with_amp) amp.on = false;
    BodyGuard guard;
    Tensor q = amp(q_), k = amp(k_), v = amp(v_), out, lse;
    const Bias bias{val(slopes), (int)rounded, val(table)};
    std::tie(out, lse) = attention_body(q, k, v, bias);
    ctx->save_for_backward({lse, q, k, v, out, bias.slopes, bias.table});
    ctx->saved_data["rounded"] = rounded;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    BodyGuard guard;
    const variable_list s = ctx->get_saved_variables();
    const Tensor &lse = s[0], &q = s[1], &k = s[2], &v = s[3], &out = s[4];
    const Bias bias{s[5], (int)ctx->saved_data["rounded"].toInt(), s[6]};
    const AttnShape shape{q.size(0), q.size(1), q.size(2), q.size(3)};
    Tensor d_out = unit_inner(grads[0].to(q.scalar_type()));
    Tensor dq, dk, dv;
    if (column_block_heads(q, k, v)) {
      // gradients laid out the same way, so that the projection's backward is one product over the whole block
      Tensor g = at::empty({shape.b, shape.t, 3, shape.h, shape.hd}, q.options());
      dq = g.select(2, 0).permute({0, 2, 1, 3});
      dk = g.select(2, 1).permute({0, 2, 1, 3});
      dv = g.select(2, 2).permute({0, 2, 1, 3});
    } else {
      dq = at::empty_like(q);
      dk = at::empty_like(k);
      dv = at::empty_like(v);
    }
    const int64_t nbytes = tfb_attention_bwd_scratch_bytes(shape.b, shape.h, shape.t, shape.hd);
    Tensor scratch = at::empty({nbytes}, q.options().dtype(at::kByte));
    attention_backward(heads_of(q), heads_of(k), heads_of(v), heads_of(out), heads_of(d_out),
                       static_cast<const float*>(lse.data_ptr()), heads_of(dq), heads_of(dk), heads_of(dv), shape, bias,
                       scratch.data_ptr(), nbytes, dtype_code(q.scalar_type()), current_stream(q));
    return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& slopes, int64_t rounded, const Tensor& table,
                 bool with_amp) {
  if (needs_node({&q, &k, &v, &slopes, &table})) return AttentionFn::apply(q, k, v, opt(slopes), rounded, opt(table), with_amp);
  Amp amp;
  if (!with_amp) amp.on = false;
  BodyGuard guard;
  Tensor q1 = amp(q), k1 = amp(k), v1 = amp(v);
  return std::get<0>(attention_body(q1, k1, v1, Bias{slopes, (int)rounded, table}));
}

// ------------------------------------------------------------------------------------------------------- softmax
static Mat unit_rows(const Tensor& t) {
  Mat m = as_rows(t);
  if (m.s1 != 1) {
    Tensor c = m.keep.contiguous();
    m = block(c.data_ptr(), m.rows, m.cols);
    m.keep = c;
  }
  if (m.rows <= 1) m.s0 = m.cols;
  return m;
}

static Tensor softmax_body(const Tensor& x) {
  TFB_ASSERT(x.is_cuda(), "Softmax expects a CUDA tensor");
  const int dtype = dtype_code(x.scalar_type());
  const Mat m = unit_rows(x);
  Tensor y = at::empty(x.sizes(), x.options());
  check(tfb_softmax_fwd(m.p, y.data_ptr(), m.rows, m.cols, m.s0, m.cols, dtype, current_stream(x)));
  return y;
}

struct SoftmaxFn : torch::autograd::Function<SoftmaxFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x) {
    BodyGuard guard;
    Tensor y = softmax_body(x);
    ctx->save_for_backward({y});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    BodyGuard guard;
    const Tensor y = ctx->get_saved_variables()[0];
    const Mat g = unit_rows(grads[0].to(y.scalar_type())), m = unit_rows(y);
    Tensor dx = at::empty(y.sizes(), y.options());
    check(tfb_softmax_bwd(g.p, m.p, dx.data_ptr(), m.rows, m.cols, g.s0, m.s0, m.cols, dtype_code(y.scalar_type()),
                          current_stream(y)));
    return {dx};
  }
};

Tensor softmax(const Tensor& x) {
  if (needs_node({&x})) return SoftmaxFn::apply(x);
  BodyGuard guard;
  return softmax_body(x);
}

// ------------------------------------------------------------------------------------------------- cross-entropy
struct CeParts {
  Tensor logits, labels, lse, loss;
};
static CeParts cross_entropy_body(Tensor logits, Tensor labels, bool f32) {
  TFB_ASSERT(logits.is_cuda() && logits.dim() == 2, "cross entropy expects a 2-D CUDA logits tensor");
  TFB_ASSERT(logits.scalar_type() == at::kHalf || logits.scalar_type() == at::kBFloat16,
             "cross entropy expects fp16/bf16 logits");
  TFB_ASSERT(labels.dim() == 1 && labels.size(0) == logits.size(0), "labels must be (N,)");
  if (logits.stride(1) != 1) logits = logits.contiguous();
  labels = labels.to(at::kLong).contiguous();
  const int64_t n = logits.size(0), v = logits.size(1);
  Tensor loss16 = at::empty({n}, logits.options()), lse = at::empty({n}, logits.options().dtype(at::kFloat)), loss32;
  if (f32) loss32 = at::empty({n}, lse.options());
  check(tfb_cross_entropy_fwd(logits.data_ptr(), static_cast<const int64_t*>(labels.data_ptr()), loss16.data_ptr(),
                              f32 ? static_cast<float*>(loss32.data_ptr()) : nullptr, static_cast<float*>(lse.data_ptr()), n, v,
                              n > 1 ? logits.stride(0) : v, dtype_code(logits.scalar_type()), current_stream(logits)));
  return {logits, labels, lse, f32 ? loss32 : loss16};
}

struct CrossEntropyFn : torch::autograd::Function<CrossEntropyFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& labels, bool f32) {
    Amp amp;
    BodyGuard guard;
    CeParts p = cross_entropy_body(amp(logits), labels, f32);
    ctx->save_for_backward({p.logits, p.labels, p.lse});
    return p.loss;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    BodyGuard guard;
    const variable_list s = ctx->get_saved_variables();
    const Tensor& logits = s[0];
    const int64_t n = logits.size(0), v = logits.size(1);
    const Tensor g = grads[0].to(logits.scalar_type());  // keeps a stride-0 expand as it is
    const int64_t gs = g.dim() == 1 && n > 1 ? g.stride(0) : 0;
    Tensor dlogits = at::empty({n, v}, logits.options());
    check(tfb_cross_entropy_bwd(logits.data_ptr(), static_cast<const int64_t*>(s[1].data_ptr()),
                                static_cast<const float*>(s[2].data_ptr()), g.data_ptr(), gs, dlogits.data_ptr(), n, v,
                                n > 1 ? logits.stride(0) : v, v, dtype_code(logits.scalar_type()), current_stream(logits)));
    return {dlogits, Tensor(), Tensor()};
  }
};

Tensor cross_entropy(const Tensor& logits, const Tensor& labels, bool f32) {
  if (needs_node({&logits})) return CrossEntropyFn::apply(logits, labels, f32);
  Amp amp;
  BodyGuard guard;
  return cross_entropy_body(amp(logits), labels, f32).loss;
}

// The model's loss: position t against label t + 1, mean over the positions that have one, in fp32.
static std::tuple<Tensor, Tensor, Tensor> lm_loss_body(Tensor& logits, Tensor labels) {
  TFB_ASSERT(logits.is_cuda() && logits.dim() == 3, "the loss expects CUDA (batch, seq, vocab) logits");
  TFB_ASSERT(logits.scalar_type() == at::kHalf || logits.scalar_type() == at::kBFloat16,
             "cross entropy expects fp16/bf16 logits");
  TFB_ASSERT(labels.dim() == 2 && labels.size(0) == logits.size(0) && labels.size(1) == logits.size(1),
             "labels must be (batch, seq)");
  logits = logits.contiguous();
  labels = labels.to(at::kLong).contiguous();
  const int64_t b = logits.size(0), t = logits.size(1), v = logits.size(2);
  Tensor rows = at::empty({2, b * t}, logits.options().dtype(at::kFloat)), loss = at::empty({}, rows.options());
  float* r = static_cast<float*>(rows.data_ptr());
  check(tfb_lm_loss_fwd(logits.data_ptr(), static_cast<const int64_t*>(labels.data_ptr()), static_cast<float*>(loss.data_ptr()),
                        r + b * t, r, b, t, v, v, dtype_code(logits.scalar_type()), current_stream(logits)));
  return {loss, labels, rows};
}

struct LmLossFn : torch::autograd::Function<LmLossFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits_, const Tensor& labels_) {
    Amp amp;
    BodyGuard guard;
    Tensor logits = amp(logits_), loss, labels, rows;
    std::tie(loss, labels, rows) = lm_loss_body(logits, labels_);
    ctx->save_for_backward({logits, labels, rows});
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    BodyGuard guard;
    const variable_list s = ctx->get_saved_variables();
    const Tensor& logits = s[0];
    const int64_t b = logits.size(0), t = logits.size(1), v = logits.size(2);
    const Tensor g = grads[0].to(at::kFloat);
    // rows of an odd vocabulary are padded to 16 bytes, as the head's products want to read them
    const int64_t ld = (v + 7) / 8 * 8;
    Tensor dlogits = at::empty({b, t, ld}, logits.options());
    if (ld != v) dlogits = dlogits.slice(2, 0, v);
    check(tfb_lm_loss_bwd(logits.data_ptr(), static_cast<const int64_t*>(s[1].data_ptr()),
                          static_cast<const float*>(s[2].data_ptr()), static_cast<const float*>(g.data_ptr()), dlogits.data_ptr(),
                          b, t, v, v, ld, dtype_code(logits.scalar_type()), current_stream(logits)));
    return {dlogits, Tensor()};
  }
};

Tensor lm_loss(const Tensor& logits, const Tensor& labels) {
  if (needs_node({&logits})) return LmLossFn::apply(logits, labels);
  Amp amp;
  BodyGuard guard;
  Tensor l = amp(logits);
  return std::get<0>(lm_loss_body(l, labels));
}

// ----------------------------------------------------------------------------------------------------- embedding
static Tensor embedding_body(const Tensor& ids, const Tensor& tok, const Tensor& pos) {
  TFB_ASSERT(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.dim() == 2,
             "embedding expects a CUDA int64 (batch, seq) tensor of token ids");
  TFB_ASSERT(tok.dim() == 2 && (tok.scalar_type() == at::kHalf || tok.scalar_type() == at::kBFloat16),
             "embedding expects a (vocab, d) fp16/bf16 table");
  const int64_t batch = ids.size(0), seq = ids.size(1), vocab = tok.size(0), d = tok.size(1);
  Tensor pc;
  if (pos.defined()) {
    TFB_ASSERT(pos.scalar_type() == tok.scalar_type() && pos.dim() == 2 && pos.size(1) == d, "position table mismatch");
    TFB_ASSERT(pos.size(0) >= seq, "sequence longer than the position table");
    pc = pos.contiguous();
  }
  Tensor ic = ids.contiguous(), tc = tok.contiguous();
  Tensor out = at::empty({batch, seq, d}, tok.options());
  check(tfb_embedding_fwd(static_cast<const int64_t*>(ic.data_ptr()), tc.data_ptr(), pc.defined() ? pc.data_ptr() : nullptr,
                          out.data_ptr(), batch, seq, d, vocab, pc.defined() ? pc.size(0) : 0, dtype_code(tok.scalar_type()),
                          current_stream(tok)));
  return out;
}

struct EmbeddingFn : torch::autograd::Function<EmbeddingFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& ids, const Tensor& tok_, const OptTensor& pos_) {
    Amp amp;
    BodyGuard guard;
    Tensor tok = amp(tok_), pos = amp(val(pos_));
    ctx->save_for_backward({ids, tok, pos});
    return embedding_body(ids, tok, pos);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    BodyGuard guard;
    const variable_list s = ctx->get_saved_variables();
    const Tensor &ids = s[0], &tok = s[1], &pos = s[2];
    // the kernels ADD: into .grad itself where it fits, else into a zeroed tensor; a frozen table gets no buffer at all
    auto target = [&](const Tensor& p, bool need) {
      GradTarget t;
      if (!p.defined() || !need) return t;
      if (grad_fits(p, p.scalar_type())) {
        t.p = p.grad().data_ptr();
      } else {
        t.fresh = at::zeros(p.sizes(), p.options());
        t.p = t.fresh.data_ptr();
      }
      return t;
    };
    const GradTarget gt = target(tok, ctx->needs_input_grad(1)), gp = target(pos, pos.defined() && ctx->needs_input_grad(2));
    if (gt.p || gp.p) {
      const int64_t batch = ids.size(0), seq = ids.size(1), vocab = tok.size(0), d = tok.size(1);
      Tensor ic = ids.contiguous(), dout = grads[0].to(tok.scalar_type()).contiguous();
      const int64_t nbytes = tfb_embedding_bwd_scratch_bytes(batch, seq, d, vocab);
      Tensor scratch = at::empty({nbytes}, tok.options().dtype(at::kByte));
      check(tfb_embedding_bwd(static_cast<const int64_t*>(ic.data_ptr()), dout.data_ptr(), gt.p, gp.p, scratch.data_ptr(), nbytes,
                              batch, seq, d, vocab, gp.p ? pos.size(0) : 0, dtype_code(tok.scalar_type()), current_stream(tok)));
    }
    return {Tensor(), gt.fresh, gp.fresh};
  }
};

Tensor embedding(const Tensor& ids, const Tensor& tok, const Tensor& pos) {
  if (needs_node({&tok, &pos})) return EmbeddingFn::apply(ids, tok, opt(pos));
  Amp amp;
  BodyGuard guard;
  return embedding_body(ids, amp(tok), amp(pos));
}

}  // namespace tfb_host
