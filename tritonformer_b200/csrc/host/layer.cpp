// One pre-LayerNorm transformer layer as one autograd node:
//   h = x + Attention(LN1(x)) Wo,   y = h + relu(LN2(h) W1 + b1) W2 + b2
// Forward is seven kernels, backward fourteen and more (sums of the biases); the residual adds, the ReLU mask and the
// sums of the residual gradients happen inside them.
#include "functions.h"

#include <ATen/ops/cat.h>
#include <ATen/ops/empty.h>

namespace tfb_host {

struct LayerSaved {  // what forward leaves for backward
  Tensor normed1, stats1, wqkv, qkv, ctx, lse, h, normed2, stats2, act;
};

static const void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// [Wq | Wk | Wv]: in place if the three already are the column blocks of one matrix (Transformer.fuse_projection_weights),
// else concatenated.
static Mat qkv_matrix(const LayerWeights& w, Tensor* cat) {
  const int64_t d = w.wq.size(1);
  const Tensor* parts[3] = {&w.wq, &w.wk, &w.wv};
  if (adjacent_columns(parts, 3, 3 * d)) {
    Mat m = block(w.wq.data_ptr(), w.wq.size(0), 3 * d);
    m.keep = w.wq;
    return m;
  }
  *cat = at::cat({w.wq, w.wk, w.wv}, 1);
  return as_matrix(*cat);
}

static void check_layer(const Tensor& x, const LayerWeights& w, int64_t heads) {
  TFB_ASSERT(x.is_cuda() && x.dim() == 3, "the layer expects a CUDA (batch, seq, d) tensor");
  const int64_t d = x.size(2), f = w.w1.size(1);
  for (const Tensor* p : {&w.wq, &w.wk, &w.wv, &w.wo, &w.w1, &w.w2}) {
    TFB_ASSERT(p->is_cuda() && p->dim() == 2, "Linear expects CUDA tensors");
    TFB_ASSERT((x.scalar_type() == at::kHalf || x.scalar_type() == at::kBFloat16) && p->scalar_type() == x.scalar_type(),
               "Linear expects matching fp16/bf16");
  }
  for (const Tensor* p : {&w.wq, &w.wk, &w.wv, &w.wo})
    TFB_ASSERT(p->size(0) == d && p->size(1) == d, "Dimension mismatch in the attention projections");
  TFB_ASSERT(w.w1.size(0) == d && w.w2.size(0) == f && w.w2.size(1) == d, "Dimension mismatch in the MLP");
  TFB_ASSERT(heads > 0 && d % heads == 0, "the number of heads must divide the hidden size");
  const std::pair<const Tensor*, int64_t> biases[2] = {{&w.b1, f}, {&w.b2, d}};
  for (const auto& b : biases)
    if (b.first->defined())
      TFB_ASSERT(b.first->scalar_type() == x.scalar_type() && b.first->numel() == b.second, "bias must be (out_features,)");
}

static Tensor layer_forward(const Tensor& x_, const LayerWeights& w, const Bias& bias, int64_t heads, double eps1, double eps2,
                            LayerSaved* s) {
  check_layer(x_, w, heads);
  const Tensor x = x_.contiguous();
  const int64_t b = x.size(0), t = x.size(1), d = x.size(2), f = w.w1.size(1), rows = b * t;
  const AttnShape shape{b, heads, t, d / heads};
  check_attention(shape, x.scalar_type());
  const int dtype = dtype_code(x.scalar_type());
  const c10::Device dev = x.device();
  cudaStream_t st = current_stream(x);
  const Epilogue plain;

  std::tie(s->normed1, s->stats1) = layernorm_forward(x, w.ln1_w, w.ln1_b, eps1);
  const Mat wqkv = qkv_matrix(w, &s->wqkv);
  s->qkv = at::empty({b, t, 3 * d}, x.options());
  gemm(block(s->normed1.data_ptr(), rows, d), wqkv, s->qkv.data_ptr(), 3 * d, plain, dtype, dev, st);

  s->ctx = at::empty({b, t, d}, x.options());
  s->lse = at::empty({b, heads, t}, x.options().dtype(at::kFloat));
  char* q = static_cast<char*>(s->qkv.data_ptr());
  const int64_t es = x.element_size(), hd = shape.hd;
  auto in = [&](int i) { return Heads{q + i * d * es, {t * 3 * d, hd, 3 * d}}; };
  const Heads out{s->ctx.data_ptr(), {t * d, hd, d}};
  attention_forward(in(0), in(1), in(2), out, static_cast<float*>(s->lse.data_ptr()), shape, bias, dtype, st);

  s->h = at::empty(x.sizes(), x.options());
  Epilogue residual;
  residual.addend = x.data_ptr();
  residual.ld_addend = d;
  gemm(block(s->ctx.data_ptr(), rows, d), as_matrix(w.wo), s->h.data_ptr(), d, residual, dtype, dev, st);

  std::tie(s->normed2, s->stats2) = layernorm_forward(s->h, w.ln2_w, w.ln2_b, eps2);
  s->act = at::empty({b, t, f}, x.options());
  Epilogue relu;
  relu.relu = true;
  relu.bias = ptr(w.b1);
  gemm(block(s->normed2.data_ptr(), rows, d), as_matrix(w.w1), s->act.data_ptr(), f, relu, dtype, dev, st);

  Tensor y = at::empty(x.sizes(), x.options());
  residual.addend = s->h.data_ptr();
  residual.bias = ptr(w.b2);
  gemm(block(s->act.data_ptr(), rows, f), as_matrix(w.w2), y.data_ptr(), d, residual, dtype, dev, st);
  return y;
}

struct LayerFn : torch::autograd::Function<LayerFn> {
  // edges: x, ln1_w, ln1_b, wq, wk, wv, wo, ln2_w, ln2_b, w1, w2, then b1 and b2 where they exist
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& ln1_w, const Tensor& ln1_b, const Tensor& wq,
                        const Tensor& wk, const Tensor& wv, const Tensor& wo, const Tensor& ln2_w, const Tensor& ln2_b,
                        const Tensor& w1, const Tensor& w2, const OptTensor& b1, const OptTensor& b2, const Bias* bias,
                        int64_t heads, double eps1, double eps2) {
    Amp a;
    BodyGuard guard;
    const LayerWeights w{a(ln1_w), a(ln1_b), a(wq), a(wk), a(wv), a(wo), a(ln2_w), a(ln2_b), a(w1), a(val(b1)), a(w2), a(val(b2))};
    Tensor x = a(x_);
    LayerSaved s;
    Tensor y = layer_forward(x, w, *bias, heads, eps1, eps2, &s);
    ctx->save_for_backward({x, w.ln1_w, w.ln1_b, w.wq, w.wk, w.wv, w.wo, w.ln2_w, w.ln2_b, w.w1, w.w2, s.normed1, s.stats1,
                            s.wqkv, s.qkv, s.ctx, s.lse, s.h, s.normed2, s.stats2, s.act, bias->slopes, bias->table});
    ctx->saved_data["i"] = std::vector<int64_t>{heads, bias->rounded, b1.has_value(), b2.has_value()};
    return y;
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    BodyGuard guard;
    const variable_list v = ctx->get_saved_variables();
    const Tensor &ln1_w = v[1], &ln1_b = v[2], &wq = v[3], &wk = v[4], &wv = v[5], &wo = v[6], &ln2_w = v[7], &ln2_b = v[8],
                 &w1 = v[9], &w2 = v[10], &normed1 = v[11], &stats1 = v[12], &wcat = v[13], &qkv = v[14], &att = v[15],
                 &lse = v[16], &h = v[17], &normed2 = v[18], &stats2 = v[19], &act = v[20];
    const Tensor x = v[0].contiguous();
    const std::vector<int64_t> ints = ctx->saved_data["i"].toIntVector();
    const int64_t heads = ints[0];
    const bool has_b1 = ints[2] != 0, has_b2 = ints[3] != 0;
    const Bias bias{v[21], (int)ints[1], v[22]};
    const int64_t b = x.size(0), t = x.size(1), d = x.size(2), f = w1.size(1), rows = b * t;
    const AttnShape shape{b, heads, t, d / heads};
    const at::ScalarType type = x.scalar_type();
    const int dtype = dtype_code(type);
    const c10::Device dev = x.device();
    auto need = [&](size_t i) { return ctx->needs_input_grad(i); };
    const bool need_b1 = has_b1 && need(11), need_b2 = has_b2 && need(11 + (has_b1 ? 1 : 0));
    const Tensor dy = grads[0].to(type).contiguous();
    const Mat mdy = block(dy.data_ptr(), rows, d);
    Tensor db1, db2;

    // where the weight gradients go (all targets exist before the side stream starts)
    GradTarget gw1, gw2, gwo, gq[3], gqkv;
    if (need(9)) gw1 = weight_target(w1, type);
    if (need(10)) gw2 = weight_target(w2, type);
    if (need(6)) gwo = weight_target(wo, type);
    const Tensor* wparts[3] = {&wq, &wk, &wv};
    bool one_product = need(3) && need(4) && need(5);
    if (one_product) {
      // one product for the three, if they can land in column blocks of one matrix
      bool fits = g_mode.accumulating.load(std::memory_order_relaxed);
      const Tensor* gparts[3];
      for (int i = 0; i < 3 && fits; ++i) {
        fits = wparts[i]->is_leaf() && wparts[i]->grad().defined() && wparts[i]->grad().scalar_type() == type;
        gparts[i] = fits ? &wparts[i]->grad() : nullptr;
      }
      if (fits && gparts[0]->sizes() == wq.sizes() && adjacent_columns(gparts, 3, 3 * d)) {
        gqkv.in_place = true;
        gqkv.p = gparts[0]->data_ptr();
        gqkv.ld = 3 * d;
        gqkv.add = !g_mode.overwrite.load(std::memory_order_relaxed);
        if (!gqkv.add)
          for (const Tensor* g : gparts) note_written(g->data_ptr());
      } else {
        one_product = false;
      }
    }
    if (!one_product)
      for (int i = 0; i < 3; ++i)
        if (need(3 + i)) gq[i] = weight_target(*wparts[i], type);
    SideWork side(x, g_mode.fork.load(std::memory_order_relaxed));
    cudaStream_t st = side.main();

    // MLP
    side.mark();
    Tensor dz = at::empty({b, t, f}, x.options());
    Epilogue mask;
    mask.mask = act.data_ptr();
    mask.ld_mask = f;
    gemm(mdy, as_matrix(w2).t(), dz.data_ptr(), f, mask, dtype, dev, st);
    if (need(10)) weight_grad(block(act.data_ptr(), rows, f), mdy, gw2, dtype, dev, side.stream());
    if (need_b2) db2 = column_sum(dy);
    const Mat mdz = block(dz.data_ptr(), rows, f);
    side.mark();
    Tensor dn = at::empty(x.sizes(), x.options());
    gemm(mdz, as_matrix(w1).t(), dn.data_ptr(), d, Epilogue{}, dtype, dev, st);
    if (need(9)) weight_grad(block(normed2.data_ptr(), rows, d), mdz, gw1, dtype, dev, side.stream());
    if (need_b1) db1 = column_sum(dz);
    Tensor da2, db2n, da1, db1n;
    Tensor dh = norm_backward(dn, h, ln2_w, ln2_b, stats2, dy, need(7), need(8), &da2, &db2n);

    // attention
    const Mat mdh = block(dh.data_ptr(), rows, d);
    side.mark();
    Tensor datt = at::empty(x.sizes(), x.options());
    gemm(mdh, as_matrix(wo).t(), datt.data_ptr(), d, Epilogue{}, dtype, dev, st);
    if (need(6)) weight_grad(block(att.data_ptr(), rows, d), mdh, gwo, dtype, dev, side.stream());
    Tensor dqkv = at::empty({b, t, 3 * d}, x.options());
    const int64_t es = x.element_size(), hd = shape.hd;
    auto blocks = [&](const Tensor& m, int i) {
      return Heads{static_cast<char*>(m.data_ptr()) + i * d * es, {t * 3 * d, hd, 3 * d}};
    };
    const Heads o{att.data_ptr(), {t * d, hd, d}}, d_o{datt.data_ptr(), {t * d, hd, d}};
    attention_backward(blocks(qkv, 0), blocks(qkv, 1), blocks(qkv, 2), o, d_o, static_cast<const float*>(lse.data_ptr()),
                       blocks(dqkv, 0), blocks(dqkv, 1), blocks(dqkv, 2), shape, bias, x, dtype, st);
    const Mat mdqkv = block(dqkv.data_ptr(), rows, 3 * d), mn1 = block(normed1.data_ptr(), rows, d);
    side.mark();
    const bool need_dx = need(0) || need(1) || need(2);
    Tensor dx, dn1;
    if (need_dx) {
      dn1 = at::empty(x.sizes(), x.options());
      const Mat wqkv = wcat.defined() ? as_matrix(wcat) : block(wq.data_ptr(), d, 3 * d);
      gemm(mdqkv, wqkv.t(), dn1.data_ptr(), d, Epilogue{}, dtype, dev, st);
    }
    if (need(3) || need(4) || need(5)) {
      cudaStream_t ss = side.stream();
      if (one_product) {
        weight_grad(mn1, mdqkv, gqkv, dtype, dev, ss);
      } else {
        for (int i = 0; i < 3; ++i)
          if (gq[i].p) {
            Mat part = mdqkv;
            part.p = static_cast<const char*>(mdqkv.p) + i * d * es;
            part.cols = d;
            weight_grad(mn1, part, gq[i], dtype, dev, ss);
          }
      }
    }
    if (need_dx) dx = norm_backward(dn1, x, ln1_w, ln1_b, stats1, dh, need(1), need(2), &da1, &db1n);
    const bool all_in_place = !(gw1.fresh.defined() || gw2.fresh.defined() || gwo.fresh.defined() || gq[0].fresh.defined() ||
                                gq[1].fresh.defined() || gq[2].fresh.defined());
    for (const Tensor& k : {dy, act, dz, normed2, dh, att, dqkv, normed1}) side.keep(k);
    side.join(all_in_place && g_mode.defer.load(std::memory_order_relaxed));
    return {dx, da1, db1n, gq[0].fresh, gq[1].fresh, gq[2].fresh, gwo.fresh, da2, db2n, gw1.fresh, gw2.fresh, db1, db2,
            Tensor(), Tensor(), Tensor(), Tensor()};
  }

  // LayerNorm backward with the residual gradient added; parameter gradients go into .grad where both fit.
  static Tensor norm_backward(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& b, const Tensor& stats,
                              const Tensor& dres, bool need_w, bool need_b, Tensor* dw, Tensor* db) {
    if (need_w && need_b && grad_fits(w, x.scalar_type()) && grad_fits(b, x.scalar_type())) {
      const bool add = !g_mode.overwrite.load(std::memory_order_relaxed);
      if (!add) {
        note_written(w.grad().data_ptr());
        note_written(b.grad().data_ptr());
      }
      return layernorm_backward(dy, x, w, stats, dres, w.grad().data_ptr(), b.grad().data_ptr(), add);
    }
    *dw = at::empty(w.sizes(), x.options());
    *db = at::empty(w.sizes(), x.options());
    return layernorm_backward(dy, x, w, stats, dres, dw->data_ptr(), db->data_ptr(), false);
  }
};

Tensor layer(const Tensor& x, const LayerWeights& w, const Bias& bias_, int64_t heads, double eps1, double eps2) {
  Bias bias = bias_;
  if (bias.table.defined()) {  // the attention reads the table in the type it computes in
    const Amp amp;
    bias.table = bias.table.to(amp.on ? amp.type : x.scalar_type());
  }
  bool grad = at::GradMode::is_enabled();
  if (grad) {
    grad = false;
    for (const Tensor* t : {&x, &w.ln1_w, &w.ln1_b, &w.wq, &w.wk, &w.wv, &w.wo, &w.ln2_w, &w.ln2_b, &w.w1, &w.b1, &w.w2, &w.b2})
      grad = grad || (t->defined() && t->requires_grad());
  }
  if (grad)
    return LayerFn::apply(x, w.ln1_w, w.ln1_b, w.wq, w.wk, w.wv, w.wo, w.ln2_w, w.ln2_b, w.w1, w.w2, opt(w.b1), opt(w.b2), &bias,
                          heads, eps1, eps2);
  Amp a;
  BodyGuard guard;
  const LayerWeights c{a(w.ln1_w), a(w.ln1_b), a(w.wq), a(w.wk), a(w.wv), a(w.wo), a(w.ln2_w), a(w.ln2_b), a(w.w1), a(w.b1), a(w.w2),
                       a(w.b2)};
  LayerSaved s;
  return layer_forward(a(x), c, bias, heads, eps1, eps2, &s);
}

}  // namespace tfb_host
