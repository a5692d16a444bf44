// One pre-LayerNorm transformer layer as one autograd node:
//   h = x + Attention(LN1(x)) Wo,   y = h + relu(LN2(h) W1 + b1) W2 + b2
// Forward is seven kernels, backward fourteen and more (sums of the biases); the residual adds, the ReLU mask and the
// sums of the residual gradients happen inside them.
#include "functions.h"

#include <ATen/ops/cat.h>
#include <ATen/ops/empty.h>

namespace tfb_host {

// Regions of one allocation.  A layer's intermediates live and die together, so they share one block instead of ten
// (an allocation costs about half a kernel launch).
class Slab {
 public:
  size_t add(int64_t bytes) {
    const size_t at = size_;
    size_ += ((size_t)bytes + 255) & ~size_t(255);
    return at;
  }
  void allocate(const Tensor& like) {
    buf = at::empty({(int64_t)size_}, like.options().dtype(at::kByte));
    base_ = static_cast<char*>(buf.data_ptr());
  }
  void attach(const Tensor& t) {
    buf = t;
    base_ = static_cast<char*>(t.data_ptr());
  }
  char* operator[](size_t at) const { return base_ + at; }
  Tensor buf;
 private:
  size_t size_ = 0;
  char* base_ = nullptr;
};

// What forward leaves for backward, in one block.
struct Saved {
  Slab slab;
  size_t normed1, stats1, qkv, ctx, lse, h, normed2, stats2, act;
  Saved(int64_t rows, int64_t d, int64_t f, int64_t heads) {
    normed1 = slab.add(rows * d * 2);
    stats1 = slab.add(rows * 8);
    qkv = slab.add(rows * 3 * d * 2);
    ctx = slab.add(rows * d * 2);
    lse = slab.add(rows * heads * 4);
    h = slab.add(rows * d * 2);
    normed2 = slab.add(rows * d * 2);
    stats2 = slab.add(rows * 8);
    act = slab.add(rows * f * 2);
  }
  float* floats(size_t at) const { return reinterpret_cast<float*>(slab[at]); }
  Tensor activations(const Tensor& x, int64_t f) const {  // relu(LN2(h) W1 + b1) as a tensor
    const int64_t rows = x.size(0) * x.size(1);
    return slab.buf.narrow(0, (int64_t)act, rows * f * 2).view(x.scalar_type()).view({x.size(0), x.size(1), f});
  }
};

static const void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// [Wq | Wk | Wv]: in place if the three already are the column blocks of one matrix (Transformer.fuse_projection_weights),
// else concatenated.
static Mat qkv_matrix(const Tensor& wq, const Tensor& wk, const Tensor& wv, Tensor* cat) {
  const int64_t d = wq.size(1);
  const Tensor* parts[3] = {&wq, &wk, &wv};
  if (adjacent_columns(parts, 3, 3 * d)) {
    Mat m = block(wq.data_ptr(), wq.size(0), 3 * d);
    m.keep = wq;
    return m;
  }
  *cat = at::cat({wq, wk, wv}, 1);
  return as_matrix(*cat);
}

static void check_layer(const Tensor& x, LayerWeights& w, int64_t heads) {
  TFB_ASSERT(x.is_cuda() && x.dim() == 3, "the layer expects a CUDA (batch, seq, d) tensor");
  TFB_ASSERT(x.scalar_type() == at::kHalf || x.scalar_type() == at::kBFloat16, "LayerNorm expects a CUDA fp16/bf16 input");
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
  if (x.size(0) == 0 || x.size(1) == 0)
    throw ArgumentError("attention: bad shape B=" + std::to_string(x.size(0)) + " H=" + std::to_string(heads) +
                        " T=" + std::to_string(x.size(1)));
  check_attention({x.size(0), heads, x.size(1), d / heads}, x.scalar_type());
  for (Tensor* p : {&w.ln1_w, &w.ln1_b, &w.ln2_w, &w.ln2_b}) {
    TFB_ASSERT(p->scalar_type() == x.scalar_type(), "LayerNorm parameters must match the input dtype");
    TFB_ASSERT(p->numel() == d, "LayerNorm parameter size mismatch");
    *p = p->contiguous();
  }
  const std::pair<Tensor*, int64_t> biases[2] = {{&w.b1, f}, {&w.b2, d}};
  for (const auto& b : biases)
    if (b.first->defined()) {
      TFB_ASSERT(b.first->scalar_type() == x.scalar_type() && b.first->numel() == b.second, "bias must be (out_features,)");
      *b.first = b.first->contiguous();
    }
}

static void norm_forward(const void* x, const Tensor& w, const Tensor& b, void* y, float* stats, int64_t rows, int64_t d,
                         double eps, int dtype, cudaStream_t st) {
  check(tfb_layernorm_fwd(x, w.data_ptr(), b.data_ptr(), y, stats, stats + rows, rows, d, d, d, (float)eps, dtype, st));
}

static Tensor layer_forward(const Tensor& x, const LayerWeights& w, const Bias& bias, int64_t heads, double eps1, double eps2,
                            Saved& s, Tensor* wcat) {
  const int64_t b = x.size(0), t = x.size(1), d = x.size(2), f = w.w1.size(1), rows = b * t;
  const AttnShape shape{b, heads, t, d / heads};
  const int dtype = dtype_code(x.scalar_type());
  const c10::Device dev = x.device();
  cudaStream_t st = current_stream(x);
  s.slab.allocate(x);
  Tensor y = at::empty(x.sizes(), x.options());

  norm_forward(x.data_ptr(), w.ln1_w, w.ln1_b, s.slab[s.normed1], s.floats(s.stats1), rows, d, eps1, dtype, st);
  gemm(block(s.slab[s.normed1], rows, d), qkv_matrix(w.wq, w.wk, w.wv, wcat), s.slab[s.qkv], 3 * d, Epilogue{}, dtype, dev, st);
  const int64_t es = x.element_size(), hd = shape.hd;
  auto in = [&](int i) { return Heads{s.slab[s.qkv] + i * d * es, {t * 3 * d, hd, 3 * d}}; };
  const Heads out{s.slab[s.ctx], {t * d, hd, d}};
  attention_forward(in(0), in(1), in(2), out, s.floats(s.lse), shape, bias, dtype, st);
  Epilogue residual;
  residual.addend = x.data_ptr();
  residual.ld_addend = d;
  gemm(block(s.slab[s.ctx], rows, d), as_matrix(w.wo), s.slab[s.h], d, residual, dtype, dev, st);

  norm_forward(s.slab[s.h], w.ln2_w, w.ln2_b, s.slab[s.normed2], s.floats(s.stats2), rows, d, eps2, dtype, st);
  Epilogue relu;
  relu.relu = true;
  relu.bias = ptr(w.b1);
  gemm(block(s.slab[s.normed2], rows, d), as_matrix(w.w1), s.slab[s.act], f, relu, dtype, dev, st);
  residual.addend = s.slab[s.h];
  residual.bias = ptr(w.b2);
  gemm(block(s.slab[s.act], rows, f), as_matrix(w.w2), y.data_ptr(), d, residual, dtype, dev, st);
  return y;
}

struct LayerFn : torch::autograd::Function<LayerFn> {
  // edges: x, ln1_w, ln1_b, wq, wk, wv, wo, ln2_w, ln2_b, w1, w2, then b1 and b2 where they exist
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& ln1_w, const Tensor& ln1_b, const Tensor& wq,
                        const Tensor& wk, const Tensor& wv, const Tensor& wo, const Tensor& ln2_w, const Tensor& ln2_b,
                        const Tensor& w1, const Tensor& w2, const OptTensor& b1, const OptTensor& b2, const Bias* bias,
                        int64_t heads, double eps1, double eps2, Tensor* act) {
    Amp a;
    BodyGuard guard;
    LayerWeights w{a(ln1_w), a(ln1_b), a(wq), a(wk), a(wv), a(wo), a(ln2_w), a(ln2_b), a(w1), a(val(b1)), a(w2), a(val(b2))};
    const Tensor x = a(x_).contiguous();
    check_layer(x, w, heads);
    Saved s(x.size(0) * x.size(1), x.size(2), w.w1.size(1), heads);
    Tensor wcat;
    Tensor y = layer_forward(x, w, *bias, heads, eps1, eps2, s, &wcat);
    if (act) *act = s.activations(x, w.w1.size(1));
    ctx->save_for_backward({x, w.ln1_w, w.ln1_b, w.wq, w.wk, w.wv, w.wo, w.ln2_w, w.ln2_b, w.w1, w.w2, wcat, s.slab.buf,
                            bias->slopes, bias->table});
    ctx->saved_data["i"] = std::vector<int64_t>{heads, bias->rounded, b1.has_value(), b2.has_value()};
    return y;
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    BodyGuard guard;
    // Saved-tensor hooks may hand back copies with strides of their own, so nothing that forward found out about the layout
    // of a saved tensor holds here: it is asked again, or the tensor made contiguous.
    const variable_list v = ctx->get_saved_variables();
    const Tensor x = v[0].contiguous(), &ln1_w = v[1], &ln1_b = v[2], &wq = v[3], &wk = v[4], &wv = v[5], &wo = v[6],
                 &ln2_w = v[7], &ln2_b = v[8], &w1 = v[9], &w2 = v[10], &wcat = v[11];
    const std::vector<int64_t> ints = ctx->saved_data["i"].toIntVector();
    const int64_t heads = ints[0];
    const bool has_b1 = ints[2] != 0, has_b2 = ints[3] != 0;
    const Bias bias{v[13], (int)ints[1], v[14]};
    const int64_t b = x.size(0), t = x.size(1), d = x.size(2), f = w1.size(1), rows = b * t;
    Saved s(rows, d, f, heads);
    s.slab.attach(v[12]);
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
    Tensor dx = at::empty(x.sizes(), x.options());
    // scratch of the whole backward; `chain` holds one after the other the gradients that only the next kernel of this
    // stream reads
    Slab k;
    const int64_t ln_partials = tfb_layernorm_bwd_partials(rows, d);
    const int64_t scratch_bytes = tfb_attention_bwd_scratch_bytes(shape.b, shape.h, shape.t, shape.hd);
    const size_t dz_at = k.add(rows * f * 2), chain_at = k.add(rows * d * 2), dh_at = k.add(rows * d * 2),
                 dqkv_at = k.add(rows * 3 * d * 2), attn_at = k.add(scratch_bytes), part_at = k.add(ln_partials * 2 * d * 4),
                 sums_at = k.add(std::max(need_b1 ? tfb_colsum_partials(rows, f) * f : 0, need_b2 ? tfb_colsum_partials(rows, d) * d : 0) * 4);
    k.allocate(x);
    float* sums = reinterpret_cast<float*>(k[sums_at]);
    SideWork side(x, g_mode.fork.load(std::memory_order_relaxed));
    cudaStream_t st = side.main();
    const Mat mdz = block(k[dz_at], rows, f), mchain = block(k[chain_at], rows, d);
    auto colsum = [&](const Mat& m, Tensor* out) {
      *out = at::empty({m.cols}, x.options());
      check(tfb_colsum(m.p, out->data_ptr(), sums, tfb_colsum_partials(m.rows, m.cols), m.rows, m.cols, m.cols, dtype, st));
    };
    // LayerNorm backward with the residual gradient added; parameter gradients go into .grad where both fit
    auto norm_backward = [&](const void* in, const Tensor& w, const Tensor& beta, const float* stats, const void* dres, void* out,
                             bool need_w, bool need_b, Tensor* dw, Tensor* db) {
      void *pw, *pb;
      bool add = false;
      if (need_w && need_b && grad_fits(w, type) && grad_fits(beta, type)) {
        pw = w.grad().data_ptr();
        pb = beta.grad().data_ptr();
        add = !g_mode.overwrite.load(std::memory_order_relaxed);
        if (!add) {
          note_written(pw);
          note_written(pb);
        }
      } else {
        *dw = at::empty(w.sizes(), x.options());
        *db = at::empty(w.sizes(), x.options());
        pw = dw->data_ptr();
        pb = db->data_ptr();
      }
      check(tfb_layernorm_bwd_acc(mchain.p, in, w.data_ptr(), stats, stats + rows, dres, out, pw, pb,
                                  reinterpret_cast<float*>(k[part_at]), ln_partials, rows, d, d, d, d, d, add ? 1 : 0, dtype, st));
    };

    // MLP
    side.mark();
    Epilogue mask;
    mask.mask = s.slab[s.act];
    mask.ld_mask = f;
    gemm(mdy, as_matrix(w2).t(), k[dz_at], f, mask, dtype, dev, st);
    if (need(10)) weight_grad(block(s.slab[s.act], rows, f), mdy, gw2, dtype, dev, side.stream());
    if (need_b2) colsum(mdy, &db2);
    side.mark();
    gemm(mdz, as_matrix(w1).t(), k[chain_at], d, Epilogue{}, dtype, dev, st);
    if (need(9)) weight_grad(block(s.slab[s.normed2], rows, d), mdz, gw1, dtype, dev, side.stream());
    if (need_b1) colsum(mdz, &db1);
    Tensor da2, db2n, da1, db1n;
    norm_backward(s.slab[s.h], ln2_w, ln2_b, s.floats(s.stats2), dy.data_ptr(), k[dh_at], need(7), need(8), &da2, &db2n);

    // attention
    const Mat mdh = block(k[dh_at], rows, d);
    side.mark();
    gemm(mdh, as_matrix(wo).t(), k[chain_at], d, Epilogue{}, dtype, dev, st);
    if (need(6)) weight_grad(block(s.slab[s.ctx], rows, d), mdh, gwo, dtype, dev, side.stream());
    const int64_t es = x.element_size(), hd = shape.hd;
    auto blocks = [&](char* m, int i) { return Heads{m + i * d * es, {t * 3 * d, hd, 3 * d}}; };
    char *qkv = s.slab[s.qkv], *dqkv = k[dqkv_at];
    const Heads o{s.slab[s.ctx], {t * d, hd, d}}, d_o{k[chain_at], {t * d, hd, d}};
    attention_backward(blocks(qkv, 0), blocks(qkv, 1), blocks(qkv, 2), o, d_o, s.floats(s.lse), blocks(dqkv, 0), blocks(dqkv, 1),
                       blocks(dqkv, 2), shape, bias, k[attn_at], scratch_bytes, dtype, st);
    const Mat mdqkv = block(dqkv, rows, 3 * d), mn1 = block(s.slab[s.normed1], rows, d);
    const bool need_dx = need(0) || need(1) || need(2);
    side.mark();
    if (need_dx) {
      Tensor cat;
      const Mat wqkv = wcat.defined() ? as_matrix(wcat) : qkv_matrix(wq, wk, wv, &cat);
      gemm(mdqkv, wqkv.t(), k[chain_at], d, Epilogue{}, dtype, dev, st);
    }
    if (one_product) {
      weight_grad(mn1, mdqkv, gqkv, dtype, dev, side.stream());
    } else if (need(3) || need(4) || need(5)) {
      cudaStream_t ss = side.stream();
      for (int i = 0; i < 3; ++i)
        if (gq[i].p) {
          Mat part = mdqkv;
          part.p = static_cast<const char*>(mdqkv.p) + i * d * es;
          part.cols = d;
          weight_grad(mn1, part, gq[i], dtype, dev, ss);
        }
    }
    if (need_dx)
      norm_backward(x.data_ptr(), ln1_w, ln1_b, s.floats(s.stats1), k[dh_at], dx.data_ptr(), need(1), need(2), &da1, &db1n);
    const bool all_in_place = !(gw1.fresh.defined() || gw2.fresh.defined() || gwo.fresh.defined() || gq[0].fresh.defined() ||
                                gq[1].fresh.defined() || gq[2].fresh.defined());
    for (const Tensor& kept : {dy, s.slab.buf, k.buf}) side.keep(kept);
    side.join(all_in_place && g_mode.defer.load(std::memory_order_relaxed));
    return {need_dx ? dx : Tensor(), da1, db1n, gq[0].fresh, gq[1].fresh, gq[2].fresh, gwo.fresh, da2, db2n, gw1.fresh, gw2.fresh, db1, db2,
            Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor layer(const Tensor& x, const LayerWeights& w, const Bias& bias_, int64_t heads, double eps1, double eps2, Tensor* act) {
  Bias bias = bias_;
  if (bias.table.defined()) {  // the attention reads the table in the type it computes in
    const Amp amp;
    bias.table = bias.table.to(amp.on ? amp.type : x.scalar_type());
  }
  if (needs_node({&x, &w.ln1_w, &w.ln1_b, &w.wq, &w.wk, &w.wv, &w.wo, &w.ln2_w, &w.ln2_b, &w.w1, &w.b1, &w.w2, &w.b2,
                  &bias.slopes, &bias.table}))
    return LayerFn::apply(x, w.ln1_w, w.ln1_b, w.wq, w.wk, w.wv, w.wo, w.ln2_w, w.ln2_b, w.w1, w.w2, opt(w.b1), opt(w.b2), &bias,
                          heads, eps1, eps2, act);
  Amp a;
  BodyGuard guard;
  LayerWeights c{a(w.ln1_w), a(w.ln1_b), a(w.wq), a(w.wk), a(w.wv), a(w.wo), a(w.ln2_w), a(w.ln2_b), a(w.w1), a(w.b1), a(w.w2),
                       a(w.b2)};
  const Tensor xc = a(x).contiguous();
  check_layer(xc, c, heads);
  Saved s(xc.size(0) * xc.size(1), xc.size(2), c.w1.size(1), heads);
  Tensor wcat;
  Tensor y = layer_forward(xc, c, bias, heads, eps1, eps2, s, &wcat);
  if (act) *act = s.activations(xc, c.w1.size(1));
  return y;
}

}  // namespace tfb_host
