// The autograd functions of the native host path (functions.cpp, layer.cpp); module.cpp binds them to Python.
#pragma once
#include <torch/csrc/autograd/custom_function.h>

#include "host.h"

namespace tfb_host {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

inline OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }
inline Tensor val(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

// The bodies run below autograd and outside autocast, whatever the caller's region.
struct BodyGuard {
  at::AutoDispatchBelowAutograd below;
  c10::impl::ExcludeDispatchKeyGuard no_autocast{c10::autocast_dispatch_keyset};
};

// Whether a call needs an autograd node.  Without one the body runs below autograd, where a tangent would be lost and a
// transform's wrapper has no memory, so what the nodes do not implement - forward mode, function transforms - is refused here,
// and so are tensors without data.
bool needs_node(std::initializer_list<const Tensor*> inputs);

// Where a weight gradient goes: into the parameter's existing .grad (added, or written in overwrite mode), when a block of
// linear.accumulate_into_grad is in force and the buffer fits, or into a new tensor that is returned to autograd.
struct GradTarget {
  void* p = nullptr;
  int64_t ld = 0;
  bool in_place = false, add = false;
  Tensor fresh;  // defined unless in_place
};
bool grad_fits(const Tensor& param, at::ScalarType type);  // accumulating, and param.grad is contiguous and of param's shape
GradTarget weight_target(const Tensor& w, at::ScalarType type);
// dW (or dW +=) = X^T dY
void weight_grad(const Mat& x, const Mat& dy, const GradTarget& g, int dtype, c10::Device device, cudaStream_t stream);

// True if the tensors are the column blocks [0, w), [w, 2w), .. of one row-major matrix of `width` columns.
bool adjacent_columns(const Tensor* const* parts, int n, int64_t width);

Tensor linear(const Tensor& x, const Tensor& w, const Tensor& bias, bool relu);
Tensor layernorm(const Tensor& x, const Tensor& alpha, const Tensor& beta, double eps);
Tensor attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& slopes, int64_t rounded, const Tensor& table,
                 bool amp);
Tensor softmax(const Tensor& x);
Tensor cross_entropy(const Tensor& logits, const Tensor& labels, bool f32);
Tensor lm_loss(const Tensor& logits, const Tensor& labels);
Tensor embedding(const Tensor& ids, const Tensor& tok, const Tensor& pos);

struct LayerWeights {
  Tensor ln1_w, ln1_b, wq, wk, wv, wo, ln2_w, ln2_b, w1, b1, w2, b2;
};
// act: where wanted, the hidden activations that the layer keeps (a view of what its node has saved)
Tensor layer(const Tensor& x, const LayerWeights& w, const Bias& bias, int64_t heads, double eps1, double eps2, Tensor* act);

}  // namespace tfb_host
