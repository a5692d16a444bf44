// Python binding of the native host path: plain CPython calls on positional arguments, the interpreter lock released
// while kernels are enqueued (the backward pass runs on another thread).
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include "functions.h"

namespace {

using namespace tfb_host;

// Positional arguments of one call; None stands for an absent tensor.
class Args {
 public:
  Args(PyObject* const* a, Py_ssize_t n, Py_ssize_t want, const char* name) : a_(a) {
    if (n != want) throw ArgumentError(std::string(name) + ": wrong number of arguments");
  }
  const Tensor& tensor() {
    PyObject* o = a_[i_++];
    if (o == Py_None) return none_;
    if (!THPVariable_Check(o)) throw ArgumentError("expected a tensor");
    return THPVariable_Unpack(o);
  }
  int64_t integer() {
    const long long v = PyLong_AsLongLong(a_[i_++]);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
  }
  double real() {
    const double v = PyFloat_AsDouble(a_[i_++]);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
  }
  bool truth() {
    const int v = PyObject_IsTrue(a_[i_++]);
    if (v < 0) throw python_error();
    return v != 0;
  }
 private:
  PyObject* const* a_;
  Py_ssize_t i_ = 0;
  Tensor none_;
};

template <typename F>
PyObject* guarded(F body) {
  HANDLE_TH_ERRORS
  return body();
  END_HANDLE_TH_ERRORS
}

template <typename F>
PyObject* tensor_result(F body) {
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = body();
  }
  return THPVariable_Wrap(out);
}

#define TFB_PY(name) PyObject* name(PyObject* self, PyObject* const* argv, Py_ssize_t argc)

PyObject* g_recorder = nullptr;  // what an operator's call goes to while torch.jit.trace records (_trace.py)

// An operator: the call itself, or while a trace is being recorded recorder(operator, *arguments).
template <typename F>
PyObject* traceable(PyObject* self, const char* name, PyObject* const* argv, Py_ssize_t argc, F body) {
  if (C10_LIKELY(!torch::jit::tracer::isTracing() || !g_recorder)) return guarded(body);
  PyObject* args = PyTuple_New(argc + 1);
  if (!args) return nullptr;
  PyObject* op = PyObject_GetAttrString(self, name);
  PyObject* out = nullptr;
  if (op) {
    PyTuple_SET_ITEM(args, 0, op);
    for (Py_ssize_t i = 0; i < argc; ++i) {
      Py_INCREF(argv[i]);
      PyTuple_SET_ITEM(args, i + 1, argv[i]);
    }
    out = PyObject_Call(g_recorder, args, nullptr);
  }
  Py_DECREF(args);
  return out;
}

TFB_PY(py_linear) {
  return traceable(self, "linear", argv, argc, [&] {
    Args a(argv, argc, 4, "linear");
    const Tensor &x = a.tensor(), &w = a.tensor(), &b = a.tensor();
    const bool relu = a.truth();
    return tensor_result([&] { return linear(x, w, b, relu); });
  });
}
TFB_PY(py_layernorm) {
  return traceable(self, "layernorm", argv, argc, [&] {
    Args a(argv, argc, 4, "layernorm");
    const Tensor &x = a.tensor(), &w = a.tensor(), &b = a.tensor();
    const double eps = a.real();
    return tensor_result([&] { return layernorm(x, w, b, eps); });
  });
}
TFB_PY(py_attention) {  // q, k, v, slopes, rounded, table, amp
  return traceable(self, "attention", argv, argc, [&] {
    Args a(argv, argc, 7, "attention");
    const Tensor &q = a.tensor(), &k = a.tensor(), &v = a.tensor(), &slopes = a.tensor();
    const int64_t rounded = a.integer();
    const Tensor& table = a.tensor();
    const bool amp = a.truth();
    return tensor_result([&] { return attention(q, k, v, slopes, rounded, table, amp); });
  });
}
TFB_PY(py_softmax) {
  return traceable(self, "softmax", argv, argc, [&] {
    Args a(argv, argc, 1, "softmax");
    const Tensor& x = a.tensor();
    return tensor_result([&] { return softmax(x); });
  });
}
TFB_PY(py_cross_entropy) {  // logits, labels, fp32 losses
  return traceable(self, "cross_entropy", argv, argc, [&] {
    Args a(argv, argc, 3, "cross_entropy");
    const Tensor &x = a.tensor(), &y = a.tensor();
    const bool f32 = a.truth();
    return tensor_result([&] { return cross_entropy(x, y, f32); });
  });
}
TFB_PY(py_lm_loss) {
  return traceable(self, "lm_loss", argv, argc, [&] {
    Args a(argv, argc, 2, "lm_loss");
    const Tensor &x = a.tensor(), &y = a.tensor();
    return tensor_result([&] { return lm_loss(x, y); });
  });
}
TFB_PY(py_embedding) {
  return traceable(self, "embedding", argv, argc, [&] {
    Args a(argv, argc, 3, "embedding");
    const Tensor &ids = a.tensor(), &tok = a.tensor(), &pos = a.tensor();
    return tensor_result([&] { return embedding(ids, tok, pos); });
  });
}
// x, ln1_w, ln1_b, wq, wk, wv, wo, ln2_w, ln2_b, w1, b1, w2, b2, slopes, rounded, table, heads, eps1, eps2
PyObject* layer_call(PyObject* const* argv, Py_ssize_t argc, Tensor* act) {
  Args a(argv, argc, 19, "layer");
  const Tensor& x = a.tensor();
  LayerWeights w;
  for (Tensor* t : {&w.ln1_w, &w.ln1_b, &w.wq, &w.wk, &w.wv, &w.wo, &w.ln2_w, &w.ln2_b, &w.w1, &w.b1, &w.w2, &w.b2})
    *t = a.tensor();
  Bias bias;
  bias.slopes = a.tensor();
  bias.rounded = (int)a.integer();
  bias.table = a.tensor();
  const int64_t heads = a.integer();
  const double eps1 = a.real(), eps2 = a.real();
  return tensor_result([&] { return layer(x, w, bias, heads, eps1, eps2, act); });
}
TFB_PY(py_layer) {
  return traceable(self, "layer", argv, argc, [&] { return layer_call(argv, argc, nullptr); });
}
TFB_PY(py_layer_and_activations) {  // (output, hidden activations): what the model's tests look at
  return guarded([&]() -> PyObject* {
    Tensor act;
    PyObject* y = layer_call(argv, argc, &act);
    return Py_BuildValue("(NN)", y, THPVariable_Wrap(act));
  });
}
TFB_PY(py_set_grad_mode) {  // accumulating, overwrite, defer, fork
  return guarded([&]() -> PyObject* {
    Args a(argv, argc, 4, "set_grad_mode");
    g_mode.accumulating = a.truth();
    g_mode.overwrite = a.truth();
    g_mode.defer = a.truth();
    g_mode.fork = a.truth();
    Py_RETURN_NONE;
  });
}
TFB_PY(py_take_written) {
  return guarded([&]() -> PyObject* {
    const std::vector<uintptr_t> v = take_written();
    PyObject* list = PyList_New((Py_ssize_t)v.size());
    if (!list) throw python_error();
    for (size_t i = 0; i < v.size(); ++i) PyList_SET_ITEM(list, (Py_ssize_t)i, PyLong_FromUnsignedLongLong(v[i]));
    return list;
  });
}
TFB_PY(py_join_weight_grads) {
  return guarded([&]() -> PyObject* {
    join_all();
    Py_RETURN_NONE;
  });
}
TFB_PY(py_gemm_workspace) {  // device index, stream handle
  return guarded([&] {
    Args a(argv, argc, 2, "gemm_workspace");
    const int64_t dev = a.integer(), stream = a.integer();
    return tensor_result([&] {
      return gemm_workspace(c10::Device(c10::kCUDA, (c10::DeviceIndex)dev), reinterpret_cast<cudaStream_t>(stream));
    });
  });
}
TFB_PY(py_set_recorder) {
  return guarded([&]() -> PyObject* {
    if (argc != 1) throw ArgumentError("set_recorder: wrong number of arguments");
    Py_INCREF(argv[0]);
    Py_XDECREF(std::exchange(g_recorder, argv[0]));
    Py_RETURN_NONE;
  });
}
TFB_PY(py_reset_workspaces) {
  return guarded([&]() -> PyObject* {
    reset_workspaces();
    Py_RETURN_NONE;
  });
}

#define TFB_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {TFB_METHOD(linear), TFB_METHOD(layernorm), TFB_METHOD(attention), TFB_METHOD(softmax),
                         TFB_METHOD(cross_entropy), TFB_METHOD(lm_loss), TFB_METHOD(embedding), TFB_METHOD(layer),
                         TFB_METHOD(layer_and_activations),
                         TFB_METHOD(set_grad_mode), TFB_METHOD(take_written), TFB_METHOD(join_weight_grads),
                         TFB_METHOD(gemm_workspace), TFB_METHOD(reset_workspaces), TFB_METHOD(set_recorder), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host path of tritonformer_b200.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
