// Native host path: allocation, launch and autograd bookkeeping of the operators above the C ABI.
//
// The kernels are a few microseconds to a few hundred long; driving each of them from a Python autograd Function
// (argument checks, three to six tensor allocations, a 20-argument foreign call, the context object) took 40-60 us,
// so that every step but the largest was bound by the interpreter.  Here one call from Python runs a whole operator,
// or a whole transformer layer, and the backward pass runs on the autograd engine's thread without the interpreter.
#pragma once
#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>

#include <atomic>
#include <mutex>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "../../../include/tritonformer_b200.h"

namespace tfb_host {

using at::Tensor;

// Raised for a bad argument; becomes an AssertionError in Python, like the reference's asserts, also where a backward raises it
// on a thread of the autograd engine (which hands the exception on and knows this base class).
struct ArgumentError : torch::PyTorchError {
  using torch::PyTorchError::PyTorchError;
  PyObject* python_type() override { return PyExc_AssertionError; }
};
#define TFB_ASSERT(cond, msg) \
  do {                        \
    if (!(cond)) throw ::tfb_host::ArgumentError(msg); \
  } while (0)

void check(int rc);  // status of a C ABI call -> exception

// ---- autocast ------------------------------------------------------------------------------------------------
// What an operator does inside an autocast region: floating CUDA tensors (but fp64) are cast to the region's
// 16-bit type and the body runs with autocast off.
struct Amp {
  bool on;
  at::ScalarType type;
  Amp();
  Tensor operator()(const Tensor& t) const;
};

// ---- how gradients are delivered (set by linear.accumulate_into_grad) ----------------------------------------------
struct GradMode {
  std::atomic<bool> accumulating{false}, overwrite{false}, defer{false}, fork{true};
};
extern GradMode g_mode;
void note_written(const void* p);
std::vector<uintptr_t> take_written();

// ---- streams and scratch -------------------------------------------------------------------------------------
inline cudaStream_t current_stream(const Tensor& t) {
  return c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
}
// Scratch of the GEMM, one per device and stream, cleared once (the kernels keep its counters zero).
Tensor gemm_workspace(c10::Device device, cudaStream_t stream);
void reset_workspaces();

// Weight-gradient products run on a side stream beside the products of the gradient chain.  One object per backward
// function: mark() before the kernels that the side work does not depend on (the chain's next product, which is launched
// first and takes its SMs first), stream() for the side stream, made to wait for that mark, join() the other way round.
// With deferred joins (accumulate_into_grad(defer_weight_grads=True)) the compute stream waits for the weight gradients of a
// function only kDeferred functions later (or at join_all), and their operands are kept alive until then, so that the
// allocator cannot hand them out again under the side kernels.
class SideWork {
 public:
  SideWork(const Tensor& like, bool enabled);
  ~SideWork();
  bool on() const { return on_; }
  cudaStream_t main() const { return main_.stream(); }
  void mark();
  cudaStream_t stream();  // the stream to launch the side work on (the compute stream if off)
  void keep(const Tensor& t) { if (on_) kept_.push_back(t); }
  void join(bool may_defer);
 private:
  bool on_, used_ = false;
  c10::cuda::CUDAStream main_, side_;
  std::vector<Tensor> kept_;
};
void join_all();

// ---- operators without autograd --------------------------------------------------------------------------------
int dtype_code(at::ScalarType t);

// A matrix of 16-bit values with element strides; `keep` owns the memory where a copy was needed.
struct Mat {
  Tensor keep;
  Tensor packed;  // keep, where tma_fit made a copy
  const void* p = nullptr;
  int64_t rows = 0, cols = 0, s0 = 0, s1 = 0;
  Mat t() const { return Mat{keep, packed, p, cols, rows, s1, s0}; }
};
Mat as_rows(const Tensor& x);                        // (.., d) -> (rows, d), one of the strides 1
Mat as_matrix(const Tensor& w);                      // a 2-D weight, one of the strides 1
Mat block(const void* p, int64_t rows, int64_t cols);  // contiguous

// Whether the GEMM can read the matrix through TMA (16-byte aligned rows); tma_fit copies one that it cannot into rows
// padded to a multiple of 16 bytes - a pass over the operand, against a kernel that runs at a twentieth of the rate.
bool tma_fits(const Mat& m);
Mat tma_fit(const Mat& m, const Tensor& like, int dtype);
// dz = act > 0 ? dy : 0 (act undefined: dy) in aligned rows; sums: its column sums, unless null
Mat grad_rows(const Mat& dy, const Tensor& act, Tensor* sums, const Tensor& like, int dtype);

struct Epilogue {
  const void* bias = nullptr;
  bool relu = false;
  const void* addend = nullptr;
  int64_t ld_addend = 0;
  const void* mask = nullptr;
  int64_t ld_mask = 0;
};
// out (row-major, leading dimension ldc) = epilogue(A B)
void gemm(const Mat& a, const Mat& b, void* out, int64_t ldc, const Epilogue& e, int dtype, c10::Device device,
          cudaStream_t stream);

std::tuple<Tensor, Tensor> layernorm_forward(const Tensor& x, const Tensor& alpha, const Tensor& beta, double eps);
// dalpha / dbeta: buffers to write, or with `add` to add to.  Returns dx.
Tensor layernorm_backward(const Tensor& dy, const Tensor& x, const Tensor& alpha, const Tensor& stats, const Tensor& dres,
                          void* dalpha, void* dbeta, bool add);
Tensor column_sum(const Tensor& x);

struct Bias {  // resolved form of the attention bias
  Tensor slopes;
  int rounded = 0;
  Tensor table;
};
struct Heads {  // (B, H, T, hd) with {b, h, t} strides, unit inner stride
  void* p;
  int64_t s[3];
};
struct AttnShape {
  int64_t b, h, t, hd;
};
void check_attention(const AttnShape& s, at::ScalarType type);
void attention_forward(const Heads& q, const Heads& k, const Heads& v, const Heads& o, float* lse, const AttnShape& s,
                       const Bias& bias, int dtype, cudaStream_t stream);
void attention_backward(const Heads& q, const Heads& k, const Heads& v, const Heads& o, const Heads& d_o, const float* lse,
                        const Heads& dq, const Heads& dk, const Heads& dv, const AttnShape& s, const Bias& bias,
                        void* scratch, int64_t scratch_bytes, int dtype, cudaStream_t stream);

}  // namespace tfb_host
