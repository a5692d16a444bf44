// Operators above the C ABI: checks, allocation and launch (host.h).
#include "host.h"

#include <ATen/autocast_mode.h>

#include <algorithm>
#include <deque>
#include <list>
#include <unordered_set>

namespace tfb_host {

GradMode g_mode;

void check(int rc) {
  if (rc == TFB_OK) return;
  const std::string msg = tfb_last_error();
  if (rc == TFB_ERR_ARG || rc == TFB_ERR_UNSUPPORTED) throw ArgumentError(msg);
  throw std::runtime_error("tritonformer_b200 (" + std::to_string(rc) + "): " + msg);
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return TFB_F16;
    case at::kBFloat16: return TFB_BF16;
    case at::kFloat: return TFB_F32;
    default: throw ArgumentError(std::string("unsupported dtype ") + c10::toString(t));
  }
}

Amp::Amp() {
  on = at::autocast::is_autocast_enabled(at::kCUDA);
  type = on && at::autocast::get_autocast_dtype(at::kCUDA) == at::kBFloat16 ? at::kBFloat16 : at::kHalf;
}

Tensor Amp::operator()(const Tensor& t) const {
  if (!on || !t.defined() || !t.is_cuda() || !t.is_floating_point() || t.scalar_type() == at::kDouble ||
      t.scalar_type() == type)
    return t;
  return t.to(type);
}

// ------------------------------------------------------------------------------------------ written gradients
static std::mutex g_written_lock;
static std::unordered_set<uintptr_t>& written_set() {
  static auto* s = new std::unordered_set<uintptr_t>();
  return *s;
}
void note_written(const void* p) {
  std::lock_guard<std::mutex> g(g_written_lock);
  written_set().insert(reinterpret_cast<uintptr_t>(p));
}
std::vector<uintptr_t> take_written() {
  std::lock_guard<std::mutex> g(g_written_lock);
  std::vector<uintptr_t> out(written_set().begin(), written_set().end());
  written_set().clear();
  return out;
}

// ------------------------------------------------------------------------------------------------ workspaces
// Newest last; at most kMaxWorkspaces per process.  An entry that falls out goes back to the caching allocator, which
// hands it out again only in the order of the stream it was allocated on, so kernels still in flight keep it.
struct Workspace {
  c10::DeviceIndex device;
  cudaStream_t stream;
  Tensor buf;
};
constexpr size_t kMaxWorkspaces = 8;
static std::mutex g_ws_lock;
static std::list<Workspace>& workspaces() {
  static auto* l = new std::list<Workspace>();  // never destroyed: the CUDA context may be gone by then
  return *l;
}

Tensor gemm_workspace(c10::Device device, cudaStream_t stream) {
  std::lock_guard<std::mutex> g(g_ws_lock);
  auto& l = workspaces();
  for (auto it = l.rbegin(); it != l.rend(); ++it) {
    if (it->stream != stream || it->device != device.index()) continue;
    if (it != l.rbegin()) l.splice(l.end(), l, std::prev(it.base()));
    return l.back().buf;
  }
  // allocated and cleared in the order of the stream that uses it
  c10::cuda::CUDAStreamGuard on(c10::cuda::getStreamFromExternal(stream, device.index()));
  Tensor buf = at::zeros({tfb_gemm_workspace_bytes()}, at::TensorOptions().device(device).dtype(at::kByte));
  l.push_back({device.index(), stream, buf});
  if (l.size() > kMaxWorkspaces) l.pop_front();
  return buf;
}

void reset_workspaces() {
  std::lock_guard<std::mutex> g(g_ws_lock);
  for (auto& w : workspaces()) w.buf.zero_();
}

// --------------------------------------------------------------------------------------------------- side work
constexpr int kDeferred = 2;  // backward functions a deferred weight gradient may lag behind
struct Pending {
  cudaEvent_t done;
  std::vector<Tensor> kept;
};
struct SideStream {
  c10::cuda::CUDAStream main, side;
  cudaEvent_t mark;
  std::vector<cudaEvent_t> free_events;
  std::deque<Pending> pending;
};
static std::mutex g_side_lock;
static std::list<SideStream>& side_streams() {
  static auto* l = new std::list<SideStream>();
  return *l;
}
static cudaEvent_t new_event() {
  cudaEvent_t e;
  TORCH_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess, "cudaEventCreate failed");
  return e;
}
static void order(cudaStream_t after, cudaStream_t before, cudaEvent_t e) {
  cudaEventRecord(e, before);
  cudaStreamWaitEvent(after, e, 0);
}
static SideStream& side_of(const c10::cuda::CUDAStream& main) {  // lock held
  for (auto& s : side_streams())
    if (s.main == main) return s;
  side_streams().push_back({main, c10::cuda::getStreamFromPool(false, main.device_index()), new_event(), {}, {}});
  return side_streams().back();
}
static void retire_oldest(SideStream& s) {  // lock held
  cudaStreamWaitEvent(s.main.stream(), s.pending.front().done, 0);
  s.free_events.push_back(s.pending.front().done);
  s.pending.pop_front();
}

SideWork::SideWork(const Tensor& like, bool enabled)
    : on_(enabled), main_(c10::cuda::getCurrentCUDAStream(like.device().index())), side_(main_) {
  if (on_) {
    std::lock_guard<std::mutex> g(g_side_lock);
    side_ = side_of(main_).side;
  }
}
SideWork::~SideWork() {
  if (on_ && used_) {  // an exception left the function early
    std::lock_guard<std::mutex> g(g_side_lock);
    order(main_.stream(), side_.stream(), side_of(main_).mark);
  }
}
void SideWork::mark() {
  if (!on_) return;
  std::lock_guard<std::mutex> g(g_side_lock);
  cudaEventRecord(side_of(main_).mark, main_.stream());
}
cudaStream_t SideWork::stream() {
  if (!on_) return main_.stream();
  std::lock_guard<std::mutex> g(g_side_lock);
  cudaStreamWaitEvent(side_.stream(), side_of(main_).mark, 0);
  used_ = true;
  return side_.stream();
}
void SideWork::join(bool may_defer) {
  if (!on_ || !used_) return;
  std::lock_guard<std::mutex> g(g_side_lock);
  SideStream& s = side_of(main_);
  used_ = false;
  if (!may_defer) {
    order(main_.stream(), side_.stream(), s.mark);
    kept_.clear();
    return;
  }
  cudaEvent_t e;
  if (s.free_events.empty()) e = new_event();
  else { e = s.free_events.back(); s.free_events.pop_back(); }
  cudaEventRecord(e, side_.stream());
  s.pending.push_back({e, std::move(kept_)});
  kept_.clear();
  while (s.pending.size() > kDeferred) retire_oldest(s);
}
void join_all() {
  std::lock_guard<std::mutex> g(g_side_lock);
  for (auto& s : side_streams())
    while (!s.pending.empty()) retire_oldest(s);
}

// ---------------------------------------------------------------------------------------------------- matrices
Mat as_rows(const Tensor& x) {
  const int64_t d = x.size(-1);
  Mat m;
  m.cols = d;
  m.rows = d ? x.numel() / d : 0;
  if (x.is_contiguous()) {
    m.s0 = d;
    m.s1 = 1;
    m.p = x.data_ptr();
    m.keep = x;
    return m;
  }
  Tensor x2 = x.reshape({-1, d});
  if (x2.stride(1) != 1 && x2.stride(0) != 1) x2 = x2.contiguous();
  m.s0 = x2.stride(0);
  m.s1 = x2.stride(1);
  m.p = x2.data_ptr();
  m.keep = x2;
  return m;
}

Mat as_matrix(const Tensor& w) {
  Tensor c = w.stride(0) != 1 && w.stride(1) != 1 ? w.contiguous() : w;
  Mat m;
  m.p = c.data_ptr();
  m.rows = c.size(0);
  m.cols = c.size(1);
  m.s0 = c.stride(0);
  m.s1 = c.stride(1);
  m.keep = c;
  return m;
}

Mat block(const void* p, int64_t rows, int64_t cols) {
  Mat m;
  m.p = p;
  m.rows = rows;
  m.cols = cols;
  m.s0 = cols;
  m.s1 = 1;
  return m;
}

bool tma_fits(const Mat& m) {
  const int64_t outer = m.s1 == 1 ? m.s0 : m.s1;
  return (reinterpret_cast<uintptr_t>(m.p) & 15) == 0 && outer > 0 && outer % 8 == 0;
}

Mat grad_rows(const Mat& dy_, const Tensor& act, Tensor* sums, const Tensor& like, int dtype) {
  Mat dy = dy_;
  if (dy.s1 != 1) {  // a transposed gradient
    Tensor c = dy.keep.contiguous();
    dy = block(c.data_ptr(), dy.rows, dy.cols);
    dy.keep = c;
  }
  const int64_t ld = (dy.cols + 7) / 8 * 8;
  const Mat a = act.defined() ? as_rows(act) : Mat{};
  Tensor out = at::empty({dy.rows, ld}, like.options()), partials;
  int64_t n = 0;
  if (sums) {
    n = tfb_colsum_partials(dy.rows, dy.cols);
    partials = at::empty({n, dy.cols}, like.options().dtype(at::kFloat));
    *sums = at::empty({dy.cols}, like.options());
  }
  check(tfb_grad_rows(dy.p, a.p, out.data_ptr(), sums ? sums->data_ptr() : nullptr,
                      sums ? static_cast<float*>(partials.data_ptr()) : nullptr, n, dy.rows, dy.cols,
                      dy.rows > 1 ? dy.s0 : dy.cols, a.p ? a.s0 : 0, ld, dtype, current_stream(like)));
  Mat m;
  m.keep = m.packed = out;
  m.p = out.data_ptr();
  m.rows = dy.rows;
  m.cols = dy.cols;
  m.s0 = ld;
  m.s1 = 1;
  return m;
}

Mat tma_fit(const Mat& m, const Tensor& like, int dtype) {
  if (tma_fits(m) || m.rows == 0 || m.cols == 0) return m;
  if (m.s1 == 1) return grad_rows(m, Tensor(), nullptr, like, dtype);
  return grad_rows(m.t(), Tensor(), nullptr, like, dtype).t();
}

void gemm(const Mat& a, const Mat& b, void* out, int64_t ldc, const Epilogue& e, int dtype, c10::Device device,
          cudaStream_t stream) {
  Tensor ws = gemm_workspace(device, stream);
  check(tfb_gemm_fused(a.p, b.p, out, e.bias, e.addend, e.ld_addend, e.mask, e.ld_mask, a.rows, b.cols, a.cols, a.s0, a.s1,
                       b.s0, b.s1, ldc, e.relu ? 1 : 0, dtype, ws.data_ptr(), ws.numel(), stream, nullptr));
}

// --------------------------------------------------------------------------------------------------- LayerNorm
static Mat ln_rows(const Tensor& t) {
  Mat m = as_rows(t);
  if (m.s1 != 1 || (m.rows > 1 && m.s0 < m.cols)) {
    Tensor c = m.keep.reshape({-1, t.size(-1)}).contiguous();
    m.keep = c;
    m.p = c.data_ptr();
    m.s0 = m.cols;
    m.s1 = 1;
  }
  if (m.rows <= 1) m.s0 = m.cols;
  return m;
}

std::tuple<Tensor, Tensor> layernorm_forward(const Tensor& x, const Tensor& alpha, const Tensor& beta, double eps) {
  TFB_ASSERT(x.is_cuda() && (x.scalar_type() == at::kHalf || x.scalar_type() == at::kBFloat16),
             "LayerNorm expects a CUDA fp16/bf16 input");
  TFB_ASSERT(alpha.scalar_type() == x.scalar_type() && beta.scalar_type() == x.scalar_type(),
             "LayerNorm parameters must match the input dtype");
  const int64_t d = x.size(-1);
  TFB_ASSERT(alpha.numel() == d && beta.numel() == d, "LayerNorm parameter size mismatch");
  Mat m = ln_rows(x);
  Tensor y = at::empty(x.sizes(), x.options());
  Tensor stats = at::empty({2, m.rows}, x.options().dtype(at::kFloat));
  float* s = static_cast<float*>(stats.data_ptr());
  Tensor ac = alpha.contiguous(), bc = beta.contiguous();
  check(tfb_layernorm_fwd(m.p, ac.data_ptr(), bc.data_ptr(), y.data_ptr(), s, s + m.rows, m.rows, d, m.s0, d, (float)eps,
                          dtype_code(x.scalar_type()), current_stream(x)));
  return {y, stats};
}

Tensor layernorm_backward(const Tensor& dy, const Tensor& x, const Tensor& alpha, const Tensor& stats, const Tensor& dres,
                          void* dalpha, void* dbeta, bool add) {
  const int64_t d = x.size(-1);
  Mat mx = ln_rows(x), my = ln_rows(dy), mr;
  if (dres.defined()) mr = ln_rows(dres);
  const int64_t rows = mx.rows;
  Tensor dx = at::empty(x.sizes(), x.options());
  const int64_t n = tfb_layernorm_bwd_partials(rows, d);
  Tensor partials = at::empty({n, 2, d}, x.options().dtype(at::kFloat));
  Tensor ac = alpha.contiguous();
  const float* s = static_cast<const float*>(stats.data_ptr());
  check(tfb_layernorm_bwd_acc(my.p, mx.p, ac.data_ptr(), s, s + rows, mr.p, dx.data_ptr(), dalpha, dbeta,
                              static_cast<float*>(partials.data_ptr()), n, rows, d, my.s0, mx.s0, mr.p ? mr.s0 : 0, d,
                              add ? 1 : 0, dtype_code(x.scalar_type()), current_stream(x)));
  return dx;
}

// ------------------------------------------------------------------------------------------ bias and ReLU gradients
Tensor column_sum(const Tensor& x) {
  Mat m = as_rows(x);
  if (m.s1 != 1) {
    Tensor c = m.keep.contiguous();
    m = block(c.data_ptr(), m.rows, m.cols);
    m.keep = c;
  }
  Tensor out = at::empty({m.cols}, x.options());
  const int64_t n = tfb_colsum_partials(m.rows, m.cols);
  Tensor partials = at::empty({n, m.cols}, x.options().dtype(at::kFloat));
  check(tfb_colsum(m.p, out.data_ptr(), static_cast<float*>(partials.data_ptr()), n, m.rows, m.cols,
                   m.rows > 1 ? m.s0 : m.cols, dtype_code(x.scalar_type()), current_stream(x)));
  return out;
}

// --------------------------------------------------------------------------------------------------- attention
void check_attention(const AttnShape& s, at::ScalarType type) {
  TFB_ASSERT(type == at::kHalf || type == at::kBFloat16, "attention expects matching fp16/bf16 inputs");
  TFB_ASSERT(s.hd == 32 || s.hd == 64 || s.hd == 128, "Only head_dims of [32,64,128] are supported.");
  TFB_ASSERT(s.t % 64 == 0, "Number of elements in sequence must be a multiple of 64");
}

void attention_forward(const Heads& q, const Heads& k, const Heads& v, const Heads& o, float* lse, const AttnShape& s,
                       const Bias& bias, int dtype, cudaStream_t stream) {
  const bool tab = bias.table.defined();
  check(tfb_attention_fwd(q.p, k.p, v.p, o.p, lse, s.b, s.h, s.t, s.hd, q.s, k.s, v.s, o.s,
                          bias.slopes.defined() ? static_cast<const float*>(bias.slopes.data_ptr()) : nullptr, bias.rounded,
                          tab ? bias.table.data_ptr() : nullptr, tab ? bias.table.stride(0) : 0, tab ? bias.table.stride(1) : 0,
                          dtype, stream, nullptr));
}

void attention_backward(const Heads& q, const Heads& k, const Heads& v, const Heads& o, const Heads& d_o, const float* lse,
                        const Heads& dq, const Heads& dk, const Heads& dv, const AttnShape& s, const Bias& bias,
                        void* scratch, int64_t scratch_bytes, int dtype, cudaStream_t stream) {
  const bool tab = bias.table.defined();
  check(tfb_attention_bwd(q.p, k.p, v.p, o.p, d_o.p, lse, dq.p, dk.p, dv.p, s.b, s.h, s.t, s.hd, q.s, k.s, v.s, o.s, d_o.s, dq.s,
                          dk.s, dv.s, bias.slopes.defined() ? static_cast<const float*>(bias.slopes.data_ptr()) : nullptr,
                          bias.rounded, tab ? bias.table.data_ptr() : nullptr, tab ? bias.table.stride(0) : 0,
                          tab ? bias.table.stride(1) : 0, scratch, scratch_bytes, dtype, stream, nullptr));
}

}  // namespace tfb_host
