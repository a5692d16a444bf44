// Fused softmax cross-entropy forward / backward for sm_100a (HBM-bound).
//
// Forward reads each logit once: every thread keeps an online (max, sum) pair in the
// log2 domain over 128-bit chunks of its row, the CTA merges the pairs, and only the
// per-row loss and log-sum-exp leave the chip.  Backward reads the logits and the saved
// log-sum-exp and writes (softmax - onehot) * grad in one pass.
#include "common.cuh"

namespace tfb {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr int CE_THREADS = 256;

__device__ __forceinline__ void online_merge(float& m, float& s, float m2, float s2) {
  const float mm = fmaxf(m, m2);
  // (-inf) - (-inf) would be NaN: an empty partner contributes nothing.
  const float a = (m == -INFINITY) ? 0.f : s * exp2f(m - mm);
  const float b = (m2 == -INFINITY) ? 0.f : s2 * exp2f(m2 - mm);
  m = mm;
  s = a + b;
}

// Label of a row: labels[row], or with shift_seq > 0 (rows = sequences of that length) the label of the next position
// of the same sequence; the last position of a sequence has none.
__device__ __forceinline__ int64_t label_of(const int64_t* __restrict__ labels, int64_t row, int64_t shift_seq) {
  if (shift_seq == 0) return labels[row];
  return (row + 1) % shift_seq == 0 ? -1 : labels[row + 1];
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(CE_THREADS) ce_fwd_kernel(
    const T* __restrict__ logits, const int64_t* __restrict__ labels, T* __restrict__ loss,
    float* __restrict__ loss_f32, float* __restrict__ lse, int vocab, int64_t ld, int64_t shift_seq) {
  grid_dependency_wait();
  allow_dependents();
  __shared__ float sm_m[CE_THREADS / 32], sm_s[CE_THREADS / 32];
  const int64_t row = blockIdx.x;
  const T* xr = logits + row * ld;
  float m = -INFINITY, s = 0.f;  // log2 domain: sum of 2^(x*log2e - m)
  if (VEC) {
    const int nvec = vocab >> 3;
    for (int c = threadIdx.x; c < nvec; c += CE_THREADS) {
      float f[8];
      unpack8<T>(ld_stream16(xr + (int64_t)c * 8), f);
      float vm = f[0];
#pragma unroll
      for (int j = 1; j < 8; ++j) vm = fmaxf(vm, f[j]);
      vm *= kLog2e;
      if (vm > m) {
        s *= exp2f(m - vm);  // m == -inf gives 0 * 0
        m = vm;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s += exp2f(fmaf(f[j], kLog2e, -m));
    }
  } else {  // rows of any alignment (a vocabulary that is no multiple of 8): vectors at the row's own boundaries
    const int shift = chunk_shift(xr), chunks = chunk_count<T>(shift, vocab);
    for (int c = threadIdx.x; c < chunks; c += CE_THREADS) {
      const Chunk k = chunk_at<T>(c, shift, vocab);
      const int n = k.last - k.first;
      float f[8];
      unpack8<T>(load8_any(xr + k.first, n), f);
      float vm = -INFINITY;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j >= n) f[j] = -INFINITY;
        vm = fmaxf(vm, f[j]);
      }
      vm *= kLog2e;
      if (vm > m) {
        s *= exp2f(m - vm);
        m = vm;
      }
      if (m != -INFINITY) {
#pragma unroll
        for (int j = 0; j < 8; ++j) s += exp2f(fmaf(f[j], kLog2e, -m));
      } else {  // nothing but -inf so far, or NaN, which fmaxf passes over: a NaN sum under a finite maximum outlives the merges
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (f[j] != f[j]) {
            m = 0.f;
            s = f[j];
          }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
    const float s2 = __shfl_xor_sync(0xffffffffu, s, o);
    online_merge(m, s, m2, s2);
  }
  if ((threadIdx.x & 31) == 0) {
    sm_m[threadIdx.x >> 5] = m;
    sm_s[threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    m = sm_m[0];
    s = sm_s[0];
    for (int w = 1; w < CE_THREADS / 32; ++w) online_merge(m, s, sm_m[w], sm_s[w]);
    const float l = (m + log2f(s)) * kLn2;
    lse[row] = l;
    const int64_t lab = label_of(labels, row, shift_seq);
    float v = 0.f;
    if (lab >= 0 && lab < vocab) v = l - Num<T>::to_f(xr[lab]);
    if (loss) loss[row] = Num<T>::from_f(v);
    if (loss_f32) loss_f32[row] = v;
  }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(CE_THREADS) ce_bwd_kernel(
    const T* __restrict__ logits, const int64_t* __restrict__ labels, const float* __restrict__ lse,
    const T* __restrict__ grad, int64_t grad_stride, const float* __restrict__ grad_all, float grad_scale,
    T* __restrict__ dlogits, int vocab, int64_t ld, int64_t dld, int64_t shift_seq) {
  grid_dependency_wait();
  allow_dependents();
  const int64_t row = blockIdx.x;
  const T* xr = logits + row * ld;
  T* dr = dlogits + row * dld;
  const int64_t lab64 = label_of(labels, row, shift_seq);
  const bool valid = lab64 >= 0 && lab64 < vocab;
  const int lab = valid ? (int)lab64 : -1;
  // one fp32 gradient for every row (of their mean), or the rows' own
  const float g = !valid ? 0.f : grad_all ? *grad_all * grad_scale : Num<T>::to_f(grad[row * grad_stride]);
  const float l2 = lse[row] * kLog2e;
  if (VEC) {
    const int nvec = vocab >> 3;
    for (int c = threadIdx.x; c < nvec; c += CE_THREADS) {
      float f[8];
      unpack8<T>(ld_stream16(xr + (int64_t)c * 8), f);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = exp2f(fmaf(f[j], kLog2e, -l2));
      const int k = lab - c * 8;
      if (k >= 0 && k < 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j == k) f[j] -= 1.f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] *= g;
      st_stream16(dr + (int64_t)c * 8, pack8<T>(f));
    }
  } else {
    const int shift = chunk_shift(dr), chunks = chunk_count<T>(shift, vocab);
    for (int c = threadIdx.x; c < chunks; c += CE_THREADS) {
      const Chunk k = chunk_at<T>(c, shift, vocab);
      float f[8];
      unpack8<T>(load8_any(xr + k.first, k.last - k.first), f);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = (exp2f(fmaf(f[j], kLog2e, -l2)) - (k.first + j == lab ? 1.f : 0.f)) * g;
      store_chunk(dr, k, f);
    }
  }
}

// out[0] = sum of n row losses / count, in a fixed order.
constexpr int CE_SUM_THREADS = 1024;
__global__ void __launch_bounds__(CE_SUM_THREADS) ce_mean_kernel(const float* __restrict__ loss, float* __restrict__ out,
                                                                 int64_t n, float count) {
  grid_dependency_wait();
  allow_dependents();
  __shared__ float part[CE_SUM_THREADS / 32];
  float s = 0.f;
  for (int64_t i = threadIdx.x; i < n; i += CE_SUM_THREADS) s += loss[i];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = warp_sum(part[threadIdx.x]);
    if (threadIdx.x == 0) *out = s / count;
  }
}

template <typename T>
static int launch_ce_fwd(const void* logits, const int64_t* labels, void* loss, float* loss_f32, float* lse, int64_t rows,
                         int64_t vocab, int64_t ld, int64_t shift_seq, cudaStream_t st) {
  const bool vec = vocab % 8 == 0 && ld % 8 == 0 && aligned16(logits);
  launch_overlapped(vec ? ce_fwd_kernel<T, true> : ce_fwd_kernel<T, false>, dim3((unsigned)rows), dim3(CE_THREADS), 0, st,
                    (const T*)logits, labels, (T*)loss, loss_f32, lse, (int)vocab, ld, shift_seq);
  return launched("cross_entropy_fwd");
}

template <typename T>
static int launch_ce_bwd(const void* logits, const int64_t* labels, const float* lse, const void* grad, int64_t grad_stride,
                         const float* grad_all, float grad_scale, void* dlogits, int64_t rows, int64_t vocab, int64_t ld,
                         int64_t dld, int64_t shift_seq, cudaStream_t st) {
  const bool vec = vocab % 8 == 0 && ld % 8 == 0 && dld % 8 == 0 && aligned16(logits) && aligned16(dlogits);
  launch_overlapped(vec ? ce_bwd_kernel<T, true> : ce_bwd_kernel<T, false>, dim3((unsigned)rows), dim3(CE_THREADS), 0, st,
                    (const T*)logits, labels, lse, (const T*)grad, grad_stride, grad_all, grad_scale, (T*)dlogits, (int)vocab,
                    ld, dld, shift_seq);
  return launched("cross_entropy_bwd");
}

}  // namespace tfb

using namespace tfb;

extern "C" int tfb_cross_entropy_fwd(const void* logits, const int64_t* labels, void* loss,
                                     float* loss_f32, float* lse, int64_t rows, int64_t vocab,
                                     int64_t logits_ld, int dtype, void* stream) {
  TFB_REQUIRE(rows >= 0 && vocab > 0 && vocab < (1LL << 31) - 8, "cross_entropy_fwd: bad shape");
  TFB_REQUIRE(logits_ld >= vocab, "cross_entropy_fwd: row stride smaller than vocab");
  if (rows == 0) return TFB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  TFB_DISPATCH_16(dtype, T, { return launch_ce_fwd<T>(logits, labels, loss, loss_f32, lse, rows, vocab, logits_ld, 0, st); })
}

extern "C" int tfb_cross_entropy_bwd(const void* logits, const int64_t* labels, const float* lse,
                                     const void* grad, int64_t grad_stride, void* dlogits,
                                     int64_t rows, int64_t vocab, int64_t logits_ld,
                                     int64_t dlogits_ld, int dtype, void* stream) {
  TFB_REQUIRE(rows >= 0 && vocab > 0 && vocab < (1LL << 31) - 8, "cross_entropy_bwd: bad shape");
  TFB_REQUIRE(logits_ld >= vocab && dlogits_ld >= vocab, "cross_entropy_bwd: row stride smaller than vocab");
  if (rows == 0) return TFB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  TFB_DISPATCH_16(dtype, T, {
    return launch_ce_bwd<T>(logits, labels, lse, grad, grad_stride, nullptr, 1.f, dlogits, rows, vocab, logits_ld, dlogits_ld, 0,
                            st);
  })
}

extern "C" int tfb_lm_loss_fwd(const void* logits, const int64_t* labels, float* loss, float* row_loss, float* lse,
                               int64_t batch, int64_t seq, int64_t vocab, int64_t logits_ld, int dtype, void* stream) {
  TFB_REQUIRE(batch >= 0 && seq > 0 && vocab > 0 && vocab < (1LL << 31) - 8, "lm_loss_fwd: bad shape");
  TFB_REQUIRE(logits_ld >= vocab, "lm_loss_fwd: row stride smaller than vocab");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t rows = batch * seq;
  if (rows > 0) {
    int rc = TFB_OK;
    TFB_DISPATCH_16(dtype, T, { rc = launch_ce_fwd<T>(logits, labels, nullptr, row_loss, lse, rows, vocab, logits_ld, seq, st); })
    if (rc) return rc;
  }
  launch_overlapped(ce_mean_kernel, dim3(1), dim3(CE_SUM_THREADS), 0, st, (const float*)row_loss, loss, rows,
                    (float)(batch * (seq - 1)));
  return launched("lm_loss_fwd");
}

extern "C" int tfb_lm_loss_bwd(const void* logits, const int64_t* labels, const float* lse, const float* grad, void* dlogits,
                               int64_t batch, int64_t seq, int64_t vocab, int64_t logits_ld, int64_t dlogits_ld, int dtype,
                               void* stream) {
  TFB_REQUIRE(batch >= 0 && seq > 0 && vocab > 0 && vocab < (1LL << 31) - 8, "lm_loss_bwd: bad shape");
  TFB_REQUIRE(logits_ld >= vocab && dlogits_ld >= vocab, "lm_loss_bwd: row stride smaller than vocab");
  if (batch == 0) return TFB_OK;
  TFB_DISPATCH_16(dtype, T, {
    return launch_ce_bwd<T>(logits, labels, lse, nullptr, 0, grad, 1.f / (float)(batch * (seq - 1)), dlogits, batch * seq, vocab,
                            logits_ld, dlogits_ld, seq, (cudaStream_t)stream);
  })
}
