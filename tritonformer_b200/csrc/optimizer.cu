// Optimizer step on the flat gradient buckets for sm_100a: loss-scale handling and AdamW with fp32 master
// weights, entirely on the device (no host read decides anything), HBM-bound.
//
//   grad_check      one pass over a bucket of 16-bit gradients: raises *found_inf if any value is not finite
//   adamw_step      per element: g = grad * inv_scale; decoupled weight decay on the fp32 master weight;
//                   m, v moment updates; bias-corrected step; the 16-bit parameter is the rounded master weight.
//                   The whole launch does nothing while *found_inf is set (the step is skipped as a whole).
//   scale_update    one thread: dynamic loss scale (back off after a skipped step, grow after `interval` good
//                   ones), the step counter (advances only when the step was taken), and clears found_inf.
// The arithmetic follows torch.optim.AdamW's single-tensor form operation by operation (decay, lerp of the
// first moment, mul + addcmul of the second, sqrt / sqrt(bias_correction2) + eps, addcdiv) with the bias
// corrections evaluated in double like the Python floats there, so the fp32 state tracks a CPU run of
// torch.optim.AdamW to the last bit or one unit beside it.
// Algorithmic bytes per element (e = 2): check e; step e (grad) + 12 read + 12 written (master, m, v) + e (param).
//
// One launch takes every bucket (OPT_BUCKETS at a time): its blocks walk one list of chunks over all of them.  With a launch
// per bucket of 32 MB, the start of a kernel (the bias corrections in double, the first loads) and its partly filled last
// round cost as much as a tenth of the pass: 151 M parameters in ten buckets took 801-817 us and take 738 (the checks
// together 93 us at 3.2 TB/s, now 58).  Evict-first loads and stores of the state with three blocks per SM, all of them
// resident, were slower (811 us).
// The check walks the list backwards, so that the step, which walks it forwards, finds the last gradients that the check has
// read in the L2.
#include "common.cuh"

namespace tfb {

constexpr int OPT_BUCKETS = 64;    // buckets per launch
constexpr int OPT_VEC = 256 * 8;   // elements a block takes in one go, eight per thread
constexpr int CHECK_UNROLL = 4;    // of these per chunk of the check: loads in flight per thread
constexpr int STEP_BLOCKS = 8;     // blocks per SM of the step

struct BucketList {
  int count;
  int end[OPT_BUCKETS];  // chunks up to and including the bucket
  int64_t n[OPT_BUCKETS];
  const void* grad[OPT_BUCKETS];
  void* param[OPT_BUCKETS];
  float *master[OPT_BUCKETS], *m[OPT_BUCKETS], *v[OPT_BUCKETS];
};

template <typename T>
__global__ void __launch_bounds__(256) grad_check_kernel(const __grid_constant__ BucketList list, int* __restrict__ found_inf) {
  grid_dependency_wait();
  allow_dependents();
  bool bad = false;
  int b = list.count - 1;
  for (int c = list.end[b] - 1 - (int)blockIdx.x; c >= 0; c -= (int)gridDim.x) {
    while (b > 0 && c < list.end[b - 1]) --b;
    const T* grad = reinterpret_cast<const T*>(list.grad[b]);
    const int64_t n = list.n[b], first = ((int64_t)(c - (b ? list.end[b - 1] : 0)) * (CHECK_UNROLL * 256) + threadIdx.x) * 8;
    if (first + (CHECK_UNROLL - 1) * OPT_VEC + 8 <= n) {
      uint4 raw[CHECK_UNROLL];
#pragma unroll
      for (int u = 0; u < CHECK_UNROLL; ++u) raw[u] = __ldcg(reinterpret_cast<const uint4*>(grad + first + u * OPT_VEC));
#pragma unroll
      for (int u = 0; u < CHECK_UNROLL; ++u) {
        float f[8];
        unpack8<T>(raw[u], f);
#pragma unroll
        for (int k = 0; k < 8; ++k) bad |= !isfinite(f[k]);
      }
    } else {
      for (int u = 0; u < CHECK_UNROLL; ++u)
        for (int k = 0; k < 8; ++k) {
          const int64_t i = first + u * OPT_VEC + k;
          if (i < n) bad |= !isfinite(Num<T>::to_f(grad[i]));
        }
    }
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicExch(found_inf, 1);
}

// Scalars worked out on the host in double and rounded once, as torch does with its Python floats.
struct AdamArgs {
  double lr, beta1, beta2d;  // enter the bias corrections, which are evaluated in double
  float beta2, eps;
  float decay;    // 1 - lr * weight_decay
  float om_beta1; // 1 - beta1
  float om_beta2; // 1 - beta2
};

__device__ __forceinline__ void adamw_one(float g, float& w, float& m, float& v, const AdamArgs& a, float step_size,
                                          float bc2_sqrt) {
  // the forms a CPU run of torch.optim.AdamW takes (found by comparing bit patterns over several steps): the
  // lerp of the first moment and the addcmul of the second are fused multiply-adds, the addcdiv is
  // value * exp_avg / denom with the product first
  w = __fmul_rn(w, a.decay);
  m = __fmaf_rn(a.om_beta1, __fsub_rn(g, m), m);
  v = __fmaf_rn(__fmul_rn(a.om_beta2, g), g, __fmul_rn(v, a.beta2));
  const float denom = __fadd_rn(__fdiv_rn(__fsqrt_rn(v), bc2_sqrt), a.eps);
  w = __fadd_rn(w, __fdiv_rn(__fmul_rn(-step_size, m), denom));
}

template <typename T>
__global__ void __launch_bounds__(256) adamw_step_kernel(const __grid_constant__ BucketList list,
                                                                      const float* __restrict__ inv_scale,
                                                                      const int* __restrict__ found_inf,
                                                                      const float* __restrict__ steps_taken, AdamArgs a) {
  __shared__ float s_corr[2];
  grid_dependency_wait();
  allow_dependents();
  if (found_inf && *found_inf) return;  // the whole step is skipped
  const float unscale = inv_scale ? *inv_scale : 1.f;
  if (threadIdx.x == 0) {
    const double t = (double)(steps_taken ? *steps_taken : 0.f) + 1.0;
    s_corr[0] = (float)(a.lr / (1.0 - pow(a.beta1, t)));
    s_corr[1] = (float)sqrt(1.0 - pow(a.beta2d, t));
  }
  __syncthreads();
  const float step_size = s_corr[0], bc2_sqrt = s_corr[1];
  const int total = list.end[list.count - 1];
  int b = 0;
  for (int c = (int)blockIdx.x; c < total; c += (int)gridDim.x) {
    while (c >= list.end[b]) ++b;
    const T* grad = reinterpret_cast<const T*>(list.grad[b]);
    T* param = reinterpret_cast<T*>(list.param[b]);
    float *master = list.master[b], *m_ = list.m[b], *v_ = list.v[b];
    const int64_t n = list.n[b], first = ((int64_t)(c - (b ? list.end[b - 1] : 0)) * 256 + threadIdx.x) * 8;
    if (first + 8 <= n) {
      const uint4 raw = ld_stream16(grad + first);
      float g[8], w[8], m[8], v[8];
      *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(master + first);
      *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(master + first + 4);
      *reinterpret_cast<float4*>(m) = *reinterpret_cast<const float4*>(m_ + first);
      *reinterpret_cast<float4*>(m + 4) = *reinterpret_cast<const float4*>(m_ + first + 4);
      *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(v_ + first);
      *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(v_ + first + 4);
      unpack8<T>(raw, g);
#pragma unroll
      for (int k = 0; k < 8; ++k) adamw_one(g[k] * unscale, w[k], m[k], v[k], a, step_size, bc2_sqrt);
      *reinterpret_cast<float4*>(master + first) = *reinterpret_cast<const float4*>(w);
      *reinterpret_cast<float4*>(master + first + 4) = *reinterpret_cast<const float4*>(w + 4);
      *reinterpret_cast<float4*>(m_ + first) = *reinterpret_cast<const float4*>(m);
      *reinterpret_cast<float4*>(m_ + first + 4) = *reinterpret_cast<const float4*>(m + 4);
      *reinterpret_cast<float4*>(v_ + first) = *reinterpret_cast<const float4*>(v);
      *reinterpret_cast<float4*>(v_ + first + 4) = *reinterpret_cast<const float4*>(v + 4);
      *reinterpret_cast<uint4*>(param + first) = pack8<T>(w);
    } else {
      for (int64_t i = first; i < n; ++i) {  // (first + 8 > n: fewer than eight)
        float w = master[i], m = m_[i], v = v_[i];
        adamw_one(Num<T>::to_f(grad[i]) * unscale, w, m, v, a, step_size, bc2_sqrt);
        master[i] = w;
        m_[i] = m;
        v_[i] = v;
        param[i] = Num<T>::from_f(w);
      }
    }
  }
}

// state[0] = loss scale, state[1] = 1 / scale, state[2] = good steps since the last change of the scale,
// state[3] = optimizer steps taken
__global__ void scale_update_kernel(float* __restrict__ state, int* __restrict__ found_inf, float growth, float backoff,
                                    int interval) {
  grid_dependency_wait();
  allow_dependents();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (*found_inf) {
    state[0] *= backoff;
    state[2] = 0.f;
  } else {
    state[3] += 1.f;
    const float good = state[2] + 1.f;
    if (good >= (float)interval) {
      state[0] *= growth;
      state[2] = 0.f;
    } else {
      state[2] = good;
    }
  }
  state[1] = 1.f / state[0];
  *found_inf = 0;
}

}  // namespace tfb

using namespace tfb;

// Hands the non-empty buckets to `launch` OPT_BUCKETS at a time, with the chunks of `chunk` elements counted up.
template <typename Fill, typename Launch>
static int for_bucket_lists(const int64_t* n, int count, int64_t chunk, Fill fill, Launch launch) {
  BucketList list;
  list.count = 0;
  int64_t chunks = 0;
  for (int i = 0; i < count; ++i) {
    const int64_t add = ceil_div(n[i], chunk);
    if (list.count == OPT_BUCKETS || (list.count && chunks + add >= (1LL << 30))) {
      if (int rc = launch(list)) return rc;
      list.count = 0;
      chunks = 0;
    }
    if (n[i] == 0) continue;
    TFB_REQUIRE(add < (1LL << 30), "optimizer: bucket too large");
    chunks += add;
    list.n[list.count] = n[i];
    list.end[list.count] = (int)chunks;
    fill(list, list.count++, i);
  }
  return list.count ? launch(list) : TFB_OK;
}

extern "C" int tfb_grad_check_many(const void* const* grads, const int64_t* n, int count, int dtype, int* found_inf, void* stream) {
  TFB_REQUIRE(count >= 0 && found_inf != nullptr && (count == 0 || (grads && n)), "grad_check: bad arguments");
  bool any = false;
  for (int i = 0; i < count; ++i) {
    TFB_REQUIRE(n[i] >= 0, "grad_check: bad arguments");
    TFB_REQUIRE(n[i] == 0 || (grads[i] != nullptr && aligned16(grads[i])), "grad_check: the gradient buffer must be 16-byte aligned");
    any |= n[i] > 0;
  }
  if (!any) return TFB_OK;
  TFB_DISPATCH_16(dtype, T, {
    return for_bucket_lists(
        n, count, CHECK_UNROLL * OPT_VEC, [&](BucketList& l, int at, int i) { l.grad[at] = grads[i]; },
        [&](const BucketList& l) {
          const int cap = sm_count() * 8, want = l.end[l.count - 1];
          launch_overlapped(grad_check_kernel<T>, dim3(want < cap ? want : cap), dim3(256), 0, (cudaStream_t)stream, l, found_inf);
          return launched("grad_check");
        });
  })
}

extern "C" int tfb_grad_check(const void* grad, int64_t n, int dtype, int* found_inf, void* stream) {
  return tfb_grad_check_many(&grad, &n, 1, dtype, found_inf, stream);
}

extern "C" int tfb_adamw_step_many(const void* const* grads, void* const* params, float* const* masters, float* const* exp_avgs,
                                   float* const* exp_avg_sqs, const int64_t* n, int count, int dtype, const float* inv_scale,
                                   const int* found_inf, const float* steps_taken, double lr, double beta1, double beta2,
                                   double eps, double weight_decay, void* stream) {
  TFB_REQUIRE(count >= 0 && (count == 0 || (grads && params && masters && exp_avgs && exp_avg_sqs && n)), "adamw_step: null list");
  bool any = false;
  for (int i = 0; i < count; ++i) {
    TFB_REQUIRE(n[i] >= 0, "adamw_step: negative size");
    if (n[i] == 0) continue;
    any = true;
    TFB_REQUIRE(grads[i] && params[i] && masters[i] && exp_avgs[i] && exp_avg_sqs[i], "adamw_step: null buffer");
    TFB_REQUIRE(aligned16(grads[i]) && aligned16(params[i]) && aligned16(masters[i]) && aligned16(exp_avgs[i]) &&
                    aligned16(exp_avg_sqs[i]),
                "adamw_step: buffers must be 16-byte aligned");
  }
  if (!any) return TFB_OK;
  TFB_REQUIRE(lr >= 0.0 && beta1 >= 0.0 && beta1 < 1.0 && beta2 >= 0.0 && beta2 < 1.0 && eps >= 0.0,
              "adamw_step: bad hyper-parameter");
  TFB_REQUIRE(1.0 - beta1 < 0.5, "adamw_step: beta1 must exceed 0.5 (the first-moment update is written for that case)");
  // hyper-parameters arrive as doubles (Python floats) and every derived scalar is rounded to fp32 once
  AdamArgs a{lr, beta1, beta2, (float)beta2, (float)eps, (float)(1.0 - lr * weight_decay), (float)(1.0 - beta1),
             (float)(1.0 - beta2)};
  TFB_DISPATCH_16(dtype, T, {
    return for_bucket_lists(
        n, count, OPT_VEC,
        [&](BucketList& l, int at, int i) {
          l.grad[at] = grads[i];
          l.param[at] = params[i];
          l.master[at] = masters[i];
          l.m[at] = exp_avgs[i];
          l.v[at] = exp_avg_sqs[i];
        },
        [&](const BucketList& l) {
          const int cap = sm_count() * STEP_BLOCKS, want = l.end[l.count - 1];
          launch_overlapped(adamw_step_kernel<T>, dim3(want < cap ? want : cap), dim3(256), 0, (cudaStream_t)stream, l, inv_scale,
                            found_inf, steps_taken, a);
          return launched("adamw_step");
        });
  })
}

extern "C" int tfb_adamw_step(const void* grad, void* param, float* master, float* exp_avg, float* exp_avg_sq,
                              int64_t n, int dtype, const float* inv_scale, const int* found_inf,
                              const float* steps_taken, double lr, double beta1, double beta2, double eps,
                              double weight_decay, void* stream) {
  return tfb_adamw_step_many(&grad, &param, &master, &exp_avg, &exp_avg_sq, &n, 1, dtype, inv_scale, found_inf, steps_taken, lr,
                             beta1, beta2, eps, weight_decay, stream);
}

extern "C" int tfb_loss_scale_update(float* state4, int* found_inf, float growth, float backoff, int interval,
                                     void* stream) {
  TFB_REQUIRE(state4 != nullptr && found_inf != nullptr, "loss_scale_update: null state");
  TFB_REQUIRE(growth >= 1.f && backoff > 0.f && backoff <= 1.f && interval > 0, "loss_scale_update: bad factors");
  launch_overlapped(scale_update_kernel, dim3(1), dim3(32), 0, (cudaStream_t)stream, state4, found_inf, growth, backoff,
                    interval);
  return launched("loss_scale_update");
}
