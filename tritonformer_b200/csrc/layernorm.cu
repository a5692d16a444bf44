// LayerNorm forward / backward for sm_100a: HBM-bound, 128-bit accesses, fp32 math.
//
// Forward : one warp per row, the row held in registers between the mean, variance and
//           write passes, so x is read once and y written once (4 bytes / element).
// Backward: a CTA owns all columns (8 per thread) and walks groups of rows; it writes dx
//           and keeps the per-column sums for dalpha / dbeta in registers, which leave the
//           CTA once as fp32 partial rows.  finalize_partials() folds those rows.
#include "common.cuh"

namespace tfb {

// ------------------------------------------------------------------------------ forward
template <typename T, int NV>
__global__ void __launch_bounds__(128) ln_fwd_vec_kernel(
    const T* __restrict__ x, const T* __restrict__ alpha, const T* __restrict__ beta,
    T* __restrict__ y, float* __restrict__ mean, float* __restrict__ rstd,
    int64_t rows, int d, int64_t x_ld, int64_t y_ld, float eps) {
  grid_dependency_wait();
  allow_dependents();
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int nvec = d >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * x_ld);
  float v[NV][8];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = i * 32 + lane;
    if (c < nvec) {
      unpack8<T>(ld_stream16(xr + c), v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) s += v[i][j];
    }
  }
  const float mu = warp_sum(s) / (float)d;
  float q = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (i * 32 + lane < nvec) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float t = v[i][j] - mu;
        q += t * t;
      }
    }
  }
  const float rs = rsqrtf(warp_sum(q) / (float)d + eps);
  if (lane == 0) {
    mean[row] = mu;
    rstd[row] = rs;
  }
  uint4* yr = reinterpret_cast<uint4*>(y + row * y_ld);
  const uint4* av = reinterpret_cast<const uint4*>(alpha);
  const uint4* bv = reinterpret_cast<const uint4*>(beta);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = i * 32 + lane;
    if (c < nvec) {
      float a[8], b[8], o[8];
      unpack8<T>(__ldg(av + c), a);
      unpack8<T>(__ldg(bv + c), b);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = a[j] * ((v[i][j] - mu) * rs) + b[j];
      st_stream16(yr + c, pack8<T>(o));
    }
  }
}

// Any d, any alignment: the row is re-read (from L1/L2) for each pass.
template <typename T>
__global__ void __launch_bounds__(128) ln_fwd_generic_kernel(
    const T* __restrict__ x, const T* __restrict__ alpha, const T* __restrict__ beta,
    T* __restrict__ y, float* __restrict__ mean, float* __restrict__ rstd,
    int64_t rows, int d, int64_t x_ld, int64_t y_ld, float eps) {
  grid_dependency_wait();
  allow_dependents();
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const T* xr = x + row * x_ld;
  float s = 0.f;
  for (int c = lane; c < d; c += 32) s += Num<T>::to_f(xr[c]);
  const float mu = warp_sum(s) / (float)d;
  float q = 0.f;
  for (int c = lane; c < d; c += 32) {
    const float t = Num<T>::to_f(xr[c]) - mu;
    q += t * t;
  }
  const float rs = rsqrtf(warp_sum(q) / (float)d + eps);
  if (lane == 0) {
    mean[row] = mu;
    rstd[row] = rs;
  }
  T* yr = y + row * y_ld;
  for (int c = lane; c < d; c += 32)
    yr[c] = Num<T>::from_f(Num<T>::to_f(alpha[c]) * ((Num<T>::to_f(xr[c]) - mu) * rs) +
                           Num<T>::to_f(beta[c]));
}

// ----------------------------------------------------------------------------- backward
constexpr int LN_RB = 4;  // rows per CTA iteration

template <typename T, bool VEC, int MAXT>
__global__ void __launch_bounds__(MAXT) ln_bwd_kernel(
    const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ alpha,
    const float* __restrict__ mean, const float* __restrict__ rstd, T* __restrict__ dx,
    float* __restrict__ partials, int64_t rows, int d, int64_t dy_ld, int64_t x_ld,
    int64_t dx_ld, const T* __restrict__ dres, int64_t dres_ld) {
  grid_dependency_wait();
  allow_dependents();
  __shared__ float red[2][32][2 * LN_RB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarp = blockDim.x >> 5;
  const int c0 = tid * 8;
  const bool active = c0 < d;
  const int ncol = active ? min(8, d - c0) : 0;  // < 8 only on the scalar path

  float a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = (j < ncol) ? Num<T>::to_f(alpha[c0 + j]) : 0.f;
  float acc_a[8], acc_b[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc_a[j] = acc_b[j] = 0.f;

  const float inv_d = 1.f / (float)d;
  int buf = 0;
  const int64_t stride = (int64_t)gridDim.x * LN_RB;
  // raw 16-byte vectors of the row group being processed and of the next one (loads for the next
  // group are in flight while this one goes through its reduction, barrier and stores)
  uint4 cx[LN_RB], cg[LN_RB], nx[LN_RB], ng[LN_RB];
  auto fetch = [&](int64_t r0, uint4 (&vx)[LN_RB], uint4 (&vg)[LN_RB]) {
    if (!VEC) return;
#pragma unroll
    for (int r = 0; r < LN_RB; ++r) {
      const int64_t row = r0 + r;
      if (row < rows && active) {
        vx[r] = ld_stream16(x + row * x_ld + c0);
        vg[r] = ld_stream16(dy + row * dy_ld + c0);
      }
    }
  };
  fetch((int64_t)blockIdx.x * LN_RB, cx, cg);
  for (int64_t r0 = (int64_t)blockIdx.x * LN_RB; r0 < rows; r0 += stride) {
    if (r0 + stride < rows) fetch(r0 + stride, nx, ng);
    uint4 rv[LN_RB];  // residual-branch gradient, needed only after the reduction
    if (VEC && dres) {
#pragma unroll
      for (int r = 0; r < LN_RB; ++r)
        if (r0 + r < rows && active) rv[r] = ld_stream16(dres + (r0 + r) * dres_ld + c0);
    }
    float xh[LN_RB][8], g[LN_RB][8];
    float s[2 * LN_RB];
#pragma unroll
    for (int r = 0; r < LN_RB; ++r) {
      const int64_t row = r0 + r;
      s[2 * r] = s[2 * r + 1] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) xh[r][j] = g[r][j] = 0.f;
      if (row < rows && active) {
        float xv[8], dv[8];
        if (VEC) {
          unpack8<T>(cx[r], xv);
          unpack8<T>(cg[r], dv);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            xv[j] = (j < ncol) ? Num<T>::to_f(x[row * x_ld + c0 + j]) : 0.f;
            dv[j] = (j < ncol) ? Num<T>::to_f(dy[row * dy_ld + c0 + j]) : 0.f;
          }
        }
        const float mu = __ldg(mean + row), rs = __ldg(rstd + row);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float h = (j < ncol) ? (xv[j] - mu) * rs : 0.f;
          xh[r][j] = h;
          g[r][j] = dv[j] * a[j];
          acc_a[j] += dv[j] * h;
          acc_b[j] += dv[j];
          s[2 * r] += g[r][j] * h;
          s[2 * r + 1] += g[r][j];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2 * LN_RB; ++i) s[i] = warp_sum(s[i]);
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < 2 * LN_RB; ++i) red[buf][warp][i] = s[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2 * LN_RB; ++i) {
      float t = 0.f;
      for (int w = 0; w < nwarp; ++w) t += red[buf][w][i];
      s[i] = t * inv_d;
    }
    buf ^= 1;
#pragma unroll
    for (int r = 0; r < LN_RB; ++r) {
      const int64_t row = r0 + r;
      if (row < rows && active) {
        const float rs = __ldg(rstd + row);
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rs * (g[r][j] - xh[r][j] * s[2 * r] - s[2 * r + 1]);
        if (VEC) {
          if (dres) {  // gradient arriving through the residual branch that forked at this LayerNorm's input
            float e[8];
            unpack8<T>(rv[r], e);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] += e[j];
          }
          st_stream16(dx + row * dx_ld + c0, pack8<T>(o));
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < ncol)
              dx[row * dx_ld + c0 + j] =
                  Num<T>::from_f(o[j] + (dres ? Num<T>::to_f(dres[row * dres_ld + c0 + j]) : 0.f));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < LN_RB; ++r) {
      cx[r] = nx[r];
      cg[r] = ng[r];
    }
  }
  if (active) {
    float* pa = partials + (int64_t)blockIdx.x * 2 * d;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j < ncol) {
        pa[c0 + j] = acc_a[j];
        pa[d + c0 + j] = acc_b[j];
      }
    }
  }
}

// Backward for vectorisable rows of at most 2048 elements: G warps share a row, a lane owns ONE
// 16-byte vector of it, so a thread keeps only 8 columns of alpha and of the dalpha / dbeta sums in
// registers.  RG such groups make a CTA; a group takes one row at a time, with the next row's vectors on their way in
// registers.  The two row sums are reduced by warp shuffles and exchanged between the G warps through shared memory behind
// a named barrier (double-buffered).
// What bounds it: the instructions a warp issues per row, one in 7 cycles at four warps per scheduler.  So the arithmetic is
// packed (two columns an instruction), nothing is copied through shared memory, and two CTAs, all that the grid has for an SM, give a
// scheduler six warps (widths up to 1024 and of 1281-1536; five at 1025-1280, three and a half at 1537-1792, four above).  With a
// cp.async ring per lane, G a power of two and four warps per scheduler: 31 instructions per element.  With the residual
// gradient and the fold of the partials, cold L2, fp16: 8192 x 1024 22.8 -> 18.0 us, 4096 x 1536 24.1 -> 15.5, 2048 x 768
// 10.2 -> 7.7, 512 x 256 8.0 -> 4.2, 4096 x 2048 25.9 -> 23.0, 32768 x 1024 58.3 -> 50.6 (5.3 TB/s).
constexpr int LN_WARPS = 12;  // of a CTA, at most
constexpr int ln_groups(int g) { return LN_WARPS / g; }
template <typename T>
__device__ __forceinline__ void unpack8_pairs(const uint4& raw, uint64_t (&v)[4]) {
  float f[8];
  unpack8<T>(raw, f);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = f2_pack(f[2 * i], f[2 * i + 1]);
}

template <typename T, int G, bool RES>
__global__ void __launch_bounds__(32 * G * ln_groups(G), LN_WARPS * 2 / (G * ln_groups(G))) ln_bwd_split_kernel(
    const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ alpha,
    const float* __restrict__ mean, const float* __restrict__ rstd, T* __restrict__ dx,
    float* __restrict__ partials, uint32_t rows, int d, uint32_t dy_ld, uint32_t x_ld, uint32_t dx_ld,
    const T* __restrict__ dres, uint32_t dres_ld) {  // (32 bits: no registers for what walks down the tensors)
  grid_dependency_wait();
  allow_dependents();
  constexpr int RG = ln_groups(G);
  extern __shared__ __align__(16) uint8_t ln_smem[];
  float* fold = reinterpret_cast<float*>(ln_smem);  // [RG][2][d]
  __shared__ float2 xch[RG][2][G];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = warp % G, rg = warp / G;
  const int c = part * 32 + lane;
  const bool has = c < (d >> 3);

  uint64_t a[4], acc_a[4], acc_b[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) a[j] = acc_a[j] = acc_b[j] = 0ull;
  if (has) unpack8_pairs<T>(__ldg(reinterpret_cast<const uint4*>(alpha) + c), a);
  const float inv_d = 1.f / (float)d;
  const uint32_t stride = gridDim.x * RG;
  uint32_t row = blockIdx.x * RG + rg;
  auto at = [&](uint32_t r, uint32_t ld) -> uint64_t { return (uint64_t)r * ld + (uint32_t)(c * 8); };
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 nx = zero, ny = zero, nr = zero;
  float n_mu = 0.f, n_rs = 0.f;
  auto fetch = [&](uint32_t r) {
    if (r >= rows) return;
    if (has) {
      nx = ld_stream16(x + at(r, x_ld));
      ny = ld_stream16(dy + at(r, dy_ld));
      if (RES) nr = ld_stream16(dres + at(r, dres_ld));
    }
    n_mu = __ldg(mean + r);
    n_rs = __ldg(rstd + r);
  };
  fetch(row);
  int parity = 0;
  for (; row < rows; row += stride) {
    uint64_t h[4], g[4];
    unpack8_pairs<T>(nx, h);
    unpack8_pairs<T>(ny, g);
    const uint4 raw = nr;
    const float mu = n_mu, rs = n_rs;
    fetch(row + stride);
    // a lane without columns holds zeros, which contribute nothing
    const uint64_t rs2 = has ? f2_pack(rs, rs) : 0ull, sh2 = has ? f2_pack(-mu * rs, -mu * rs) : 0ull;
    uint64_t s1 = 0ull, s2 = 0ull;
    const uint64_t one = f2_pack(1.f, 1.f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      h[j] = f2_fma(h[j], rs2, sh2);          // normalised input
      acc_a[j] = f2_fma(g[j], h[j], acc_a[j]);
      acc_b[j] = f2_fma(g[j], one, acc_b[j]);
      g[j] = f2_mul(g[j], a[j]);              // alpha-scaled gradient
      s1 = f2_fma(g[j], h[j], s1);
      s2 = f2_add(g[j], s2);
    }
    float t1, t2;
    {
      float lo, hi;
      f2_unpack(s1, lo, hi);
      t1 = lo + hi;
      f2_unpack(s2, lo, hi);
      t2 = lo + hi;
      // both sums in five exchanges: after the first, the lower half of the warp carries t1 and the upper half t2
      const bool up = lane & 16;
      float v = (up ? t2 : t1) + __shfl_xor_sync(0xffffffffu, up ? t1 : t2, 16);
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      if (G == 1) {
        t1 = __shfl_sync(0xffffffffu, v, 0);
        t2 = __shfl_sync(0xffffffffu, v, 16);
      } else {
        // all G warps of the group take the same number of rows, so the barrier counts match
        if ((lane & 15) == 0) reinterpret_cast<float*>(&xch[rg][parity][part])[lane >> 4] = v;
        asm volatile("bar.sync %0, %1;" ::"r"(1 + rg), "r"(32 * G) : "memory");
        t1 = t2 = 0.f;
#pragma unroll
        for (int i = 0; i < G; ++i) {
          const float2 u = xch[rg][parity][i];
          t1 += u.x;
          t2 += u.y;
        }
        parity ^= 1;
      }
    }
    // dx = rstd * (g - h * mean(g h) - mean(g)) as two fused multiply-adds per element
    const float k1 = -rs * t1 * inv_d, k2 = -rs * t2 * inv_d;
    const uint64_t k1p = f2_pack(k1, k1), k2p = f2_pack(k2, k2);
    uint64_t res[4];
    if (RES) unpack8_pairs<T>(raw, res);
    float o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint64_t v = f2_fma(rs2, g[j], f2_fma(k1p, h[j], k2p));
      if (RES) v = f2_add(v, res[j]);  // gradient arriving through the residual branch that forked at this LayerNorm's input
      f2_unpack(v, o[2 * j], o[2 * j + 1]);
    }
    if (has) st_stream16(dx + at(row, dx_ld), pack8<T>(o));
  }
  // the groups' sums are added in their order, so the result does not depend on timing
  if (has) {
    uint64_t* f = reinterpret_cast<uint64_t*>(fold + (size_t)rg * 2 * d + c * 8);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f[j] = acc_a[j];
      f[d / 2 + j] = acc_b[j];
    }
  }
  __syncthreads();
  float* pa = partials + (int64_t)blockIdx.x * 2 * d;
  for (int i = threadIdx.x; i < 2 * d; i += blockDim.x) {
    float t = fold[i];
#pragma unroll 4
    for (int k = 1; k < RG; ++k) t += fold[(size_t)k * 2 * d + i];
    pa[i] = t;
  }
}

// 32 columns per CTA; the rows are spread over the CTA's warps (32 for many partial rows, 8 otherwise), so
// that each thread has only a few dependent-free loads to wait for.
template <typename T>
__global__ void __launch_bounds__(1024) finalize_partials_kernel(
    const float* __restrict__ partials, int64_t n, int ncols, int split, T* __restrict__ out0,
    T* __restrict__ out1, int accumulate) {
  grid_dependency_wait();
  allow_dependents();
  __shared__ float sm[32][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5, nry = blockDim.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (c < ncols)
    for (int64_t r = ry; r < n; r += nry) s += partials[r * ncols + c];
  sm[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && c < ncols) {
    for (int i = 1; i < nry; ++i) s += sm[i][cx];
    T* dst = c < split ? out0 + c : out1 + (c - split);
    if (accumulate) s += Num<T>::to_f(*dst);  // the sums are added to what the output already holds
    *dst = Num<T>::from_f(s);
  }
}

template <typename T>
int finalize_partials(const float* partials, int64_t n, int ncols, int split, void* out0,
                      void* out1, cudaStream_t st, int accumulate) {
  launch_overlapped(finalize_partials_kernel<T>, dim3((unsigned)ceil_div(ncols, 32)), dim3(n > 64 ? 1024 : 256), 0, st,
                    partials, n, ncols, split, (T*)out0, (T*)out1, accumulate);
  return launched("finalize_partials");
}
template int finalize_partials<__half>(const float*, int64_t, int, int, void*, void*, cudaStream_t, int);
template int finalize_partials<__nv_bfloat16>(const float*, int64_t, int, int, void*, void*, cudaStream_t, int);

static int ln_bwd_threads(int64_t d) { return (int)(ceil_div(ceil_div(d, 8), 32) * 32); }

template <typename T>
static int ln_bwd_launch(const void* dy, const void* x, const void* alpha, const float* mean,
                         const float* rstd, void* dx, void* dalpha, void* dbeta, float* partials,
                         int64_t n_partials, int64_t rows, int d, int64_t dy_ld, int64_t x_ld,
                         int64_t dx_ld, bool vec, int threads, cudaStream_t st, const void* dres = nullptr,
                         int64_t dres_ld = 0, int accumulate = 0) {
#define TFB_LN_BWD(V, MT)                                                                     \
  launch_overlapped(ln_bwd_kernel<T, V, MT>, dim3((unsigned)n_partials), dim3(threads), 0, st, \
      (const T*)dy, (const T*)x, (const T*)alpha, mean, rstd, (T*)dx, partials, rows, d, dy_ld, \
      x_ld, dx_ld, (const T*)dres, dres_ld)
  constexpr int64_t kWide = 1LL << 31;
  if (vec && d <= 2048 && aligned16(alpha) && rows < kWide && dy_ld < kWide && x_ld < kWide && dx_ld < kWide && dres_ld < kWide) {
    const T *gp = (const T*)dy, *xp = (const T*)x, *ap = (const T*)alpha, *rp = (const T*)dres;
    T* op = (T*)dx;
    const dim3 grid((unsigned)n_partials);
    // at most LN_WARPS / G groups of 2 d <= 512 G floats each: 24 KB
#define TFB_LN_SPLIT(G, RES)                                                                                             \
  launch_overlapped(ln_bwd_split_kernel<T, G, RES>, grid, dim3(32 * G * ln_groups(G)), (size_t)ln_groups(G) * 2 * d * 4, st, gp, xp, ap, \
                    mean, rstd, op, partials, (uint32_t)rows, d, (uint32_t)dy_ld, (uint32_t)x_ld, (uint32_t)dx_ld, rp, (uint32_t)dres_ld)
#define TFB_LN_GROUP(G)                                                                                                  \
  case G:                                                                                                                \
    if (dres) TFB_LN_SPLIT(G, true);                                                                                     \
    else TFB_LN_SPLIT(G, false);                                                                                         \
    break
    switch ((d + 255) / 256) {
      TFB_LN_GROUP(1);
      TFB_LN_GROUP(2);
      TFB_LN_GROUP(3);
      TFB_LN_GROUP(4);
      TFB_LN_GROUP(5);
      TFB_LN_GROUP(6);
      TFB_LN_GROUP(7);
      TFB_LN_GROUP(8);
    }
#undef TFB_LN_GROUP
#undef TFB_LN_SPLIT
  } else if (vec && threads <= 256) TFB_LN_BWD(true, 256);
  else if (vec) TFB_LN_BWD(true, 1024);
  else if (threads <= 256) TFB_LN_BWD(false, 256);
  else TFB_LN_BWD(false, 1024);
#undef TFB_LN_BWD
  int rc = launched("layernorm_bwd");
  if (rc) return rc;
  return finalize_partials<T>(partials, n_partials, 2 * d, d, dalpha, dbeta, st, accumulate);
}

}  // namespace tfb

using namespace tfb;

extern "C" int tfb_layernorm_fwd(const void* x, const void* alpha, const void* beta, void* y,
                                 float* mean, float* rstd, int64_t rows, int64_t d, int64_t x_ld,
                                 int64_t y_ld, float eps, int dtype, void* stream) {
  TFB_REQUIRE(rows >= 0 && d > 0 && d < (1 << 30), "layernorm_fwd: bad shape rows=%lld d=%lld",
              (long long)rows, (long long)d);
  TFB_REQUIRE(x_ld >= d && y_ld >= d, "layernorm_fwd: row stride smaller than d");
  if (rows == 0) return TFB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned grid = (unsigned)ceil_div(rows, 4);
  const bool vec = (d % 8 == 0) && (x_ld % 8 == 0) && (y_ld % 8 == 0) && aligned16(x) &&
                   aligned16(y) && aligned16(alpha) && aligned16(beta) && d <= 2048;
  TFB_DISPATCH_16(dtype, T, {
    const T *xp = (const T*)x, *ap = (const T*)alpha, *bp = (const T*)beta;
    T* yp = (T*)y;
    if (!vec) {
      launch_overlapped(ln_fwd_generic_kernel<T>, dim3(grid), dim3(128), 0, st, xp, ap, bp, yp, mean, rstd, rows, (int)d, x_ld, y_ld, eps);
    } else if (d <= 256) {
      launch_overlapped(ln_fwd_vec_kernel<T, 1>, dim3(grid), dim3(128), 0, st, xp, ap, bp, yp, mean, rstd, rows, (int)d, x_ld, y_ld, eps);
    } else if (d <= 512) {
      launch_overlapped(ln_fwd_vec_kernel<T, 2>, dim3(grid), dim3(128), 0, st, xp, ap, bp, yp, mean, rstd, rows, (int)d, x_ld, y_ld, eps);
    } else if (d <= 1024) {
      launch_overlapped(ln_fwd_vec_kernel<T, 4>, dim3(grid), dim3(128), 0, st, xp, ap, bp, yp, mean, rstd, rows, (int)d, x_ld, y_ld, eps);
    } else {
      launch_overlapped(ln_fwd_vec_kernel<T, 8>, dim3(grid), dim3(128), 0, st, xp, ap, bp, yp, mean, rstd, rows, (int)d, x_ld, y_ld, eps);
    }
  })
  return launched("layernorm_fwd");
}

extern "C" int64_t tfb_layernorm_bwd_partials(int64_t rows, int64_t d) {
  (void)d;
  int64_t n = ceil_div(rows, 16);
  const int64_t cap = 148 * 2;  // two CTAs per SM
  if (n > cap) n = cap;
  return n < 1 ? 1 : n;
}

extern "C" int tfb_layernorm_bwd_acc(const void* dy, const void* x, const void* alpha, const float* mean,
                                     const float* rstd, const void* dres, void* dx, void* dalpha, void* dbeta,
                                     float* partials, int64_t n_partials, int64_t rows, int64_t d, int64_t dy_ld,
                                     int64_t x_ld, int64_t dres_ld, int64_t dx_ld, int accumulate, int dtype,
                                     void* stream) {
  TFB_REQUIRE(rows > 0 && d > 0, "layernorm_bwd: bad shape rows=%lld d=%lld", (long long)rows,
              (long long)d);
  if (d > 8192) return fail(TFB_ERR_UNSUPPORTED, "layernorm_bwd: d=%lld > 8192", (long long)d);
  TFB_REQUIRE(n_partials == tfb_layernorm_bwd_partials(rows, d),
              "layernorm_bwd: scratch must hold tfb_layernorm_bwd_partials() rows");
  TFB_REQUIRE(dy_ld >= d && x_ld >= d && dx_ld >= d && (!dres || dres_ld >= d),
              "layernorm_bwd: row stride smaller than d");
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = (d % 8 == 0) && (x_ld % 8 == 0) && (dy_ld % 8 == 0) && (dx_ld % 8 == 0) &&
                   aligned16(x) && aligned16(dy) && aligned16(dx) &&
                   (!dres || (aligned16(dres) && dres_ld % 8 == 0));
  const int threads = ln_bwd_threads(d);
  TFB_DISPATCH_16(dtype, T, {
    return ln_bwd_launch<T>(dy, x, alpha, mean, rstd, dx, dalpha, dbeta, partials, n_partials, rows,
                            (int)d, dy_ld, x_ld, dx_ld, vec, threads, st, dres, dres_ld, accumulate ? 1 : 0);
  })
}

extern "C" int tfb_layernorm_bwd_res(const void* dy, const void* x, const void* alpha, const float* mean,
                                     const float* rstd, const void* dres, void* dx, void* dalpha, void* dbeta,
                                     float* partials, int64_t n_partials, int64_t rows, int64_t d, int64_t dy_ld,
                                     int64_t x_ld, int64_t dres_ld, int64_t dx_ld, int dtype, void* stream) {
  return tfb_layernorm_bwd_acc(dy, x, alpha, mean, rstd, dres, dx, dalpha, dbeta, partials, n_partials, rows, d,
                               dy_ld, x_ld, dres_ld, dx_ld, 0, dtype, stream);
}

extern "C" int tfb_layernorm_bwd(const void* dy, const void* x, const void* alpha,
                                 const float* mean, const float* rstd, void* dx, void* dalpha,
                                 void* dbeta, float* partials, int64_t n_partials, int64_t rows,
                                 int64_t d, int64_t dy_ld, int64_t x_ld, int64_t dx_ld, int dtype,
                                 void* stream) {
  return tfb_layernorm_bwd_res(dy, x, alpha, mean, rstd, nullptr, dx, dalpha, dbeta, partials, n_partials, rows,
                               d, dy_ld, x_ld, 0, dx_ld, dtype, stream);
}

// ------------------------------------------------------------------------------------------
// LayerNorm backward without caller-provided scratch.
//
// Some hosts of this library cannot hand it scratch memory: a binding that marshals only the
// operator's own inputs and outputs, or a service whose device memory is carved up once at
// start-up and which keeps cudaMalloc / cudaFree (device-wide synchronising calls) off its
// request path.  For them the fp32 partial column sums live in the fixed device array below
// instead of a buffer the caller allocates.  The array belongs to the library image: every
// GPU that loads the library carries it (kStaticRows * 2 * kStaticMaxD floats) until exit.
constexpr int kStaticRows = 296;    // partial rows (two CTAs per SM)
constexpr int kStaticMaxD = 4096;   // widest supported row
static __device__ __align__(256) float g_ln_static_scratch[(size_t)kStaticRows * 2 * kStaticMaxD];

namespace {
struct StaticScratch {
  std::atomic<float*> ptr[64];
};
StaticScratch g_static_scratch;

// Device address of the array on the current device.  `g_ln_static_scratch` named in host code
// is only a handle for the runtime, not something a kernel may dereference; the address has
// to be asked for once per device, with that device current.
int static_scratch_for_current_device(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64)
    return tfb::fail(TFB_ERR_LAUNCH, "layernorm_bwd_static: cudaGetDevice: %s", cudaGetErrorString(e));
  float* p = g_static_scratch.ptr[dev].load(std::memory_order_acquire);
  if (!p) {
    void* sym = nullptr;
    e = cudaGetSymbolAddress(&sym, g_ln_static_scratch);
    if (e != cudaSuccess || !sym)
      return tfb::fail(TFB_ERR_LAUNCH, "layernorm_bwd_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    p = static_cast<float*>(sym);
    g_static_scratch.ptr[dev].store(p, std::memory_order_release);
  }
  *out = p;
  return TFB_OK;
}
}  // namespace

extern "C" int tfb_layernorm_bwd_static(const void* dy, const void* x, const void* alpha, const float* mean,
                                        const float* rstd, void* dx, void* dalpha, void* dbeta, int64_t rows,
                                        int64_t d, int64_t dy_ld, int64_t x_ld, int64_t dx_ld, int dtype,
                                        void* stream) {
  TFB_REQUIRE(rows > 0 && d > 0, "layernorm_bwd_static: bad shape rows=%lld d=%lld", (long long)rows, (long long)d);
  if (d > kStaticMaxD)
    return fail(TFB_ERR_UNSUPPORTED,
                "layernorm_bwd_static: d=%lld exceeds the built-in scratch (rows of at most %d elements); "
                "use tfb_layernorm_bwd with caller-provided scratch",
                (long long)d, kStaticMaxD);
  TFB_REQUIRE(dy_ld >= d && x_ld >= d && dx_ld >= d, "layernorm_bwd_static: row stride smaller than d");
  float* scratch = nullptr;
  int rc = static_scratch_for_current_device(&scratch);
  if (rc) return rc;
  int64_t n = ceil_div(rows, 16);
  if (n > kStaticRows) n = kStaticRows;
  // Every one of the n partial rows is rewritten in full by the first kernel before the second
  // reads it, so nothing in the array has to be cleared between calls.
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = (d % 8 == 0) && (x_ld % 8 == 0) && (dy_ld % 8 == 0) && (dx_ld % 8 == 0) && aligned16(x) &&
                   aligned16(dy) && aligned16(dx);
  const int threads = ln_bwd_threads(d);
  TFB_DISPATCH_16(dtype, T, {
    return ln_bwd_launch<T>(dy, x, alpha, mean, rstd, dx, dalpha, dbeta, scratch, n, rows, (int)d, dy_ld, x_ld,
                            dx_ld, vec, threads, st);
  })
}
