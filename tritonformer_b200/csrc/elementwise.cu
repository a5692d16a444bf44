// ReLU gradient mask and column sums (bias gradient) for sm_100a: HBM-bound,
// 128-bit accesses, fp32 accumulation.
#include "common.cuh"

namespace tfb {

template <typename T> int finalize_partials(const float*, int64_t, int, int, void*, void*, cudaStream_t, int);

template <typename T>
__global__ void __launch_bounds__(256) relu_bwd_vec_kernel(const uint4* __restrict__ dy,
                                                           const uint4* __restrict__ act,
                                                           uint4* __restrict__ dz, int64_t nvec) {
  grid_dependency_wait();
  allow_dependents();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += stride) {
    float g[8], a[8];
    unpack8<T>(ld_stream16(dy + i), g);
    unpack8<T>(ld_stream16(act + i), a);
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = a[j] > 0.f ? g[j] : 0.f;
    st_stream16(dz + i, pack8<T>(g));
  }
}

template <typename T>
__global__ void __launch_bounds__(256) relu_bwd_scalar_kernel(const T* __restrict__ dy, const T* __restrict__ act,
                                                              T* __restrict__ dz, int64_t n) {
  grid_dependency_wait();
  allow_dependents();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    dz[i] = Num<T>::to_f(act[i]) > 0.f ? dy[i] : Num<T>::from_f(0.f);
}

// grid (ceil(cols/256), n_partials); block 256 = 32 column lanes (8 columns each) x 8 row lanes.
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) colsum_kernel(const T* __restrict__ x, float* __restrict__ partials,
                                                     int64_t rows, int cols, int64_t ld) {
  grid_dependency_wait();
  allow_dependents();
  __shared__ float sm[8][32][9];
  const int cl = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int c0 = (blockIdx.x * 32 + cl) * 8;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (c0 < cols) {
    const int ncol = min(8, cols - c0);
    for (int64_t r = (int64_t)blockIdx.y * 8 + rl; r < rows; r += (int64_t)gridDim.y * 8) {
      if (VEC) {
        float f[8];
        unpack8<T>(ld_stream16(x + r * ld + c0), f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += f[j];
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < ncol) acc[j] += Num<T>::to_f(x[r * ld + c0 + j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) sm[rl][cl][j] = acc[j];
  __syncthreads();
  // 256 threads fold 8 row lanes for 32*8 columns
  const int cc = threadIdx.x;  // column within the CTA's 256
  const int col = blockIdx.x * 256 + cc;
  if (col < cols) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += sm[i][cc >> 3][cc & 7];
    partials[(int64_t)blockIdx.y * cols + col] = s;
  }
}

// dz = act > 0 ? dy : 0 (act may be null: a copy) with the column sums of dz on the way: what the backward of a linear
// layer needs before its two products, in one pass over dy and act.  dy and act may have any alignment and pitch; dz has
// 16-byte aligned rows, so that the products can read it through TMA whatever the layer's width (a copy with act and
// sums null packs an operand the same way).  The work of a CTA is the one of colsum_kernel, four rows of a thread in
// flight; each lane fetches what its eight elements lie in, one aligned vector or two.  Both kernels add the rows of a column in the same
// order.
constexpr int GR_ROWS = 4, GR_COLS = 248;
template <typename T>
__global__ void __launch_bounds__(256) grad_rows_kernel(const T* __restrict__ dy, const T* __restrict__ act,
                                                        T* __restrict__ dz, float* __restrict__ partials, int64_t rows,
                                                        int cols, int64_t dy_ld, int64_t act_ld, int64_t dz_ld) {
  grid_dependency_wait();
  allow_dependents();
  __shared__ float sm[8][32][9];
  const int cl = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int c0 = (blockIdx.x * 32 + cl) * 8;
  const int n = min(8, cols - c0);
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (n > 0) {
    const int64_t step = (int64_t)gridDim.y * 8;
    for (int64_t r0 = (int64_t)blockIdx.y * 8 + rl; r0 < rows; r0 += step * GR_ROWS) {
      uint4 g[GR_ROWS], a[GR_ROWS];
#pragma unroll
      for (int i = 0; i < GR_ROWS; ++i) {
        const int64_t r = r0 + i * step;
        if (r >= rows) continue;
        g[i] = load8_any(dy + r * dy_ld + c0, n);
        if (act) a[i] = load8_any(act + r * act_ld + c0, n);
      }
#pragma unroll
      for (int i = 0; i < GR_ROWS; ++i) {
        const int64_t r = r0 + i * step;
        if (r >= rows) continue;
        float f[8];
        unpack8<T>(g[i], f);
        if (act) {
          float m[8];
          unpack8<T>(a[i], m);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = m[j] > 0.f ? f[j] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (j >= n) f[j] = 0.f;  // the padding of a row
          acc[j] += f[j];
        }
        *reinterpret_cast<uint4*>(dz + r * dz_ld + c0) = pack8<T>(f);
      }
    }
  }
  if (!partials) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) sm[rl][cl][j] = acc[j];
  __syncthreads();
  const int cc = threadIdx.x, col = blockIdx.x * 256 + cc;
  if (col < cols) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += sm[i][cc >> 3][cc & 7];
    partials[(int64_t)blockIdx.y * cols + col] = s;
  }
}

// The same for misaligned rows, several of them per warp.
// A warp takes 31 output vectors (248 columns) of a row.  All lanes of a row share one misalignment: lane l loads the aligned
// vector that the l-th output begins in, and the rest of that output is in its neighbour's, so a row is loaded once.  Bound by
// the loads: a thread requests its vectors of GR_ROWS rows before it uses the first.  (Each lane fetching both of its aligned vectors
// itself made every row two dependent loads deep per lane.)  Cold L2, fp16: 5015 x 2930 with mask and sums and their fold
// 39.6 -> 25.6 us (3.4 TB/s of dy, act and dz), a copy of 5015 x 1477 12.0 -> 8.7, of 1477 x 2930 7.4 -> 5.9, of 1024 x 50257
// 57.5 -> 43.1 (4.8 TB/s).
// Loads that vector.  One that holds no wanted byte is not touched; one that does never crosses the end of an allocation.
template <typename T>
__device__ __forceinline__ uint4 load_row_vec(const T* row, int c0, int cols) {
  const uintptr_t v = reinterpret_cast<uintptr_t>(row + c0) & ~uintptr_t(15);
  return v < reinterpret_cast<uintptr_t>(row + cols) ? ld_stream16(reinterpret_cast<const void*>(v)) : make_uint4(0, 0, 0, 0);
}
// The eight elements that begin `off` bytes into this lane's vector (nothing of use in lane 31).
__device__ __forceinline__ uint4 shift_row_vec(const uint4& v, uint32_t off) {
  uint32_t w[8] = {v.x, v.y, v.z, v.w, __shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1),
                   __shfl_down_sync(0xffffffffu, v.z, 1), __shfl_down_sync(0xffffffffu, v.w, 1)};
  if (off & 8) {
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
  }
  if (off & 4) {
#pragma unroll
    for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
  }
  const uint32_t bits = (off & 2) * 8;
  return make_uint4(__funnelshift_r(w[0], w[1], bits), __funnelshift_r(w[1], w[2], bits), __funnelshift_r(w[2], w[3], bits),
                    __funnelshift_r(w[3], w[4], bits));
}
template <typename T, bool ACT>
__global__ void __launch_bounds__(256, ACT ? 3 : 4) grad_rows_shift_kernel(const T* __restrict__ dy, const T* __restrict__ act,
                                                                                 T* __restrict__ dz, float* __restrict__ partials,
                                                                                 int64_t rows, int cols, int64_t dy_ld, int64_t act_ld,
                                                                                 int64_t dz_ld) {
  grid_dependency_wait();
  allow_dependents();
  __shared__ float sm[8][32][9];
  const int cl = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int c0 = blockIdx.x * GR_COLS + cl * 8;
  const int n = cl == 31 ? 0 : min(8, cols - c0);  // columns this lane writes, none where not positive
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  const int64_t step = (int64_t)gridDim.y * 8;
  for (int64_t r0 = (int64_t)blockIdx.y * 8 + rl; r0 < rows; r0 += step * GR_ROWS) {  // the same for all lanes of a warp
    uint4 g[GR_ROWS], a[ACT ? GR_ROWS : 1];
#pragma unroll
    for (int i = 0; i < GR_ROWS; ++i) {
      const int64_t r = r0 + i * step;
      if (r >= rows) break;
      g[i] = load_row_vec(dy + r * dy_ld, c0, cols);
      if (ACT) a[i] = load_row_vec(act + r * act_ld, c0, cols);
    }
#pragma unroll
    for (int i = 0; i < GR_ROWS; ++i) {
      const int64_t r = r0 + i * step;
      if (r >= rows) break;
      float f[8];
      unpack8<T>(shift_row_vec(g[i], (uint32_t)reinterpret_cast<uintptr_t>(dy + r * dy_ld) & 15), f);
      if (ACT) {
        float m[8];
        unpack8<T>(shift_row_vec(a[i], (uint32_t)reinterpret_cast<uintptr_t>(act + r * act_ld) & 15), m);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = m[j] > 0.f ? f[j] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j >= n) f[j] = 0.f;  // the padding of a row
        acc[j] += f[j];
      }
      if (n > 0) *reinterpret_cast<uint4*>(dz + r * dz_ld + c0) = pack8<T>(f);
    }
  }
  if (!partials) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) sm[rl][cl][j] = acc[j];
  __syncthreads();
  const int cc = threadIdx.x, col = blockIdx.x * GR_COLS + cc;
  if (cc < GR_COLS && col < cols) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += sm[i][cc >> 3][cc & 7];
    partials[(int64_t)blockIdx.y * cols + col] = s;
  }
}

}  // namespace tfb

using namespace tfb;

extern "C" int tfb_grad_rows(const void* dy, const void* act, void* dz, void* sums, float* partials, int64_t n_partials,
                             int64_t rows, int64_t cols, int64_t dy_ld, int64_t act_ld, int64_t dz_ld, int dtype,
                             void* stream) {
  TFB_REQUIRE(rows >= 0 && cols > 0 && cols < (1LL << 31) - 256, "grad_rows: bad shape");
  TFB_REQUIRE(dy_ld >= 0 && (!act || act_ld >= 0), "grad_rows: negative row stride");  // rows may repeat or overlap: only read
  TFB_REQUIRE(aligned16(dz) && dz_ld % 8 == 0 && dz_ld >= ceil_div(cols, 8) * 8, "grad_rows: dz rows must be 16-byte aligned");
  TFB_REQUIRE(!sums || (partials && n_partials == tfb_colsum_partials(rows, cols)),
              "grad_rows: scratch must hold tfb_colsum_partials() rows");
  if (rows == 0 && !sums) return TFB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  // Rows that begin on 16-byte boundaries (the ordinary widths) need no shifting, and 248 columns a CTA would leave a width like 256 a
  // second block of CTAs with one lane at work; with less than two rows a warp the shifting has nothing to overlap with.  Warm L2, fp16,
  // plain kernel and shifting one: 8192 x 1024 with mask 6.8 and 11.9 us, 1920 x 256 1.7 and 2.9, 5015 x 2928 13.7 and 19.9;
  // misaligned, 1 row a warp: 475 x 1346 2.2 and 2.45, 2048 x 498 3.1 and 3.8; 1.5 rows: 7168 x 250 3.6 and 6.0; from 2 rows on they are within
  // 5 % (10000 x 130 4.4 and 4.5, 2000 x 1111 4.5 and 4.6) or the shifting one is ahead (60000 x 205 22.7 and 17.0), and with a cold L2
  // it is by 9-78 % (2000 x 1111 7.6 and 6.0, 1000 x 3999 10.9 and 8.4).
  const int64_t slices = tfb_colsum_partials(rows, cols);
  const bool whole = aligned16(dy) && dy_ld % 8 == 0 && (!act || (aligned16(act) && act_ld % 8 == 0));
  const bool shift = !whole && rows >= 16 * slices;  // eight warps share a slice's rows
  const dim3 grid((unsigned)ceil_div(cols, shift ? GR_COLS : 256), (unsigned)slices);
#define TFB_GRAD_ROWS(...)                                                                                        \
  launch_overlapped(__VA_ARGS__, grid, dim3(256), 0, st, (const T*)dy, (const T*)act, (T*)dz, sums ? partials : nullptr, rows, \
                    (int)cols, dy_ld, act_ld, dz_ld)
  TFB_DISPATCH_16(dtype, T, {
    if (!shift) TFB_GRAD_ROWS(grad_rows_kernel<T>);
    else if (act) TFB_GRAD_ROWS((grad_rows_shift_kernel<T, true>));
    else TFB_GRAD_ROWS((grad_rows_shift_kernel<T, false>));
    const int rc = launched("grad_rows");
    if (rc || !sums) return rc;
    return finalize_partials<T>(partials, n_partials, (int)cols, (int)cols, sums, nullptr, st, 0);
  })
#undef TFB_GRAD_ROWS
}

extern "C" int tfb_relu_bwd(const void* dy, const void* act, void* dz, int64_t n, int dtype,
                            void* stream) {
  TFB_REQUIRE(n >= 0, "relu_bwd: negative size");
  if (n == 0) return TFB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = n % 8 == 0 && aligned16(dy) && aligned16(act) && aligned16(dz);
  TFB_DISPATCH_16(dtype, T, {
    if (vec) {
      const int64_t nvec = n / 8;
      const unsigned grid = (unsigned)(ceil_div(nvec, 256) < 148 * 16 ? ceil_div(nvec, 256) : 148 * 16);
      launch_overlapped(relu_bwd_vec_kernel<T>, dim3(grid), dim3(256), 0, st, (const uint4*)dy, (const uint4*)act, (uint4*)dz, nvec);
    } else {
      const unsigned grid = (unsigned)(ceil_div(n, 256) < 148 * 16 ? ceil_div(n, 256) : 148 * 16);
      launch_overlapped(relu_bwd_scalar_kernel<T>, dim3(grid), dim3(256), 0, st, (const T*)dy, (const T*)act, (T*)dz, n);
    }
  })
  return launched("relu_bwd");
}

extern "C" int64_t tfb_colsum_partials(int64_t rows, int64_t cols) {
  // enough row slices to fill the machine given ceil(cols/256) column CTAs, four of them per SM (what grad_rows_shift_kernel makes of it is
  // its 248 columns, and three per SM with a mask: its grid then runs a few CTAs, or a third of them, past a wave)
  const int64_t col_ctas = ceil_div(cols, 256);
  int64_t n = ceil_div(148 * 4, col_ctas);
  const int64_t max_n = ceil_div(rows, 8);
  if (n > max_n) n = max_n;
  return n < 1 ? 1 : n;
}

extern "C" int tfb_colsum(const void* x, void* out, float* partials, int64_t n_partials,
                          int64_t rows, int64_t cols, int64_t x_ld, int dtype, void* stream) {
  TFB_REQUIRE(rows > 0 && cols > 0 && cols < (1 << 30), "colsum: bad shape");
  TFB_REQUIRE(x_ld >= cols, "colsum: row stride smaller than cols");
  TFB_REQUIRE(n_partials == tfb_colsum_partials(rows, cols),
              "colsum: scratch must hold tfb_colsum_partials() rows");
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = cols % 8 == 0 && x_ld % 8 == 0 && aligned16(x);
  dim3 grid((unsigned)ceil_div(cols, 256), (unsigned)n_partials);
  TFB_DISPATCH_16(dtype, T, {
    if (vec) launch_overlapped(colsum_kernel<T, true>, dim3(grid), dim3(256), 0, st, (const T*)x, partials, rows, (int)cols, x_ld);
    else launch_overlapped(colsum_kernel<T, false>, dim3(grid), dim3(256), 0, st, (const T*)x, partials, rows, (int)cols, x_ld);
    int rc = launched("colsum");
    if (rc) return rc;
    return finalize_partials<T>(partials, n_partials, (int)cols, (int)cols, out, out, st, 0);
  })
}
