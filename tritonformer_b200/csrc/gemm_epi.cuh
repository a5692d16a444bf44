// Epilogue shared by the tcgen05 GEMM kernels: a warp turns its 32 rows x (64 STEPS) columns of the accumulator in tensor
// memory into 16-bit output, 64 columns (one swizzled 32 x 64 box in shared memory, one TMA store) at a time.
//
// A tile's epilogue runs a few times per CTA, so what it costs is latencies and the fetching of its instructions: unrolled over 64
// columns with every option inside the innermost loop it took 2.4-3.4 k cycles per 64 columns whatever the options were (per-CTA time
// stamps, warm or cold); in rolled steps of 16 columns with each option behind one uniform branch 1.7 k, four latencies of tensor memory
// among them; with all 64 columns read at once and each option a pass over them behind its branch, less.  (Where different
// kernels follow each other with a cold L2, the longer code costs some of that again: a linear layer's three products of
// 1280 x 128 x 896 19.5 us with the rolled form, 22.2 so, with a warm L2 16.6 and 16.7.)  Products of M 2048, fp16, L2 hot, rolled and now:
// N 3072 K 768 with mask 14.2 and 12.4 us, without 12.4 and 11.8, N 2304 K 768 8.8 and 8.1, N 768 K 768 6.2 and 5.8; M 768 N 3072 K 2048
// 11.7 and 11.1; M 8192 N 1024 K 4096 55.8 and 54.
#pragma once
#include "gemm_sched.cuh"

namespace tfb {

template <typename T> struct EpiArgs {
  DirectOut<T> out;                       // also carries bias, relu, addend, mask and their pitches
  const CUtensorMap *tm_c, *tm_x;         // output box, addend / mask box
  uint8_t *stage_c, *stage_x;             // this warp's two 4 KB boxes
  uint64_t* x_full;                       // the addend / mask box has landed
  bool use_x, x_is_addend, direct;
  const T* mask_direct;                   // a mask beside an addend: read from global memory
};

// Adds this tile's partial sums (slots of the CTAs behind this one, `slot` = the first of them at this thread's row, in
// float4, `stride` float4 between slots) to the accumulator in tensor memory, in the order of the slots.
template <int STEPS>
__device__ __forceinline__ void add_partials(uint32_t taddr, const float4* slot, int64_t stride, int parts, int rows) {
#pragma unroll 1
  for (int st = 0; st < STEPS * 2; ++st) {
    uint32_t r[32];
    tmem_ld32(taddr + st * 32, r);
    tc_wait_ld();
#pragma unroll 1
    for (int c = 0; c < parts; ++c) {
      const float4* src = slot + c * stride + st * 8 * rows;
      float4 v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = __ldcg(src + e * rows);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        r[4 * e] = __float_as_uint(__uint_as_float(r[4 * e]) + v[e].x);
        r[4 * e + 1] = __float_as_uint(__uint_as_float(r[4 * e + 1]) + v[e].y);
        r[4 * e + 2] = __float_as_uint(__uint_as_float(r[4 * e + 2]) + v[e].z);
        r[4 * e + 3] = __float_as_uint(__uint_as_float(r[4 * e + 3]) + v[e].w);
      }
    }
    tmem_st32(taddr + st * 32, r);
  }
  tc_wait_st();
}

// Writes the accumulator's partial sums to this CTA's slot (same layout: [group of 4 columns][row]).
template <int STEPS>
__device__ __forceinline__ void store_partials(uint32_t taddr, float4* slot, int rows) {
#pragma unroll 1
  for (int st = 0; st < STEPS * 2; ++st) {
    uint32_t r[32];
    tmem_ld32(taddr + st * 32, r);
    tc_wait_ld();
    float4* dst = slot + st * 8 * rows;
#pragma unroll
    for (int e = 0; e < 8; ++e)
      __stcg(dst + e * rows, make_float4(__uint_as_float(r[4 * e]), __uint_as_float(r[4 * e + 1]),
                                         __uint_as_float(r[4 * e + 2]), __uint_as_float(r[4 * e + 3])));
  }
}

// One row's 16 columns from `col` on: bias, ReLU, addend or mask from the staged box (two 16-byte chunks at soff0 / soff1).
template <typename T>
__device__ __forceinline__ void finish16(const EpiArgs<T>& a, float (&f)[16], int row, int col, uint32_t soff0, uint32_t soff1) {
  const DirectOut<T>& o = a.out;
  if (o.bias) {
    if (col + 16 <= o.N) {
      float b[8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        unpack8<T>(__ldg(reinterpret_cast<const uint4*>(o.bias + col) + h), b);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[h * 8 + j] += b[j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (col + j < o.N) f[j] += Num<T>::to_f(o.bias[col + j]);
    }
  }
  if (o.relu) {
#pragma unroll
    for (int j = 0; j < 16; ++j) f[j] = fmaxf(f[j], 0.f);
  }
  if (a.use_x) {
    float x[16];
    {
      float t[8];
      unpack8<T>(*reinterpret_cast<const uint4*>(a.stage_x + soff0), t);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = t[j];
      unpack8<T>(*reinterpret_cast<const uint4*>(a.stage_x + soff1), t);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[8 + j] = t[j];
    }
    if (a.x_is_addend) {
#pragma unroll
      for (int j = 0; j < 16; ++j) f[j] += x[j];
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) f[j] = x[j] > 0.f ? f[j] : 0.f;
    }
  }
  if (a.mask_direct && row < o.M) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (col + j < o.N && !(Num<T>::to_f(a.mask_direct[(int64_t)row * o.ld_mask + col + j]) > 0.f)) f[j] = 0.f;
  }
}

// The whole epilogue of a warp's share of a tile.  `ok` turns false when a bounded wait ran out.
template <typename T>
__device__ __forceinline__ void epilogue_tile(const EpiArgs<T>& a, int steps, uint32_t taddr, int row0, int n0, int lane, uint32_t& x_phase,
                                              volatile int* abort_flag, int code, bool& ok) {
  if (a.direct) {
#pragma unroll 1
    for (int st = 0; st < steps * 2; ++st) {
      if (n0 + st * 32 >= a.out.N) break;
      uint32_t r[32];
      tmem_ld32(taddr + st * 32, r);
      tc_wait_ld();
      store_direct<T>(a.out, r, reinterpret_cast<float*>((st & 1) ? a.stage_x : a.stage_c), row0, n0 + st * 32, lane);
    }
    return;
  }
#pragma unroll 1
  for (int st = 0; st < steps; ++st) {
    const int col0 = n0 + st * 64;
    if (a.use_x) {
      if (!mbar_wait(a.x_full, x_phase, code, abort_flag)) { ok = false; return; }
      x_phase ^= 1;
    }
    // Without an addend the two boxes alternate, so only the store before the last has to have been read; with one, the
    // other box holds the addend.
    uint8_t* box = !a.use_x && (st & 1) ? a.stage_x : a.stage_c;
    if (lane == 0) {
      if (a.use_x) tma_store_wait_read();
      else tma_store_wait_read_but1();
    }
    __syncwarp();
    if (!a.mask_direct && (!a.out.bias || col0 + 64 <= a.out.N)) {
      // All 64 columns in flight at once.  (A mask beside an addend, or a bias that ends within the step: the rolled form below.)
      uint32_t r[64];
      tmem_ld64(taddr + st * 64, r);
      tc_wait_ld();
      if (a.out.bias) {
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          float b[8];
          unpack8<T>(__ldg(reinterpret_cast<const uint4*>(a.out.bias + col0) + v), b);
#pragma unroll
          for (int j = 0; j < 8; ++j) r[8 * v + j] = __float_as_uint(__uint_as_float(r[8 * v + j]) + b[j]);
        }
      }
      if (a.out.relu) {
#pragma unroll
        for (int j = 0; j < 64; ++j) r[j] = __float_as_uint(fmaxf(__uint_as_float(r[j]), 0.f));
      }
      if (a.use_x) {
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          float x[8];
          unpack8<T>(*reinterpret_cast<const uint4*>(a.stage_x + lane * 128 + ((v ^ (lane & 7)) << 4)), x);
          if (a.x_is_addend) {
#pragma unroll
            for (int j = 0; j < 8; ++j) r[8 * v + j] = __float_as_uint(__uint_as_float(r[8 * v + j]) + x[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) r[8 * v + j] = x[j] > 0.f ? r[8 * v + j] : 0u;
          }
        }
      }
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[8 * v + j]);
        *reinterpret_cast<uint4*>(box + lane * 128 + ((v ^ (lane & 7)) << 4)) = pack8<T>(f);
      }
    } else {
      uint32_t r[2][16];
      tmem_ld16(taddr + st * 64, r[0]);
#pragma unroll 1
      for (int c = 0; c < 4; c += 2) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          tc_wait_ld();
          if (c + u + 1 < 4) tmem_ld16(taddr + st * 64 + (c + u + 1) * 16, r[u ^ 1]);
          float f[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(r[u][j]);
          const int v = (c + u) * 2;  // 16-byte chunk of the row
          const uint32_t soff0 = lane * 128 + ((v ^ (lane & 7)) << 4), soff1 = lane * 128 + (((v + 1) ^ (lane & 7)) << 4);
          finish16<T>(a, f, row0 + lane, col0 + (c + u) * 16, soff0, soff1);
          float lo[8], hi[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            lo[j] = f[j];
            hi[j] = f[8 + j];
          }
          *reinterpret_cast<uint4*>(box + soff0) = pack8<T>(lo);
          *reinterpret_cast<uint4*>(box + soff1) = pack8<T>(hi);
        }
      }
    }
    fence_proxy_async_smem();  // staged output visible to the TMA unit; addend box reads are done
    __syncwarp();
    if (lane == 0) {
      if (col0 < a.out.N && row0 < a.out.M) tma_store_2d(a.tm_c, box, col0, row0);
      tma_store_commit();
      if (a.use_x && st + 1 < steps) {  // next box: the next step of this tile (step 0 of the next tile is issued by the caller)
        mbar_expect_tx(a.x_full, 4096);
        tma_load_2d(a.stage_x, a.tm_x, col0 + 64, row0, a.x_full);
      }
    }
  }
}

}  // namespace tfb
