// What the tcgen05 GEMM kernels share: the one-wave kernel's plan, element-wise output, and the one-CTA kernel's work
// distribution ("stream-K").
//
// A worker is a persistent CTA.  The first sk_tiles output tiles are cut along K into
// one equal, contiguous range of k-blocks per worker; the remaining tiles are handed out whole,
// round-robin, after that.  A worker whose range starts inside a tile computes a partial tile: it
// writes it (fp32) to its own workspace slot and raises the tile's arrival counter.  The worker that
// owns the tile's first k-blocks - the last piece of its own range, so the others are done long
// before - adds the partials in worker order and runs the epilogue.  The order of the sum is fixed, so
// results do not depend on timing.
#pragma once
#include "tc05.cuh"

namespace tfb {

// Plan of the one-wave kernel (gemm_tile_tc05.cu): tile width (0: not for it), workers that share a tile's contraction, and the
// cycles its model gives the product.
struct TilePlan {
  int bn, split;
  bool pair;  // on CTA pairs
  int64_t cycles;
  int code() const { return bn ? 1 + (bn / 64) * 2 + (pair ? 1 : 0) + 16 * split : 0; }  // for the debug interface
};
TilePlan gemm_tile_plan(int64_t M, int64_t N, int64_t K, bool b_mn, int sms);
TilePlan gemm_plan(int64_t M, int64_t N, int64_t K, bool b_mn);  // with the switches in force
int gemm_pair_plan(int64_t M, int64_t N, int64_t K, bool a_mn, bool b_mn, bool b_rows_64);  // the same for the pair kernel's tile width

constexpr int kFlagBytes = 8192;  // head of the workspace: arrival counters, zero between kernels

struct Segments {
  int kblocks, tiles, workers;
  int64_t it, hi;  // cursor and end of this worker's k-block range in the split region
  int next_tile;   // next whole tile
  __device__ Segments(int kblocks_, int tiles_, int sk_tiles, int workers_, int worker) {
    kblocks = kblocks_;
    tiles = tiles_;
    workers = workers_;
    const int64_t sk_iters = (int64_t)sk_tiles * kblocks;
    it = sk_iters * worker / workers;
    hi = sk_iters * (worker + 1) / workers;
    next_tile = sk_tiles + worker;
  }
  // Next segment: k-blocks [kb0, kb1) of `tile`.  kb0 > 0: a partial to hand over; kb0 == 0 and
  // kb1 < kblocks: the part that collects the others; otherwise a whole tile.
  __device__ bool next(int& tile, int& kb0, int& kb1) {
    if (it < hi) {
      tile = (int)(it / kblocks);
      kb0 = (int)(it % kblocks);
      const int64_t left = hi - it;
      kb1 = (left < kblocks - kb0) ? kb0 + (int)left : kblocks;
      it += kb1 - kb0;
      return true;
    }
    if (next_tile < tiles) {
      tile = next_tile;
      kb0 = 0;
      kb1 = kblocks;
      next_tile += workers;
      return true;
    }
    return false;
  }
};

// Number of workers after `worker` whose ranges reach into `tile` (their partials are added by it).
__device__ __forceinline__ int partials_expected(int tile, int kblocks, int sk_tiles, int workers, int worker) {
  const int64_t sk_iters = (int64_t)sk_tiles * kblocks;
  const int64_t tile_end = (int64_t)(tile + 1) * kblocks;
  int c = worker + 1;
  while (c < workers && sk_iters * c / workers < tile_end) ++c;
  return c - worker - 1;
}

// Bounded wait until *flag reaches `expect` (acquire).  Same limit and status word as mbar_wait.
__device__ __forceinline__ bool flag_wait(const int* flag, int expect, int code, volatile int* abort_flag) {
  const uint64_t t0 = global_ns();
  for (;;) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (v >= expect) return true;
    if (*abort_flag) return false;
    if (global_ns() - t0 > kWaitLimitNs) break;
    __nanosleep(64);
  }
  *abort_flag = 1;
  atomicCAS(&g_dev_status, 0, code);
  return false;
}

// Epilogue output that TMA boxes cannot carry (a row pitch that is no multiple of 16 bytes, an unaligned base): the
// 32 x 32 block of fp32 accumulators of a warp (thread = row) is turned through a 4 KB swizzled box in shared memory, so
// that a warp then touches consecutive elements of one row.  Bias, ReLU, addend and mask are applied there, coalesced as
// well, and the value is rounded once.
template <typename T> struct DirectOut {
  T* c;
  const T *bias, *addend, *mask;
  int64_t ldc, ld_addend, ld_mask;
  int M, N, relu;
};
template <typename T>
__device__ __forceinline__ void store_direct(const DirectOut<T>& o, const uint32_t (&r)[32], float* box, int row0, int col0,
                                             int lane) {
#pragma unroll
  for (int v = 0; v < 8; ++v)
    *reinterpret_cast<uint4*>(box + lane * 32 + ((v ^ (lane & 7)) << 2)) =
        make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
  __syncwarp();
  const int col = col0 + lane;
  const int rows = o.M - row0 < 32 ? o.M - row0 : 32;
  if (col < o.N) {
    const float b = o.bias ? Num<T>::to_f(o.bias[col]) : 0.f;
    T* c = o.c + (int64_t)row0 * o.ldc + col;
    const T* add = o.addend ? o.addend + (int64_t)row0 * o.ld_addend + col : nullptr;
    const T* mask = o.mask ? o.mask + (int64_t)row0 * o.ld_mask + col : nullptr;
#pragma unroll 8
    for (int i = 0; i < rows; ++i) {
      float f = box[i * 32 + (((lane >> 2) ^ (i & 7)) << 2) + (lane & 3)] + b;
      if (o.relu) f = fmaxf(f, 0.f);
      if (add) f += Num<T>::to_f(add[(int64_t)i * o.ld_addend]);
      if (mask && !(Num<T>::to_f(mask[(int64_t)i * o.ld_mask]) > 0.f)) f = 0.f;
      c[(int64_t)i * o.ldc] = Num<T>::from_f(f);
    }
  }
  __syncwarp();  // the box may be overwritten
}

}  // namespace tfb
