// tcgen05 GEMM for outputs that one wave of CTAs covers: one output tile per cluster, nothing persistent.
//
//   C[M,N] = mask(act(A·B + bias) + addend), same contract as gemm_tc05.cu.
//
// What bounds these products is the chain of latencies of ONE tile (first operands, last product, epilogue, store) and, for
// longer contractions, the operand traffic from the L2 (about 10-15 TB/s for the whole chip), so the kernel is built to
// keep that chain short and, where it matters, the tile wide:
//   - set-up and the block barrier come before griddepcontrol.wait, and so does an L2 prefetch of the first B tiles (the
//     weights, in a forward pass; a prefetch reads nothing that could be stale, L2 is where the writes land);
//   - a worker is one CTA (tile 128 x 64 or 128 x 128) or a CTA pair (256 x 128, 192 or 256, tcgen05 with cta_group::2: half
//     the operand bytes per flop at 256 x 256);
//   - the contraction is cut over the workers of a cluster (1, 2, 4 or 8), which exchange fp32 partial tiles through
//     distributed shared memory: each sums and finishes its share of the tile's columns, in rank order (the sum does not
//     depend on timing), a row per thread (through staging in the ring, so that a warp's stores are consecutive, was slower:
//     M 2048 N 768 K 3072 13.7 against 12.9 us).  Through a workspace in global memory with arrival counters the same exchange took 4-5 us;
//   - little code: the roles' loops are rolled, and a tile's last steps run once per CTA (see gemm_epi.cuh).
// Back to back, L2 hot, fp16, with the cluster's first barrier in its release form, one thread that sets everything up, no early
// addend and the rolled epilogue, and now: M 2048 N 768 K 768 6.9 and 6.0 us (with addend 7.5, 6.8), M 2048 N 768 K 3072 13.6 and 12.9 (with
// addend 17.2, 14.0), M 2048 N 2304 K 768 9.6 and 8.2, M 768 N 768 K 2048 8.8 and 8.1, M 64 N 768 K 3072 with addend 6.7 and 5.8.
// Warps: 0 TMA producer, 1 MMA issuer (of the pair's first CTA), then the epilogue.
#include "gemm_epi.cuh"
#include <string.h>
#include <type_traits>

namespace tfb {

extern std::atomic<int> g_gemm_debug;

constexpr int GT_M = 128;  // rows per CTA
constexpr int GT_K = 64;

bool gemm_needs_direct(const void* c, int64_t ldc, const void* bias, const void* addend, int64_t ld_addend, const void* mask,
                       int64_t ld_mask);

template <int BN, bool PAIR, bool B_MN> struct TileCfg {
  static constexpr int BC = PAIR ? BN / 2 : BN;         // columns of B that a CTA loads
  static constexpr int CHUNKS = (BC + 63) / 64;         // in 64-column boxes where B is MN-major
  static constexpr int A_BYTES = GT_M * GT_K * 2;
  static constexpr int B_BYTES = CHUNKS * 8192;
  static constexpr int LOAD_BYTES = A_BYTES + (B_MN ? B_BYTES : BC * 128);
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int EPI_WARPS = PAIR ? 8 : 4;        // one or two per TMEM lane quarter
  static constexpr int THREADS = 64 + 32 * EPI_WARPS;
  static constexpr int BOX_BYTES = 2 * EPI_WARPS * 4096;
  static constexpr int MAX_STAGES = 6;
  static constexpr int SMEM_LIMIT = 227 * 1024 - 512;
  static constexpr int TMEM_COLS = BN <= 64 ? 64 : BN <= 128 ? 128 : 256;
};

struct TileParams {
  void* C;
  const void *bias, *addend, *mask;
  int M, N, K;
  int64_t ldc, ld_addend, ld_mask;
  int relu, direct;
  int tiles_m;
  int split;    // workers per cluster, each with a share of K
  int stages;   // ring depth
};

__device__ __forceinline__ uint32_t gt_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t gt_map(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void gt_store_remote(uint32_t addr, const uint32_t* v) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void gt_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
// no memory ordering: 1.0-1.3 k cycles less than the release form at this point
__device__ __forceinline__ void gt_cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void gt_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void gt_cluster_sync() {
  gt_cluster_arrive();
  gt_cluster_wait();
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* m, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(m), "r"(c0), "r"(c1) : "memory");
}
// Pair forms: the load's bytes are counted on the barrier of the pair's first CTA; one commit arrives at both CTAs.
__device__ __forceinline__ void gt_load_pair(void* dst, const CUtensorMap* m, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(m), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void gt_mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void gt_commit_pair(uint64_t* bar, uint16_t ctas) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)), "h"(ctas)
               : "memory");
}

// Eight columns of one row straight to global memory (vectors where the pitches allow them).  Their addend and mask vectors are
// requested ahead (`Extra`).
struct Extra {
  uint4 add, mask;
};
template <typename T>
__device__ __forceinline__ void request_extra(const TileParams& p, Extra& x, int row, int col) {
  if (p.direct || row >= p.M || col + 8 > p.N) return;
  if (p.addend) x.add = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.addend) + (int64_t)row * p.ld_addend + col);
  if (p.mask) x.mask = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.mask) + (int64_t)row * p.ld_mask + col);
}
template <typename T>
__device__ __forceinline__ void finish_row8(const TileParams& p, float (&f)[8], const Extra& x, int row, int col) {
  if (row >= p.M || col >= p.N) return;
  const T *bias = reinterpret_cast<const T*>(p.bias), *addend = reinterpret_cast<const T*>(p.addend),
          *mask = reinterpret_cast<const T*>(p.mask);
  T* c = reinterpret_cast<T*>(p.C) + (int64_t)row * p.ldc + col;
  if (!p.direct && col + 8 <= p.N) {
    float t[8];
    if (bias) {
      unpack8<T>(__ldg(reinterpret_cast<const uint4*>(bias + col)), t);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += t[j];
    }
    if (p.relu) {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = fmaxf(f[j], 0.f);
    }
    if (addend) {
      unpack8<T>(x.add, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += t[j];
    }
    if (mask) {
      unpack8<T>(x.mask, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = t[j] > 0.f ? f[j] : 0.f;
    }
    *reinterpret_cast<uint4*>(c) = pack8<T>(f);
    return;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (col + j >= p.N) break;
    float v = f[j];
    if (bias) v += Num<T>::to_f(bias[col + j]);
    if (p.relu) v = fmaxf(v, 0.f);
    if (addend) v += Num<T>::to_f(addend[(int64_t)row * p.ld_addend + col + j]);
    if (mask && !(Num<T>::to_f(mask[(int64_t)row * p.ld_mask + col + j]) > 0.f)) v = 0.f;
    c[j] = Num<T>::from_f(v);
  }
}

template <typename T, int BN, bool PAIR, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(TileCfg<BN, PAIR, B_MN>::THREADS, 1)
    gemm_tile_tc05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmX, const TileParams p) {
  using Cfg = TileCfg<BN, PAIR, B_MN>;
  constexpr int WIDTH = PAIR ? 2 : 1;  // CTAs per worker
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t bars[2 * Cfg::MAX_STAGES + 1 + Cfg::EPI_WARPS];
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_word;
  uint64_t *full = bars, *empty = bars + Cfg::MAX_STAGES, *acc_full = bars + 2 * Cfg::MAX_STAGES, *x_full = acc_full + 1;
  volatile int* abort_flag = &abort_word;
  uint8_t* boxes = smem + p.stages * Cfg::STAGE_BYTES;  // [epilogue warp][2] staging boxes; with a split, the partial sums of
  float4* recv = reinterpret_cast<float4*>(boxes);      // the other workers instead

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (PAIR || p.split > 1) ? (int)gt_cluster_rank() : 0;
  const int part = rank / WIDTH, side = rank % WIDTH;  // which worker of the cluster, which CTA of the worker
  const int tile = (int)blockIdx.x / (WIDTH * p.split);
  const int m0 = (tile % p.tiles_m) * (GT_M * WIDTH) + side * GT_M;  // this CTA's rows
  const int n0 = (tile / p.tiles_m) * BN;
  const int nb = n0 + side * Cfg::BC;                                // this CTA's columns of B
  const int kblocks = (p.K + GT_K - 1) / GT_K;
  const int kb0 = kblocks * part / p.split, kb1 = kblocks * (part + 1) / p.split;

  // the three parts of the set-up run on warps of their own (on two of them, one part after the other: M 2048 N 768
  // K 3072 12.9, now 12.5 us, M 768 N 3072 K 2048 11.9 and 11.7, M 768 N 768 K 2048 8.0 and 7.8)
  if (warp == 2 && lane == 0) {
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(acc_full, 1);
    for (int i = 0; i < Cfg::EPI_WARPS; ++i) mbar_init(&x_full[i], 1);
    abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 3 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
#pragma unroll 1
    for (int kb = kb0; kb < kb1 && kb < kb0 + p.stages; ++kb) {
      if (B_MN) {
#pragma unroll
        for (int i = 0; i < Cfg::CHUNKS; ++i) tma_prefetch_2d(&tmB, nb + i * 64, kb * GT_K);
      } else {
        tma_prefetch_2d(&tmB, kb * GT_K, nb);
      }
    }
  }
  if (warp == 1) {
    __syncwarp();
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                   "r"((uint32_t)Cfg::TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      tmem_alloc(&tmem_holder, Cfg::TMEM_COLS);
    }
  }
  tc_fence_before();
  __syncthreads();
  // Every CTA of the cluster runs, with its barriers and tensor memory ready, before another one signals or writes to it.
  // (The barriers' initialisation has a fence of its own: the arrival orders nothing else.)
  if (PAIR || p.split > 1) {
    gt_cluster_arrive_relaxed();
    gt_cluster_wait();
  }
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  // everything above touches only this cluster's shared memory, tensor memory and kernel parameters (and the L2)
  grid_dependency_wait();
  allow_dependents();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
#pragma unroll 1
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, 0x100 | stage, abort_flag)) break;
        uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
        uint8_t* sb = sa + Cfg::A_BYTES;
        const int k0 = kb * GT_K;
        if (side == 0) mbar_expect_tx(&full[stage], WIDTH * Cfg::LOAD_BYTES);  // the first CTA's barrier counts both
        const uint32_t bar = PAIR ? gt_map(smem_u32(&full[stage]), (uint32_t)(rank & ~1)) : 0u;
        auto load = [&](void* dst, const CUtensorMap* m, int c0, int c1) {
          if (PAIR) gt_load_pair(dst, m, c0, c1, bar);
          else tma_load_2d(dst, m, c0, c1, &full[stage]);
        };
        if (A_MN) {
#pragma unroll
          for (int i = 0; i < GT_M / 64; ++i) load(sa + i * 8192, &tmA, m0 + i * 64, k0);
        } else {
          load(sa, &tmA, k0, m0);
        }
        if (B_MN) {
#pragma unroll
          for (int i = 0; i < Cfg::CHUNKS; ++i) load(sb + i * 8192, &tmB, nb + i * 64, k0);
        } else {
          load(sb, &tmB, k0, nb);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (side == 0) {
      // the whole warp runs the loop and one elected lane issues: the descriptors stay in uniform registers
      constexpr uint32_t idesc =
          instr_desc_f16(GT_M * WIDTH, BN, std::is_same<T, __nv_bfloat16>::value ? 1 : 0, A_MN ? 1 : 0, B_MN ? 1 : 0);
      const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
      const uint32_t s0 = smem_u32(smem);
      const uint16_t ctas = (uint16_t)(3u << (rank & ~1));
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
#pragma unroll 1
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], phase, 0x200 | stage, abort_flag))) { ok = false; break; }
        const uint32_t sa = s0 + stage * Cfg::STAGE_BYTES, sb = sa + Cfg::A_BYTES;
        const uint64_t ad = A_MN ? smem_desc_sw128(sa, 8192, 1024) : smem_desc_sw128(sa, 16, 1024);
        const uint64_t bd = B_MN ? smem_desc_sw128(sb, 8192, 1024) : smem_desc_sw128(sb, 16, 1024);
#pragma unroll
        for (int k = 0; k < GT_K / 16; ++k) {
          const uint64_t ak = desc_advance(ad, k * (A_MN ? 2048 : 32)), bk = desc_advance(bd, k * (B_MN ? 2048 : 32));
          if (elect_one()) {
            if (PAIR) gt_mma_pair(tb, ak, bk, idesc, ((kb - kb0) | k) ? 1u : 0u);
            else tc_mma_ss(tb, ak, bk, idesc, ((kb - kb0) | k) ? 1u : 0u);
          }
        }
        if (elect_one()) {
          if (PAIR) gt_commit_pair(&empty[stage], ctas);
          else tc_commit(&empty[stage]);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (ok && elect_one()) {
        if (PAIR) gt_commit_pair(acc_full, ctas);
        else tc_commit(acc_full);
      }
    }
    __syncwarp();
  } else {
    constexpr int HALVES = Cfg::EPI_WARPS / 4;  // warps per TMEM lane quarter: they share the columns
    const int q = warp & 3, ew = warp - 2, half = ew >> 2;
    const int row0 = m0 + q * 32;
    // an earlier kernel that gave up leaves the status set: then nothing is written
    const bool dead = *(volatile int*)&g_dev_status != 0;
    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
    if (p.split == 1) {
      constexpr int FIRST = (BN / 64 + HALVES - 1) / HALVES;  // 64-column steps of the first half; the rest is the second's
      const int col = half * FIRST * 64, steps = half == 0 ? FIRST : BN / 64 - FIRST;
      const bool use_x = !p.direct && (p.addend != nullptr || p.mask != nullptr);
      const EpiArgs<T> epi{{reinterpret_cast<T*>(p.C), reinterpret_cast<const T*>(p.bias), reinterpret_cast<const T*>(p.addend),
                            reinterpret_cast<const T*>(p.mask), p.ldc, p.ld_addend, p.ld_mask, p.M, p.N, p.relu},
                           &tmC, &tmX, boxes + ew * 8192, boxes + ew * 8192 + 4096, &x_full[ew], use_x, p.addend != nullptr,
                           p.direct != 0, (p.addend != nullptr && p.mask != nullptr) ? reinterpret_cast<const T*>(p.mask) : nullptr};
      if (use_x && !dead && lane == 0) {  // in flight while the main loop runs; waited for by epilogue_tile, or below
        mbar_expect_tx(&x_full[ew], 4096);
        tma_load_2d(epi.stage_x, &tmX, n0 + col, row0, &x_full[ew]);
      }
      uint32_t x_phase = 0;
      bool ok = true;
      ok = mbar_wait(acc_full, 0, 0x400, abort_flag);
      tc_fence_after();
      __syncwarp();
      if (PAIR) gt_cluster_arrive_relaxed();  // matched by the wait before the exit
      if (ok && !dead) {
        epilogue_tile<T>(epi, steps, taddr + col, row0, n0 + col, lane, x_phase, abort_flag, 0x500 | ew, ok);
      } else if (use_x && !dead) {  // no CTA leaves with a load into its shared memory on the way (a millisecond at most)
        const uint64_t t0 = global_ns();
        while (!mbar_try_wait(&x_full[ew], 0) && global_ns() - t0 < 1000000) {
        }
      }
      if (lane == 0) tma_store_wait_read();  // the boxes have been read; the kernel's end completes the writes
    } else {
      // Column slice r of the tile goes to worker r (the CTA of the same side): [source][group of 4 columns][row], so that the
      // 32 lanes of a warp write 512 contiguous bytes.  Sources are numbered without the receiver itself.  The columns of a
      // slice are shared by the HALVES warps of a lane quarter.
      // Eight columns at a time, with the next ones' addend on its way: what this costs is latencies and the fetching of its
      // instructions.  (32 columns at a time in the exchange and 16 behind it, in code of three times the size, was as fast or up to 5 % faster
      // in a loop over one product, but not where products follow each other: a linear layer's three of 1344 x 320 x 960 20.0 us
      // against 19.7, of 2048 x 1792 x 320 26.2 against 25.4, with a cold L2 27.0 against 25.2 and 33.5 against 31.0; the layer of
      // 8512 x 256 x 2624 85.5 against 77.6.)
      const int slice = BN / p.split, lo = half * (slice / HALVES), hi = lo + slice / HALVES;
      const int trow = q * 32 + lane, row = row0 + lane, first = n0 + part * slice;
      Extra ex;
      if (!dead) request_extra<T>(p, ex, row, first + lo);
      bool ok = mbar_wait(acc_full, 0, 0x400, abort_flag);
      tc_fence_after();
      if (ok) {
#pragma unroll 1
        for (int i = 1; i < p.split; ++i) {
          const int to = (part + i) % p.split;
          const int slot = part < to ? part : part - 1;
          const uint32_t dst = gt_map(smem_u32(recv + slot * (slice / 4) * GT_M + trow), (uint32_t)(to * WIDTH + side));
#pragma unroll 1
          for (int c = lo; c < hi; c += 8) {
            uint32_t v[8];
            tmem_ld8(taddr + to * slice + c, v);
            tc_wait_ld();
            gt_store_remote(dst + (c / 4) * GT_M * 16, v);
            gt_store_remote(dst + (c / 4 + 1) * GT_M * 16, v + 4);
          }
        }
      }
      __syncwarp();
      gt_cluster_sync();
      if (ok && !dead && *abort_flag == 0) {
#pragma unroll 1
        for (int c = lo; c < hi; c += 8) {
          uint32_t own[8];
          tmem_ld8(taddr + part * slice + c, own);
          float f[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = 0.f;
          tc_wait_ld();
#pragma unroll 1
          for (int r = 0; r < p.split; ++r) {  // in rank order
            float4 a, b;
            if (r == part) {
              a = make_float4(__uint_as_float(own[0]), __uint_as_float(own[1]), __uint_as_float(own[2]), __uint_as_float(own[3]));
              b = make_float4(__uint_as_float(own[4]), __uint_as_float(own[5]), __uint_as_float(own[6]), __uint_as_float(own[7]));
            } else {
              const float4* src = recv + ((r < part ? r : r - 1) * (slice / 4) + c / 4) * GT_M + trow;
              a = src[0];
              b = src[GT_M];
            }
            f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
            f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
          }
          finish_row8<T>(p, f, ex, row, first + c);
          if (c + 8 < hi) request_extra<T>(p, ex, row, first + c + 8);
        }
      }
    }
  }
  if (warp < 2) {  // the epilogue warps are in the middle of, or past, these
    if (p.split > 1) gt_cluster_sync();
    else if (PAIR) gt_cluster_arrive_relaxed();
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  // A pair's CTAs leave when both have seen the accumulator complete: nothing reads or signals the other one after that.
  // (With a split the exchange's barrier already says so.)
  if (PAIR && p.split == 1) gt_cluster_wait();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)Cfg::TMEM_COLS) : "memory");
    else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------- host side
template <typename T, int BN, bool PAIR, bool A_MN, bool B_MN>
static int launch_tile(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const CUtensorMap& tmX,
                       TileParams& p, int tiles, cudaStream_t st) {
  using Cfg = TileCfg<BN, PAIR, B_MN>;
  auto kern = gemm_tile_tc05_kernel<T, BN, PAIR, A_MN, B_MN>;
  static std::atomic<uint64_t> attr_done{0};
  if (int rc0 = ensure_dynamic_smem(kern, Cfg::SMEM_LIMIT, attr_done, "gemm_tile_tc05")) return rc0;
  // behind the ring: the staging boxes, or the partial tiles of split - 1 workers, a slice of the columns each
  const int tail = p.split > 1 ? GT_M * (BN / p.split) * (p.split - 1) * 4 : Cfg::BOX_BYTES;
  const int room = (Cfg::SMEM_LIMIT - 1024 - tail) / Cfg::STAGE_BYTES;
  if (p.stages > Cfg::MAX_STAGES) p.stages = Cfg::MAX_STAGES;
  if (p.stages > room) p.stages = room;
  const int workers = tiles * p.split, cluster = p.split * (PAIR ? 2 : 1);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(workers * (PAIR ? 2 : 1)));
  cfg.blockDim = dim3(Cfg::THREADS);
  cfg.dynamicSmemBytes = (size_t)(p.stages * Cfg::STAGE_BYTES + tail + 1024);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (!g_plain_launch.load(std::memory_order_relaxed)) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  (void)cudaLaunchKernelEx(&cfg, kern, tmA, tmB, tmC, tmX, static_cast<const TileParams&>(p));
  return launched("gemm_tile_tc05");
}

template <typename T, int BN, bool PAIR>
static int dispatch_tile(bool a_mn, bool b_mn, const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC,
                         const CUtensorMap& tmX, TileParams& p, int tiles, cudaStream_t st) {
  if (a_mn && b_mn) return launch_tile<T, BN, PAIR, true, true>(tmA, tmB, tmC, tmX, p, tiles, st);
  if (a_mn) return launch_tile<T, BN, PAIR, true, false>(tmA, tmB, tmC, tmX, p, tiles, st);
  if (b_mn) return launch_tile<T, BN, PAIR, false, true>(tmA, tmB, tmC, tmX, p, tiles, st);
  return launch_tile<T, BN, PAIR, false, false>(tmA, tmB, tmC, tmX, p, tiles, st);
}

// Cycles of the one-wave kernel for a plan: a fixed chain of latencies, the k-blocks of a CTA, the exchange of a split.  What
// a k-block costs is mostly what an SM can take in from the L2, about 62 bytes a cycle (measured over tiles, splits and
// contraction lengths: 24 KB 400-430 cycles, 32 KB 480-540, whatever the tensor core would need).
// (The fixed part, the per-column part and the exchange were fitted to an epilogue and a set-up that were slower than the present ones.)
static int64_t tile_cycles(int bn, bool pair, int split, bool b_mn, int64_t kblocks) {
  const int64_t bytes = 16384 + (pair ? (b_mn ? (bn / 2 + 63) / 64 * 8192 : bn / 2 * 128) : bn * 128);
  const int64_t mma = pair ? bn * 2 : bn * 2 + 60;
  const int64_t per = bytes / 60 > mma ? bytes / 60 : mma;
  return 5000 + (pair ? 1000 : 0) + bn * 8 + ceil_div(kblocks, split) * per + (split > 1 ? 1800 + 200 * split + bn * 8 : 0);
}

// CTAs that run at the same time in clusters of `cluster`, one CTA per SM (clusters do not fill every GPC: 16 clusters of 8
// took two waves here).  Asked from the runtime once per device and size.
static int cluster_room(int cluster, int sms) {
  if (cluster == 1) return sms;
  static std::atomic<int> known[64][9] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  int room = known[dev][cluster].load(std::memory_order_relaxed);
  if (room == 0) {
    auto kern = gemm_tile_tc05_kernel<__half, 128, true, false, false>;
    constexpr int smem = 160 * 1024;  // more than half of an SM's
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TileCfg<128, true, false>::SMEM_LIMIT);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)cluster * 64);
    cfg.blockDim = dim3(TileCfg<128, true, false>::THREADS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
      (void)cudaGetLastError();
      n = sms * 3 / 4 / cluster;
    }
    room = n * cluster;
    known[dev][cluster].store(room, std::memory_order_relaxed);
  }
  return room < sms ? room : sms;
}

TilePlan gemm_tile_plan(int64_t M, int64_t N, int64_t K, bool b_mn, int sms) {
  TilePlan best{0, 0, false, 0};
  const int64_t kblocks = ceil_div(K, GT_K);
  const int dbg = g_gemm_debug.load(), forced = (dbg >> 16) & 0xfff;  // tuning switch: a plan's code
  for (int pair = 0; pair <= 1; ++pair) {
    if (pair && (M <= GT_M || N < 64)) break;
    for (int bn = pair ? 128 : 64; bn <= (pair ? 256 : 128); bn += 64) {
      const int64_t tiles = ceil_div(M, pair ? 2 * GT_M : GT_M) * ceil_div(N, bn);
      for (int split = 1; split <= (pair ? 4 : 8); split *= 2) {
        const int cluster = split * (pair ? 2 : 1);
        if (kblocks < split || tiles * cluster > cluster_room(cluster, sms) || ((dbg & 1) && split > 1)) break;
        const TilePlan plan{bn, split, pair != 0, tile_cycles(bn, pair != 0, split, b_mn, kblocks)};
        if (forced && forced != plan.code()) continue;
        if (best.bn == 0 || plan.cycles < best.cycles) best = plan;
      }
    }
  }
  return best;
}

int gemm_tile_tc05(const TilePlan& plan, const void* a, const void* b, void* c, const void* bias, const void* addend,
                   int64_t ld_addend, const void* mask, int64_t ld_mask, int64_t M, int64_t N, int64_t K, int64_t a_sm,
                   int64_t a_sk, int64_t b_sk, int64_t b_sn, int64_t ldc, int relu, int dtype, cudaStream_t st) {
  const bool a_mn = (a_sk != 1), b_mn = (b_sk != 1);
  const bool direct = gemm_needs_direct(c, ldc, bias, addend, ld_addend, mask, ld_mask);
  CUtensorMap tmA, tmB, tmC, tmX;
  int rc;
  if (plan.split == 1 && !direct) {  // a split writes rows, not boxes
    uint64_t dims[2] = {(uint64_t)N, (uint64_t)M}, str[1] = {(uint64_t)ldc * 2};
    uint32_t box[2] = {64, 32};
    if ((rc = encode_tmap_sw128(&tmC, c, dtype, 2, dims, str, box))) return rc;
    const void* xp = addend ? addend : mask;
    str[0] = (uint64_t)(addend ? ld_addend : ld_mask) * 2;
    if (xp) { if ((rc = encode_tmap_sw128(&tmX, xp, dtype, 2, dims, str, box))) return rc; }
    else tmX = tmC;
  } else {
    memset(&tmC, 0, sizeof(tmC));
    tmX = tmC;
  }
  {
    uint64_t dims[2], str[1];
    uint32_t box[2];
    if (a_mn) { dims[0] = (uint64_t)M; dims[1] = (uint64_t)K; str[0] = (uint64_t)a_sk * 2; box[0] = 64; box[1] = GT_K; }
    else      { dims[0] = (uint64_t)K; dims[1] = (uint64_t)M; str[0] = (uint64_t)a_sm * 2; box[0] = GT_K; box[1] = GT_M; }
    if ((rc = encode_tmap_sw128(&tmA, a, dtype, 2, dims, str, box))) return rc;
    if (b_mn) { dims[0] = (uint64_t)N; dims[1] = (uint64_t)K; str[0] = (uint64_t)b_sk * 2; box[0] = 64; box[1] = GT_K; }
    else      { dims[0] = (uint64_t)K; dims[1] = (uint64_t)N; str[0] = (uint64_t)b_sn * 2; box[0] = GT_K; box[1] = (uint32_t)(plan.pair ? plan.bn / 2 : plan.bn); }
    if ((rc = encode_tmap_sw128(&tmB, b, dtype, 2, dims, str, box))) return rc;
  }
  TileParams p;
  p.C = c; p.bias = bias; p.addend = addend; p.mask = mask;
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.ldc = ldc; p.ld_addend = ld_addend; p.ld_mask = ld_mask;
  p.relu = relu; p.direct = direct;
  p.tiles_m = (int)ceil_div(M, plan.pair ? 2 * GT_M : GT_M);
  p.split = plan.split;
  const int64_t per_cta = ceil_div(ceil_div(K, GT_K), plan.split);
  const int tiles = p.tiles_m * (int)ceil_div(N, plan.bn);
  p.stages = (int)(per_cta < 64 ? per_cta : 64);  // cut to the shared memory there is at launch
  TFB_DISPATCH_16(dtype, T, {
    if (!plan.pair && plan.bn == 64) return dispatch_tile<T, 64, false>(a_mn, b_mn, tmA, tmB, tmC, tmX, p, tiles, st);
    if (!plan.pair) return dispatch_tile<T, 128, false>(a_mn, b_mn, tmA, tmB, tmC, tmX, p, tiles, st);
    if (plan.bn == 128) return dispatch_tile<T, 128, true>(a_mn, b_mn, tmA, tmB, tmC, tmX, p, tiles, st);
    if (plan.bn == 192) return dispatch_tile<T, 192, true>(a_mn, b_mn, tmA, tmB, tmC, tmX, p, tiles, st);
    return dispatch_tile<T, 256, true>(a_mn, b_mn, tmA, tmB, tmC, tmX, p, tiles, st);
  })
}

}  // namespace tfb
