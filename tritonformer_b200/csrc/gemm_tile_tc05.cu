// tcgen05 GEMM for outputs that one wave of CTAs covers: one 128 x BN tile per cluster of S CTAs, nothing persistent.
//
//   C[M,N] = mask(act(A·B + bias) + addend), same contract as gemm_tc05.cu.
//
// What bounds these products is the chain of latencies of ONE tile (first operands, last product, epilogue, store), not
// throughput, so the kernel is built to keep that chain short:
//   - set-up and the block barrier come before griddepcontrol.wait, and so does an L2 prefetch of the first B tiles (the
//     weights, in a forward pass; a prefetch reads nothing that could be stale, L2 is where the writes land);
//   - the contraction is cut over the S CTAs of a cluster (1, 2, 4 or 8), which exchange fp32 partial tiles through
//     distributed shared memory: each CTA sums and finishes BN / S columns of the tile, in rank order (the sum does not
//     depend on timing).  Through a workspace in global memory with arrival counters the same exchange took 4-5 us;
//   - short rolled code everywhere (see gemm_epi.cuh).
// Warps: 0 TMA producer, 1 MMA issuer, 2-5 epilogue.  fp16 512 x 256 x 1024: see the table in the launch rule below.
#include "gemm_epi.cuh"
#include <string.h>
#include <type_traits>

namespace tfb {

constexpr int GT_M = 128;
constexpr int GT_K = 64;
constexpr int GT_THREADS = 192;

bool gemm_needs_direct(const void* c, int64_t ldc, const void* bias, const void* addend, int64_t ld_addend, const void* mask,
                       int64_t ld_mask);

template <int BN> struct TileCfg {
  static constexpr int A_BYTES = GT_M * GT_K * 2;
  static constexpr int B_BYTES = BN * GT_K * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int MAX_STAGES = (BN == 64) ? 6 : 5;
  static constexpr int BOX_BYTES = 8 * 4096;  // two staging boxes per epilogue warp
};

struct TileParams {
  void* C;
  const void *bias, *addend, *mask;
  int M, N, K;
  int64_t ldc, ld_addend, ld_mask;
  int relu, direct;
  int tiles_m;
  int split;    // CTAs per cluster, each with a share of K
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
__device__ __forceinline__ void gt_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* m, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(m), "r"(c0), "r"(c1) : "memory");
}

// Eight columns of one row straight to global memory (vectors where the pitches allow them).
template <typename T>
__device__ __forceinline__ void finish_row8(const TileParams& p, float (&f)[8], int row, int col) {
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
      unpack8<T>(*reinterpret_cast<const uint4*>(addend + (int64_t)row * p.ld_addend + col), t);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += t[j];
    }
    if (mask) {
      unpack8<T>(*reinterpret_cast<const uint4*>(mask + (int64_t)row * p.ld_mask + col), t);
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

template <typename T, int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(GT_THREADS) gemm_tile_tc05_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                    const __grid_constant__ CUtensorMap tmB,
                                                                    const __grid_constant__ CUtensorMap tmC,
                                                                    const __grid_constant__ CUtensorMap tmX,
                                                                    const TileParams p) {
  using Cfg = TileCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t bars[2 * Cfg::MAX_STAGES + 5];
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_word;
  uint64_t *full = bars, *empty = bars + Cfg::MAX_STAGES, *acc_full = bars + 2 * Cfg::MAX_STAGES, *x_full = acc_full + 1;
  volatile int* abort_flag = &abort_word;
  uint8_t* boxes = smem + p.stages * Cfg::STAGE_BYTES;                  // [4 warps][2] staging boxes; with a split, the
  float4* recv = reinterpret_cast<float4*>(boxes);                      // partials of the other CTAs instead

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = p.split > 1 ? (int)gt_cluster_rank() : 0;
  const int tile = (int)blockIdx.x / p.split;
  const int m0 = (tile % p.tiles_m) * GT_M, n0 = (tile / p.tiles_m) * BN;
  const int kblocks = (p.K + GT_K - 1) / GT_K;
  const int kb0 = kblocks * rank / p.split, kb1 = kblocks * (rank + 1) / p.split;

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(acc_full, 1);
    for (int i = 0; i < 4; ++i) mbar_init(&x_full[i], 1);
    abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
#pragma unroll 1
    for (int kb = kb0; kb < kb1 && kb < kb0 + p.stages; ++kb) {
      if (B_MN) {
#pragma unroll
        for (int i = 0; i < BN / 64; ++i) tma_prefetch_2d(&tmB, n0 + i * 64, kb * GT_K);
      } else {
        tma_prefetch_2d(&tmB, kb * GT_K, n0);
      }
    }
  }
  if (warp == 1) {
    __syncwarp();
    tmem_alloc(&tmem_holder, BN);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  // first use of the cluster barrier: every CTA of the cluster runs before another one writes to its shared memory
  if (p.split > 1) gt_cluster_arrive();
  // everything above touches only this CTA's shared memory, tensor memory and kernel parameters (and the L2)
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
        mbar_expect_tx(&full[stage], Cfg::STAGE_BYTES);
        const int k0 = kb * GT_K;
        if (A_MN) {
#pragma unroll
          for (int i = 0; i < GT_M / 64; ++i) tma_load_2d(sa + i * 8192, &tmA, m0 + i * 64, k0, &full[stage]);
        } else {
          tma_load_2d(sa, &tmA, k0, m0, &full[stage]);
        }
        if (B_MN) {
#pragma unroll
          for (int i = 0; i < BN / 64; ++i) tma_load_2d(sb + i * 8192, &tmB, n0 + i * 64, k0, &full[stage]);
        } else {
          tma_load_2d(sb, &tmB, k0, n0, &full[stage]);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // the whole warp runs the loop and one elected lane issues: the descriptors stay in uniform registers
    constexpr uint32_t idesc = instr_desc_f16(GT_M, BN, std::is_same<T, __nv_bfloat16>::value ? 1 : 0, A_MN ? 1 : 0, B_MN ? 1 : 0);
    const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t s0 = smem_u32(smem);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
#pragma unroll 1
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], phase, 0x200 | stage, abort_flag))) { ok = false; break; }
      tc_fence_after();
      const uint32_t sa = s0 + stage * Cfg::STAGE_BYTES, sb = sa + Cfg::A_BYTES;
      const uint64_t ad = A_MN ? smem_desc_sw128(sa, 8192, 1024) : smem_desc_sw128(sa, 16, 1024);
      const uint64_t bd = B_MN ? smem_desc_sw128(sb, 8192, 1024) : smem_desc_sw128(sb, 16, 1024);
#pragma unroll
      for (int k = 0; k < GT_K / 16; ++k)
        if (elect_one())
          tc_mma_ss(tb, desc_advance(ad, k * (A_MN ? 2048 : 32)), desc_advance(bd, k * (B_MN ? 2048 : 32)), idesc,
                    ((kb - kb0) | k) ? 1u : 0u);
      if (elect_one()) tc_commit(&empty[stage]);
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
    if (ok && elect_one()) tc_commit(acc_full);
    __syncwarp();
  } else {
    const int q = warp & 3, ew = warp - 2;
    const int row0 = m0 + q * 32;
    // an earlier kernel that gave up leaves the status set: then nothing is written
    const bool dead = *(volatile int*)&g_dev_status != 0;
    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
    if (p.split == 1) {
      const bool use_x = !p.direct && (p.addend != nullptr || p.mask != nullptr);
      const EpiArgs<T> epi{{reinterpret_cast<T*>(p.C), reinterpret_cast<const T*>(p.bias), reinterpret_cast<const T*>(p.addend),
                            reinterpret_cast<const T*>(p.mask), p.ldc, p.ld_addend, p.ld_mask, p.M, p.N, p.relu},
                           &tmC, &tmX, boxes + ew * 8192, boxes + ew * 8192 + 4096, &x_full[ew], use_x, p.addend != nullptr,
                           p.direct != 0, (p.addend != nullptr && p.mask != nullptr) ? reinterpret_cast<const T*>(p.mask) : nullptr};
      if (use_x && lane == 0) {  // in flight while the main loop runs
        mbar_expect_tx(&x_full[ew], 4096);
        tma_load_2d(epi.stage_x, &tmX, n0, row0, &x_full[ew]);
      }
      bool ok = mbar_wait(acc_full, 0, 0x400, abort_flag);
      tc_fence_after();
      uint32_t x_phase = 0;
      if (ok && !dead) epilogue_tile<T, BN / 64>(epi, taddr, row0, n0, lane, x_phase, abort_flag, 0x500 | ew, ok);
      if (lane == 0) tma_store_wait_all();
    } else {
      bool ok = mbar_wait(acc_full, 0, 0x400, abort_flag);
      tc_fence_after();
      // column slice r of the tile goes to the CTA of rank r: [source][group of 4 columns][row], so that the 32 lanes of a
      // warp write 512 contiguous bytes
      const int slice = BN / p.split;
      const int trow = q * 32 + lane;
      __syncwarp();
      gt_cluster_wait();
      if (ok) {
#pragma unroll 1
        for (int i = 1; i < p.split; ++i) {
          const int to = (rank + i) % p.split;
          const uint32_t dst = gt_map(smem_u32(recv + (rank * (slice / 4)) * GT_M + trow), (uint32_t)to);
#pragma unroll 1
          for (int c = 0; c < slice; c += 8) {
            uint32_t v[8];
            tmem_ld8(taddr + to * slice + c, v);
            tc_wait_ld();
            gt_store_remote(dst + (c / 4) * GT_M * 16, v);
            gt_store_remote(dst + (c / 4 + 1) * GT_M * 16, v + 4);
          }
        }
      }
      __syncwarp();
      gt_cluster_arrive();
      gt_cluster_wait();
      if (ok && !dead && *abort_flag == 0) {
#pragma unroll 1
        for (int c = 0; c < slice; c += 8) {
          uint32_t own[8];
          tmem_ld8(taddr + rank * slice + c, own);
          tc_wait_ld();
          float f[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = 0.f;
#pragma unroll 1
          for (int r = 0; r < p.split; ++r) {
            float4 lo, hi;
            if (r == rank) {
              lo = make_float4(__uint_as_float(own[0]), __uint_as_float(own[1]), __uint_as_float(own[2]), __uint_as_float(own[3]));
              hi = make_float4(__uint_as_float(own[4]), __uint_as_float(own[5]), __uint_as_float(own[6]), __uint_as_float(own[7]));
            } else {
              const float4* src = recv + (r * (slice / 4) + c / 4) * GT_M + trow;
              lo = src[0];
              hi = src[GT_M];
            }
            f[0] += lo.x; f[1] += lo.y; f[2] += lo.z; f[3] += lo.w;
            f[4] += hi.x; f[5] += hi.y; f[6] += hi.z; f[7] += hi.w;
          }
          finish_row8<T>(p, f, row0 + lane, n0 + rank * slice + c);
        }
      }
    }
  }
  if (p.split > 1 && warp < 2) {  // the epilogue warps passed both above
    gt_cluster_wait();
    gt_cluster_arrive();
    gt_cluster_wait();
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
}

// ------------------------------------------------------------------------------- host side
template <typename T, int BN, bool A_MN, bool B_MN>
static int launch_tile(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const CUtensorMap& tmX,
                       const TileParams& p, int tiles, cudaStream_t st) {
  using Cfg = TileCfg<BN>;
  auto kern = gemm_tile_tc05_kernel<T, BN, A_MN, B_MN>;
  static std::atomic<uint64_t> attr_done{0};
  constexpr int most = Cfg::MAX_STAGES * Cfg::STAGE_BYTES + GT_M * BN * 4 + 1024;
  static_assert(most <= 227 * 1024 - 512, "shared memory");
  if (int rc0 = ensure_dynamic_smem(kern, most, attr_done, "gemm_tile_tc05")) return rc0;
  // with a split the partials of split - 1 CTAs, BN / split columns each (slots of all ranks are laid out, one unused)
  const int tail = p.split > 1 ? GT_M * BN * 4 : Cfg::BOX_BYTES;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * p.split));
  cfg.blockDim = dim3(GT_THREADS);
  cfg.dynamicSmemBytes = (size_t)(p.stages * Cfg::STAGE_BYTES + tail + 1024);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (!g_plain_launch.load(std::memory_order_relaxed)) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (p.split > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)p.split;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  (void)cudaLaunchKernelEx(&cfg, kern, tmA, tmB, tmC, tmX, p);
  return launched("gemm_tile_tc05");
}

template <typename T, int BN>
static int dispatch_tile(bool a_mn, bool b_mn, const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC,
                         const CUtensorMap& tmX, const TileParams& p, int tiles, cudaStream_t st) {
  if (a_mn && b_mn) return launch_tile<T, BN, true, true>(tmA, tmB, tmC, tmX, p, tiles, st);
  if (a_mn) return launch_tile<T, BN, true, false>(tmA, tmB, tmC, tmX, p, tiles, st);
  if (b_mn) return launch_tile<T, BN, false, true>(tmA, tmB, tmC, tmX, p, tiles, st);
  return launch_tile<T, BN, false, false>(tmA, tmB, tmC, tmX, p, tiles, st);
}

// The tile kernel's plan for a product: BN and the split that the model below puts lowest, or bn = 0 when the output needs
// more than one wave of CTAs.  Cycles of a CTA: a fixed chain of latencies, its k-blocks at the rate shared memory feeds the
// tensor core (24 and 32 KB per k-block at 128 B/clk), the exchange of a split.
TilePlan gemm_tile_plan(int64_t M, int64_t N, int64_t K, int sms) {
  TilePlan best{0, 0, 0};
  const int64_t tm = ceil_div(M, GT_M), kblocks = ceil_div(K, GT_K);
  for (int bn = 64; bn <= 128; bn *= 2) {
    const int64_t tiles = tm * ceil_div(N, bn);
    if (tiles > sms) continue;
    for (int split = 1; split <= 8; split *= 2) {
      // clusters of 4 and 8 CTAs do not fill every GPC
      if (tiles * split > (split <= 2 ? sms : split == 4 ? sms * 15 / 16 : sms * 7 / 8) || kblocks < split) break;
      const int64_t cycles = 3000 + ceil_div(kblocks, split) * (bn == 64 ? 200 : 270) + (split > 1 ? 1000 + 100 * split : bn == 128 ? 600 : 0);
      if (best.bn == 0 || cycles < best.cycles) best = TilePlan{bn, split, cycles};
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
    else      { dims[0] = (uint64_t)K; dims[1] = (uint64_t)N; str[0] = (uint64_t)b_sn * 2; box[0] = GT_K; box[1] = (uint32_t)plan.bn; }
    if ((rc = encode_tmap_sw128(&tmB, b, dtype, 2, dims, str, box))) return rc;
  }
  TileParams p;
  p.C = c; p.bias = bias; p.addend = addend; p.mask = mask;
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.ldc = ldc; p.ld_addend = ld_addend; p.ld_mask = ld_mask;
  p.relu = relu; p.direct = direct;
  p.tiles_m = (int)ceil_div(M, GT_M);
  p.split = plan.split;
  const int64_t per_cta = ceil_div(ceil_div(K, GT_K), plan.split);
  const int tiles = p.tiles_m * (int)ceil_div(N, plan.bn);
  const int most = plan.bn == 64 ? TileCfg<64>::MAX_STAGES : TileCfg<128>::MAX_STAGES;
  p.stages = (int)(per_cta < most ? per_cta : most);
  TFB_DISPATCH_16(dtype, T, {
    if (plan.bn == 64) return dispatch_tile<T, 64>(a_mn, b_mn, tmA, tmB, tmC, tmX, p, tiles, st);
    return dispatch_tile<T, 128>(a_mn, b_mn, tmA, tmB, tmC, tmX, p, tiles, st);
  })
}

}  // namespace tfb
