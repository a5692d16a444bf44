// tcgen05 GEMM on CTA pairs (cta_group::2) for sm_100a: one 256 x 256 or 256 x 192 output tile per pair of SMs.
//
// Same contract as gemm_tc05.cu (C = mask(act(A·B + bias) + addend), either operand K- or MN-major),
// for outputs large enough to give every pair of SMs tiles.  Why a second kernel: the one-CTA kernel
// moves 48 KB of operands from L2 to shared memory per 128 x 256 x 64 block of work and is bound by
// that traffic; here the two CTAs of a cluster each load their own 128 rows of A and HALF of the B
// tile (32 KB per CTA for the same work), and the pair's tensor cores read B from both halves.
//
// Per CTA (both CTAs of the pair run the same code; "leader" = cluster rank 0):
//   warp 0   : TMA producer - its A rows and its half of B into a 5-stage ring; the copies signal the
//              LEADER's full barrier (cp.async.bulk.tensor with .cta_group::2, no multicast)
//   warp 1   : leader only: issues tcgen05.mma.cta_group::2 (M 256 over the pair, N 256 or 192, K 16) and
//              commits ring slots / finished accumulators to the barriers of BOTH CTAs
//   warps 2-9: epilogue of this CTA's 128 rows from its own TMEM (two accumulator buffers), as in the
//              one-CTA kernel; the buffer is handed back by an arrival on the leader's barrier
// Every wait is bounded (mbar_wait); the two cluster-wide barriers (after set-up, before exit) are
// reached unconditionally by both CTAs.
#include "gemm_epi.cuh"
#include <string.h>
#include <type_traits>

namespace tfb {

bool gemm_needs_direct(const void* c, int64_t ldc, const void* bias, const void* addend, int64_t ld_addend, const void* mask,
                       int64_t ld_mask);

constexpr int GP_M = 128;    // rows per CTA
constexpr int GP_K = 64;
constexpr int GP_EPI_WARPS = 8;  // 4, or 8 (two warps per TMEM lane quarter, half of the columns each)
constexpr int GP_THREADS = 64 + 32 * GP_EPI_WARPS;
constexpr int GP_A_BYTES = GP_M * GP_K * 2;
constexpr int GP_EPI_BYTES = GP_EPI_WARPS * 4096;  // one staging box per epilogue warp
template <int BN> struct PairCfg {   // BN: columns per pair tile, 192 or 256
  static constexpr int NH = BN / 2;  // columns of B loaded per CTA
  static constexpr int STAGES = 5;
  static constexpr int B_BYTES = NH * GP_K * 2;
  static constexpr int STAGE_BYTES = GP_A_BYTES + B_BYTES;
  // B contiguous along N comes in boxes of BOX columns by GP_K rows.  Half of 192 columns is no multiple of 64, so its boxes
  // are 32 columns (64 bytes) wide, with the 64-byte swizzle.
  static constexpr int BOX = NH % 64 == 0 ? 64 : 32;
  static constexpr int FIRST = (BN / 64 + 1) / 2;  // 64-column steps of the first half of the epilogue warps
  static constexpr int OFF_EPI_C = STAGES * STAGE_BYTES;
  static constexpr int OFF_EPI_X = OFF_EPI_C + GP_EPI_BYTES;
  static constexpr int OFF_BAR = OFF_EPI_X + GP_EPI_BYTES;
  static constexpr int SMEM_BYTES = OFF_BAR + 1024 + 256;
  static_assert(NH % BOX == 0 && STAGE_BYTES % 1024 == 0 && SMEM_BYTES <= 227 * 1024, "tile width");
};
constexpr int GP_TMEM_COLS = 512;

struct PairParams {
  void* C;
  const void* bias;
  const void* addend;
  const void* mask;
  int M, N, K;
  int64_t ldc, ld_addend, ld_mask;
  int relu;
  int direct;          // C, addend, mask or bias cannot go through TMA boxes: element-wise coalesced stores (store_direct)
  int tiles_m, tiles_n;  // in 256 x BN pair tiles
};

// ---- cluster / pair primitives ------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* holder, uint32_t ncols) {  // one warp in each CTA
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Tile load into this CTA's shared memory whose completion is counted on a barrier that may live in
// the peer CTA (bar_cluster_addr is a shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, int c0, int c1,
                                                 uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(m), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tc_mma_ss_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One arrival on the barrier at this shared-memory offset in BOTH CTAs of the pair once every MMA
// issued so far by this thread has retired.
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(smem_u32(bar)), "h"((uint16_t)3)
      : "memory");
}

template <typename T, int BN, bool A_MN, bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
    gemm_pair_tc05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmX,
                          const PairParams p) {
  using Cfg = PairCfg<BN>;
  constexpr int GP_STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* full = bars;                       // [STAGES] both producers -> leader's MMA (leader's copy is used)
  uint64_t* empty = bars + GP_STAGES;          // [STAGES] leader's MMA -> each CTA's producer
  uint64_t* acc_full = bars + 2 * GP_STAGES;   // [2] leader's MMA -> each CTA's epilogue
  uint64_t* acc_empty = acc_full + 2;          // [2] both epilogues -> leader's MMA (leader's copy is used)
  uint64_t* x_full = acc_empty + 2;            // [4] addend / mask box of an epilogue warp landed
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(x_full + GP_EPI_WARPS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < GP_STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 2 * GP_EPI_WARPS);  // the epilogue warps of both CTAs
    }
    for (int i = 0; i < GP_EPI_WARPS; ++i) mbar_init(&x_full[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    __syncwarp();
    tmem_alloc_pair(tmem_holder, GP_TMEM_COLS);
  }
  tc_fence_before();
  __syncthreads();
  // The peer's barriers and tensor memory are ready before anything is signalled across the pair.  (The barriers'
  // initialisation has a fence of its own: the arrival orders nothing else, and costs 1 k cycles less that way.)
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  // set-up above is local to the pair and may overlap the previous kernel's tail; global memory comes after
  grid_dependency_wait();
  allow_dependents();

  const int num_tiles = p.tiles_m * p.tiles_n;
  const int kblocks = (p.K + GP_K - 1) / GP_K;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < num_tiles; tile += num_pairs) {
        const int m0 = (tile % p.tiles_m) * (2 * GP_M) + (int)rank * GP_M;  // this CTA's rows
        const int n0 = (tile / p.tiles_m) * BN + (int)rank * Cfg::NH;       // this CTA's half of B
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, 0x700 | stage, abort_flag)) { ok = false; break; }
          uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + GP_A_BYTES;
          // the leader's barrier counts the bytes of both CTAs
          if (leader) mbar_expect_tx(&full[stage], 2 * Cfg::STAGE_BYTES);
          const uint32_t bar = map_to_cta(smem_u32(&full[stage]), 0);
          const int k0 = kb * GP_K;
          if (A_MN) {
#pragma unroll
            for (int i = 0; i < GP_M / 64; ++i) tma_load_2d_pair(sa + i * 8192, &tmA, m0 + i * 64, k0, bar);
          } else {
            tma_load_2d_pair(sa, &tmA, k0, m0, bar);
          }
          if (B_MN) {
#pragma unroll
            for (int i = 0; i < Cfg::NH / Cfg::BOX; ++i)
              tma_load_2d_pair(sb + i * (Cfg::BOX * GP_K * 2), &tmB, n0 + i * Cfg::BOX, k0, bar);
          } else {
            tma_load_2d_pair(sb, &tmB, k0, n0, bar);
          }
          if (++stage == GP_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------------- MMA issuer (leader only)
    // The whole warp runs the loop and one elected lane issues each instruction: warp-uniform code keeps the operand
    // descriptors in the uniform registers the tensor core reads them from.
    if (leader) {
      constexpr uint32_t idesc = instr_desc_f16(2 * GP_M, BN, std::is_same<T, __nv_bfloat16>::value ? 1 : 0,
                                                A_MN ? 1 : 0, B_MN ? 1 : 0);
      const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0), s0 = smem_u32(smem);
      int stage = 0;
      uint32_t phase = 0;
      int buf = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < num_tiles; tile += num_pairs) {
        if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], acc_phase ^ 1, 0x800 | buf, abort_flag))) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tb + buf * 256;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], phase, 0x900 | stage, abort_flag))) { ok = false; break; }
          const uint32_t sa = s0 + stage * Cfg::STAGE_BYTES, sb = sa + GP_A_BYTES;
          const uint64_t ad = A_MN ? smem_desc_sw128(sa, 8192, 1024) : smem_desc_sw128(sa, 16, 1024);
          const uint64_t bd = !B_MN ? smem_desc_sw128(sb, 16, 1024)
                              : Cfg::BOX == 64 ? smem_desc_sw128(sb, 8192, 1024) : smem_desc_sw64(sb, 4096, 512);
          // K-major: 16 elements = 32 bytes along the swizzled row; MN-major: 16 k-rows of a box
#pragma unroll
          for (int k = 0; k < GP_K / 16; ++k) {
            const uint64_t ak = desc_advance(ad, k * (A_MN ? 2048 : 32)), bk = desc_advance(bd, k * (B_MN ? Cfg::BOX * 32 : 32));
            if (elect_one()) tc_mma_ss_pair(d_tmem, ak, bk, idesc, (kb | k) ? 1u : 0u);
          }
          if (elect_one()) tc_commit_pair(&empty[stage]);  // both producers may refill the slot once these MMAs have read it
          if (++stage == GP_STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (elect_one()) tc_commit_pair(&acc_full[buf]);  // both epilogues
        buf ^= 1;
        if (buf == 0) acc_phase ^= 1;
      }
    }
  } else {
    // ---------------------------------------------------------------------- epilogue (both CTAs)
    const int q = warp & 3;   // TMEM lane quarter this warp may read
    const int ew = warp - 2;  // 0 .. EPI_WARPS-1
    const int half = ew >> 2; // with eight epilogue warps: which half of the tile's columns
    const T* bias = reinterpret_cast<const T*>(p.bias);
    uint8_t* stage_c = smem + Cfg::OFF_EPI_C + ew * 4096;
    uint8_t* stage_x = smem + Cfg::OFF_EPI_X + ew * 4096;
    // at most one of addend / mask travels through the TMA box; a second one is read directly
    const bool use_x = !p.direct && (p.addend != nullptr || p.mask != nullptr);
    const EpiArgs<T> epi{{reinterpret_cast<T*>(p.C), bias, reinterpret_cast<const T*>(p.addend), reinterpret_cast<const T*>(p.mask),
                          p.ldc, p.ld_addend, p.ld_mask, p.M, p.N, p.relu},
                         &tmC, &tmX, stage_c, stage_x, &x_full[ew], use_x, p.addend != nullptr, p.direct != 0,
                         (p.addend != nullptr && p.mask != nullptr) ? reinterpret_cast<const T*>(p.mask) : nullptr};
    const int first = half * Cfg::FIRST * 64;                             // first column of this warp's share of a tile
    const int steps = half == 0 ? Cfg::FIRST : BN / 64 - Cfg::FIRST;      // of 64 columns
    int buf = 0;
    uint32_t acc_phase = 0, x_phase = 0;
    bool ok = true;
    // an earlier kernel that gave up leaves the status set: then nothing is written
    const bool dead = *(volatile int*)&g_dev_status != 0;
    if (lane == 0) {
      if (!p.direct) tma_prefetch_desc(&tmC);
      if (use_x) tma_prefetch_desc(&tmX);
    }
    for (int tile = pair; ok && tile < num_tiles; tile += num_pairs) {
      const int m0 = (tile % p.tiles_m) * (2 * GP_M) + (int)rank * GP_M;
      const int n0 = (tile / p.tiles_m) * BN + first;
      const int row0 = m0 + q * 32;
      if (use_x && !dead && lane == 0) {  // box of step 0, in flight while the main loop still runs
        mbar_expect_tx(&x_full[ew], 4096);
        tma_load_2d(stage_x, &tmX, n0, row0, &x_full[ew]);
      }
      if (!mbar_wait(&acc_full[buf], acc_phase, 0xa00 | buf, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256 + first;
      if (!dead) epilogue_tile<T>(epi, steps, taddr, row0, n0, lane, x_phase, abort_flag, 0xb00 | ew, ok);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[buf]), 0));
      buf ^= 1;
      if (buf == 0) acc_phase ^= 1;
    }
    if (lane == 0) tma_store_wait_read();  // the boxes have been read; the kernel's end completes the writes
  }

  // Unwind: every role has left its loop (normally or through a bounded wait).
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  // neither CTA leaves (or frees tensor memory) while the other may still signal its barriers or
  // have MMAs reading its shared memory
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, GP_TMEM_COLS);
  }
}

template <typename T, int BN, bool A_MN, bool B_MN>
static int launch_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const CUtensorMap& tmX,
                       const PairParams& p, int grid, cudaStream_t st) {
  auto kern = gemm_pair_tc05_kernel<T, BN, A_MN, B_MN>;
  static std::atomic<uint64_t> attr_done{0};
  if (int rc0 = ensure_dynamic_smem(kern, PairCfg<BN>::SMEM_BYTES, attr_done, "gemm_pair_tc05")) return rc0;
  launch_overlapped(kern, dim3(grid), dim3(GP_THREADS), PairCfg<BN>::SMEM_BYTES, st, tmA, tmB, tmC, tmX, p);
  return launched("gemm_pair_tc05");
}

template <typename T, int BN>
static int dispatch_pair(bool a_mn, bool b_mn, const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC,
                         const CUtensorMap& tmX, const PairParams& p, int grid, cudaStream_t st) {
  if constexpr (BN == 256)  // (see gemm_pair_width)
    if (a_mn && b_mn) return launch_pair<T, BN, true, true>(tmA, tmB, tmC, tmX, p, grid, st);
  if (a_mn) return launch_pair<T, BN, true, false>(tmA, tmB, tmC, tmX, p, grid, st);
  if (b_mn) return launch_pair<T, BN, false, true>(tmA, tmB, tmC, tmX, p, grid, st);
  return launch_pair<T, BN, false, false>(tmA, tmB, tmC, tmX, p, grid, st);
}

// 256 x 256 tiles the output offers; the caller takes this kernel when they fill the pairs of SMs.
int64_t gemm_pair_tiles(int64_t M, int64_t N) { return ceil_div(M, 2 * GP_M) * ceil_div(N, 256); }

// Tile width.  A k-block of a 256 x 256 tile takes 528 cycles of its pair and one of a 256 x 192 tile 462 (what an SM takes in
// from the L2, 32 and 28 KB at 62 bytes a cycle), so the narrow tile, which moves a sixth more operand bytes for the
// same product, is for outputs whose last wave of wide tiles is mostly empty: as many waves of narrow ones.  M 4096 N 1536, two
// waves of either, wide and narrow: B contiguous along K: K 4608 49.0 and 42.7 us, K 6144 64.4 and 59.3; along N: K 1536 21.6 and 19.7,
// K 6144 66.9 and 61.6; M 2112 N 3072 K 1024 16.4 and 15.3 (35 such products with B along K: 1.02 to 1.17 times as fast).
// B contiguous along N comes in rows of 64 bytes, and rows that do not begin on multiples of 64 touch a half more of the L2's
// sectors instead of a quarter: M 3320 N 1464 K 1840 24.6 and 27.5, M 2960 N 2296 K 1808 26.6 and 28.8, M 3328 N 1488 K 1184 16.3 and
// 15.9.  With A contiguous along M as well the narrow tile wins nothing even on aligned rows: M 1448 N 6624 K 952 21.0 and 21.5, M 968
// N 6464 K 5576 66.5 and 66.9, M 1552 N 5696 K 2544 41.4 and 41.2.
int gemm_pair_width(int64_t M, int64_t N, bool a_mn, bool b_mn, bool b_rows_64, int sms) {
  if (b_mn && (a_mn || !b_rows_64)) return 256;
  const int64_t pairs = sms / 2, tm = ceil_div(M, 2 * GP_M);
  const int64_t wide = ceil_div(tm * ceil_div(N, 256), pairs) * 528, narrow = ceil_div(tm * ceil_div(N, 192), pairs) * 462;
  return narrow * 100 < wide * 95 ? 192 : 256;
}

int gemm_pair_tc05(const void* a, const void* b, void* c, const void* bias, const void* addend, int64_t ld_addend,
                   const void* mask, int64_t ld_mask, int64_t M, int64_t N, int64_t K, int64_t a_sm, int64_t a_sk,
                   int64_t b_sk, int64_t b_sn, int64_t ldc, int relu, int dtype, int sms, cudaStream_t st) {
  const bool a_mn = (a_sk != 1), b_mn = (b_sk != 1);
  const int width = gemm_pair_width(M, N, a_mn, b_mn, reinterpret_cast<uintptr_t>(b) % 64 == 0 && b_sk % 32 == 0, sms);
  CUtensorMap tmA, tmB, tmC, tmX;
  int rc;
  const bool direct = gemm_needs_direct(c, ldc, bias, addend, ld_addend, mask, ld_mask);
  {
    uint64_t dims[2] = {(uint64_t)N, (uint64_t)M}, str[1] = {(uint64_t)ldc * 2};
    uint32_t box[2] = {64, 32};
    if (direct) memset(&tmC, 0, sizeof(tmC));
    else if ((rc = encode_tmap_sw128(&tmC, c, dtype, 2, dims, str, box))) return rc;
    const void* xp = direct ? nullptr : addend ? addend : mask;
    str[0] = (uint64_t)(addend ? ld_addend : ld_mask) * 2;
    if (xp) { if ((rc = encode_tmap_sw128(&tmX, xp, dtype, 2, dims, str, box))) return rc; }
    else tmX = tmC;
  }
  {
    uint64_t dims[2], str[1];
    uint32_t box[2];
    if (a_mn) { dims[0] = (uint64_t)M; dims[1] = (uint64_t)K; str[0] = (uint64_t)a_sk * 2; box[0] = 64; box[1] = GP_K; }
    else      { dims[0] = (uint64_t)K; dims[1] = (uint64_t)M; str[0] = (uint64_t)a_sm * 2; box[0] = GP_K; box[1] = GP_M; }
    if ((rc = encode_tmap_sw128(&tmA, a, dtype, 2, dims, str, box))) return rc;
    const bool narrow = width == 192;
    if (b_mn) { dims[0] = (uint64_t)N; dims[1] = (uint64_t)K; str[0] = (uint64_t)b_sk * 2; box[0] = narrow ? 32 : 64; box[1] = GP_K; }
    else      { dims[0] = (uint64_t)K; dims[1] = (uint64_t)N; str[0] = (uint64_t)b_sn * 2; box[0] = GP_K; box[1] = (uint32_t)(width / 2); }
    if ((rc = b_mn && narrow ? encode_tmap_sw64(&tmB, b, dtype, 2, dims, str, box) : encode_tmap_sw128(&tmB, b, dtype, 2, dims, str, box)))
      return rc;
  }
  PairParams p;
  p.C = c; p.bias = bias; p.addend = addend; p.mask = mask;
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.ldc = ldc; p.ld_addend = ld_addend; p.ld_mask = ld_mask;
  p.relu = relu; p.direct = direct;
  p.tiles_m = (int)ceil_div(M, 2 * GP_M); p.tiles_n = (int)ceil_div(N, width);
  const int64_t tiles = (int64_t)p.tiles_m * p.tiles_n;
  // The tiles are handed out whole: cutting the tiles of a partial last wave along K (tried, also with the cut tiles done
  // first) balances the pairs but does not shorten the kernel - with fewer pairs busy in the last wave each runs its
  // k-blocks faster, and the partial tiles add traffic.  Products with fewer tiles than pairs run on the one-wave kernel.
  const int64_t pairs = tiles < sms / 2 ? tiles : sms / 2;
  const int grid = (int)(2 * pairs);
  TFB_DISPATCH_16(dtype, T, {
    if (width == 192) return dispatch_pair<T, 192>(a_mn, b_mn, tmA, tmB, tmC, tmX, p, grid, st);
    return dispatch_pair<T, 256>(a_mn, b_mn, tmA, tmB, tmC, tmX, p, grid, st);
  })
}

}  // namespace tfb
