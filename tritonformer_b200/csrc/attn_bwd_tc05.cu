// Causal flash attention backward on tcgen05 / TMEM for sm_100a (head_dim 32 or 64; 128: attn_bwd128_tc05.cu).
//
// An item is a (128-key tile, batch*head); a CTA walks its query tiles at or below the diagonal.  The grid has one block per
// item, but a CTA that is nearly done with its item takes over a block that has not been launched yet (cluster launch
// control: that launch is cancelled and its block index handed over), so tensor memory, barriers and the ring stay set up
// from item to item.  With a fresh CTA per item, 8.9 k of the 53 k cycles of an average item at T 2048 were spent outside the
// walk.  A list dealt out in advance would do the same, but not beside the weight-gradient products of another stream, which
// hold some of the SMs.  K and V are doubled as well, so that the next item's scores run ahead like those of
// any next tile, and an item's dV and dK are written behind the arithmetic of the next item's first tile.
// Backward with its two small passes, fp16: B4 H16 T2048 hd64 208 -> 194 us.
// Everything is computed transposed (rows = keys) so that the per-query statistics (log-sum-exp,
// delta) are per-column constants and no row reductions are needed:
//   Sᵀ  = K Q_iᵀ                 dPᵀ = V dO_iᵀ                      (tensor cores -> TMEM)
//   Pᵀ  = 2^(Sᵀ·c + bias - lse)  dSᵀ = Pᵀ ∘ (dPᵀ - delta)            (compute warps -> smem, 16 bit)
//   dV += Pᵀ dO_i     dK += dSᵀ Q_i     dQ_i = dS K                  (tensor cores -> TMEM)
// dV and dK stay in TMEM for the whole walk; dQ_i is added to an fp32 global accumulator (TMA
// reduce-add) because every key tile contributes to it; a small kernel scales and rounds the
// accumulator afterwards.
// A 128 x 64 swizzled panel of 16-bit values is at the same time a K-major operand with 128 rows
// and an MN-major operand with 128 contraction rows, so each of K, V, Q_i, dO_i, dSᵀ sits in
// shared memory once and serves two products.
//
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warps 4-7 drain dQ_i, warps 8-23 compute (thread = TMEM lane, four
// warps per lane quarter, each taking a quarter of the columns).
// Pᵀ goes into the 64 TMEM columns that are left instead of shared memory and is
// the A operand of the dV product.
// The scores of tile i+1 are issued as soon as the compute warps hold the scores of tile i in
// registers, ahead of the gradient products of tile i, so the compute warps find them ready and work on tile
// i+1 while the tensor core finishes tile i.
// A sequence that is no multiple of 128: the rows past its end are zeros in shared memory (TMA fill); as queries they get
// exact zeros for P and dS and their rows of dQ are left out (the accumulator's next rows are another slice's), as keys the
// mask keeps them from every query and their rows are not stored.  head_dim 32 runs on the
// head_dim 64 kernel with zero columns.
// (Sub-tiles of 64 queries on two CTAs per SM with half of tensor and shared memory each, tried here as well: 205-218 us against
// 191 at B4 H16 T2048 fp16, 165 against 89 at B1 H8 T4096.  A sub-tile's chain takes 4.3 k cycles even alone on an SM, nearly as
// long as a whole tile's 5.5 k, and the two CTAs share what it waits for.)
// TMEM columns: [0,128) Sᵀ; [128,256) dPᵀ; [256,320) dV; then dK; then dQ_i; then Pᵀ.
#define TFB_STATUS_FROM_LAUNCH
#include "attn.cuh"
#include "tc05.cuh"
#include <type_traits>

namespace tfb {

extern std::atomic<int> g_attn_debug;

constexpr float kLog2eB = 1.4426950408889634f;
constexpr int FB_T = 128;           // tile edge (keys and queries)
constexpr int FB_CWARPS = 16;        // compute warps: 4 TMEM lane quarters x 4 column quarters
// Warpgroups: TMA, MMA and two idle warps; four dQ-drain warps; the compute warps.  The block is launched with 80 registers a
// thread (six warps per scheduler); the first two groups hand some of theirs on to the compute warps.  (More than 88 for these
// left the MMA warp spilling: 179 against 172 us.  At 88 they still spill, 16 to 32 bytes a thread; how much depends on as little as the
// layout of the parameters.)  Backward with its two small passes, in microseconds: in 22 warps with the drain
// warps last, with the warpgroups, and now, with the registers moved as well and the packed arithmetic on blocks that know whether
// they meet the diagonal: B4 H16 T2048 fp16 189.6, 172.2, 172.3, exact slopes 195.9, 183.8, 175.2; B3 H11 T1472 bf16 67.0, 61.3, 61.7;
// B3 H16 T704 bf16 with the rounded table 38.0, 33.8, 32.0; B2 H12 T1024 fp16 33.8, 30.7, 30.8.
constexpr int FB_FIRST_C = 8;       // first compute warp
constexpr int FB_THREADS = 32 * (FB_FIRST_C + FB_CWARPS);
constexpr int FB_REGS = 80, FB_REGS_ISSUE = 56, FB_REGS_DRAIN = 72, FB_REGS_COMPUTE = 88;
static_assert(128 * (FB_REGS_ISSUE + FB_REGS_DRAIN + 4 * FB_REGS_COMPUTE) <= FB_THREADS * FB_REGS, "registers of the block");

constexpr int HD = 64;
constexpr int TILE_BYTES = FB_T * 128;   // 128 rows x 64 x 2 B
// Query-side ring depth: the gradient products of tile i-1 still read their Q / dO while the scores of tile i+1 are issued
// (with two, the load of tile i+1 could only start when tile i-1 had retired, and its latency showed up as a wait for scores on
// every tile).
constexpr int QS = 3;
// K and V of two items: the next item's scores run ahead of the current item's last products like those of
// any next tile.  (With one, the walk stood still for 7.9 k cycles from item to item.)
constexpr int KVS = 2;
constexpr int OFF_K = 0;                              // [KVS][K, V]
constexpr int OFF_V = TILE_BYTES;
constexpr int OFF_Q = KVS * 2 * TILE_BYTES;           // [QS]
constexpr int OFF_DO = OFF_Q + QS * TILE_BYTES;       // [QS]
constexpr int OFF_DS = OFF_DO + QS * TILE_BYTES;      // dSᵀ 128 x 128 x 2 B
constexpr int OFF_STAT = OFF_DS + 32768;              // [2 parities][16 compute warps][lse2[32], delta[32]] fp32
// dQ_i staging for the TMA reduction: a box of 32 rows x 128 B (32 columns) per drain warp, which its two chunks pass through
// one after the other.
constexpr int OFF_DQ = OFF_STAT + 8192;
constexpr int OFF_BAR = OFF_DQ + 4 * 4096;
constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
constexpr int COL_S = 0, COL_DP = 128, COL_DV = 256, COL_DK = 256 + HD, COL_DQ = 256 + 2 * HD;
// Pᵀ (16-bit, two queries per column): the A operand of the dV product, which then reads only dO from shared memory
constexpr int COL_PT = 256 + 3 * HD;

struct FbParams {
  int* status;    // the library's status word
  const float* lse;
  const float* delta;
  void *dk, *dv;
  int64_t sdk_b, sdk_h, sdk_t, sdv_b, sdv_h, sdv_t;
  int H, T, hd;   // hd: the real head_dim, 32 or 64
  int BH, group;  // batch*heads; how many of them are walked together (their tiles share the L2)
  float scale;
  const float* slopes;
  int debug;  // bit 5: per-slice item order (test switch)
};

__device__ __forceinline__ float ex2_approx_b(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  typename Num<T>::T2 h = Num<T>::from_f2(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// RAGGED: T is no multiple of 128 (a run-time branch in the compute and drain loops cost whole tiles 1 %: B4 H16 T2048 hd64
// fp16 193 against 191 us, spilled registers).
template <typename T, int BIAS, bool RAGGED>
__global__ void __launch_bounds__(FB_THREADS, 1) attn_bwd_tc05_kernel(const __grid_constant__ CUtensorMap tmQ,
                                                                      const __grid_constant__ CUtensorMap tmK,
                                                                      const __grid_constant__ CUtensorMap tmV,
                                                                      const __grid_constant__ CUtensorMap tmDO,
                                                                      const __grid_constant__ CUtensorMap tmDQ,
                                                                      const FbParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* s_stat = reinterpret_cast<float*>(smem + OFF_STAT);  // [2 parities][16 warps][lse2[32], delta[32]]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* q_full = bars + 0;       // [3] Q_i and dO_i landed
  uint64_t* q_empty = bars + 3;      // [3] products reading them retired
  uint64_t* s_full = bars + 6;       // Sᵀ and dPᵀ in TMEM
  uint64_t* pds_full = bars + 7;     // Pᵀ and dSᵀ in smem (and Sᵀ, dPᵀ consumed)
  uint64_t* dq_full = bars + 8;      // dV, dK, dQ_i products retired
  uint64_t* dq_free = bars + 9;      // dQ_i read out of TMEM
  uint64_t* s_free = bars + 10;      // Sᵀ and dPᵀ read out of TMEM: the next scores may overwrite them
  uint64_t* kv_full = bars + 12;     // [KVS] K and V of an item landed
  uint64_t* kv_empty = bars + 14;    // [KVS] the item's last products have retired: K and V may be replaced
  uint64_t* acc_free = bars + 16;    // dV and dK of an item have been read out of TMEM
  uint64_t* next_full = bars + 17;   // the answer to the request for another item has landed
  uint64_t* next_empty = bars + 18;  // every role has read it
  uint8_t* next_item = reinterpret_cast<uint8_t*>(bars + 20);  // the answer, 16 bytes
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 22);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Items (key tile, batch*head) are numbered longest walk first: within a group of batch*head slices the key tiles with the
  // longest walk (tile 0) of EVERY slice come first, so the tail of the kernel is made of short ones.
  const int nq = (p.T + FB_T - 1) / FB_T;
  struct Item {
    int kt, bh;  // (the rest follows from these where it is needed: few registers live through the walk)
  };
  auto item_of = [&](int block) -> Item {
    Item w;
    if (p.debug & 32) {  // per-slice order (test switch)
      w.kt = block % nq;
      w.bh = block / nq;
    } else {
      const int g = block / (nq * p.group), r = block % (nq * p.group);
      const int gsz = min(p.group, p.BH - g * p.group);
      w.kt = r / gsz;
      w.bh = g * p.group + r % gsz;
    }
    return w;
  };
  // The item after the CTA's n-th one: false when there is none.  Read by every role once per item; `alone`: by one lane.
  auto next_of = [&](int n, Item& w, bool alone) -> bool {
    bool ok = mbar_wait(next_full, n & 1, 0x2800, abort_flag);
    if (!alone) ok = __all_sync(0xffffffffu, ok) != 0;
    if (!ok) return false;
    int block;
    bool more = clc_answer(next_item, block);
    fence_proxy_async_smem();  // read, before the next answer is written
    if (!alone) {  // the same in every lane: tells the compiler so, and with it that the operand descriptors are uniform
      more = __all_sync(0xffffffffu, more) != 0;
      block = __shfl_sync(0xffffffffu, block, 0);
    }
    if (alone || lane == 0) mbar_arrive(next_empty);
    if (more) w = item_of(block);
    return more;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < KVS; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    for (int i = 0; i < 3; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(pds_full, FB_CWARPS);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, 4);
    mbar_init(s_free, FB_CWARPS);
    mbar_init(acc_free, FB_CWARPS);
    mbar_init(next_full, 1);
    mbar_init(next_empty, 2 + FB_CWARPS + 4);  // producer, MMA issuer, compute warps, drain warps
    mbar_fence_init();
  }
  if (warp == 1) {
    __syncwarp();
    tmem_alloc(tmem_holder, 512);
  }
  // set-up above is CTA-local and may overlap the previous kernel's tail; global memory comes after
  grid_dependency_wait();
  allow_dependents();
  if (threadIdx.x == 0) {
    *status_slot() = p.status;
    *abort_flag = (*(volatile int*)p.status != 0) ? 1 : 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const bool dead = *abort_flag != 0;

  if (warp < 4) {
  regs_down<FB_REGS_ISSUE>();
  if (warp == 0) {
    // --------------------------------------------------------------------- TMA producer
    if (lane == 0 && !dead) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      tma_prefetch_desc(&tmDO);
      Item w = item_of(blockIdx.x);
      int g = 0;  // tiles of the CTA so far: the phases of every barrier run on across its items
      bool ok = true;
      // K and V of the CTA's n-th item
      auto load_kv = [&](int n) -> bool {
        const int ks = n % KVS, b = w.bh / p.H, h = w.bh % p.H;
        if (n >= KVS && !mbar_wait(&kv_empty[ks], (n / KVS - 1) & 1, 0x2110 | ks, abort_flag)) return false;
        mbar_expect_tx(&kv_full[ks], 2 * TILE_BYTES);
        uint8_t* dst = smem + OFF_K + ks * 2 * TILE_BYTES;
        tma_load_4d(dst, &tmK, 0, w.kt * FB_T, h, b, &kv_full[ks]);
        tma_load_4d(dst + TILE_BYTES, &tmV, 0, w.kt * FB_T, h, b, &kv_full[ks]);
        return true;
      };
      for (int n = 0; ok; ++n) {
        ok = load_kv(n);
        for (int it = 0; it < nq - w.kt && ok; ++it, ++g) {
          const int st = g % QS;
          const uint32_t ph = (g / QS) & 1;
          if (!mbar_wait(&q_empty[st], ph ^ 1, 0x2100 | st, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&q_full[st], 2 * TILE_BYTES);
          const int i0 = (w.kt + it) * FB_T, b = w.bh / p.H, h = w.bh % p.H;
          tma_load_4d(smem + OFF_Q + st * TILE_BYTES, &tmQ, 0, i0, h, b, &q_full[st]);
          tma_load_4d(smem + OFF_DO + st * TILE_BYTES, &tmDO, 0, i0, h, b, &q_full[st]);
        }
        // Asked for only now, with the item's last loads issued: asked for at its start, the CTAs with the longest items
        // would take the first of the remaining ones.
        if (ok && n > 0) ok = mbar_wait(next_empty, (n - 1) & 1, 0x2120, abort_flag);
        if (!ok) break;
        mbar_expect_tx(next_full, 16);
        clc_request(next_item, next_full);
        ok = next_of(n, w, true);
      }
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------------------- MMA issuer
    // The whole warp runs this code and one elected lane issues each tcgen05 instruction.  With the loop in a
    // single lane the operand descriptors live in ordinary registers and every instruction pays for moving
    // them to the uniform registers the tensor core reads (measured: 63 cycles per M128 N64 K16 instruction
    // against 49 with warp-uniform code, and 80-120 in this kernel, where it made the issue of a tile's 32
    // instructions the longest item of the step).
    if (!dead) {
      constexpr int fmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
      constexpr uint32_t idesc_s = instr_desc_f16(128, 128, fmt, 0, 0);   // Sᵀ, dPᵀ : both K-major
      constexpr uint32_t idesc_kv = instr_desc_f16(128, HD, fmt, 0, 1);   // dV, dK  : A K-major, B MN-major
      constexpr uint32_t idesc_q = instr_desc_f16(128, HD, fmt, 1, 1);    // dQ      : both MN-major
      // read from shared memory: tell the compiler it is uniform
      const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
      // operand descriptors of every buffer in both roles; each MMA only advances the start address
      // (K-major: lbo unused, 8-row groups 1024 B apart; MN-major: 64-element chunks one 16 KB panel apart,
      // 8-row groups 1024 B apart)
      const uint32_t s0 = smem_u32(smem);
      const uint64_t dk_k = smem_desc_sw128(s0 + OFF_K, 16, 1024);
      const uint64_t dk_mn = smem_desc_sw128(s0 + OFF_K, 16384, 1024);
      const uint64_t dv_k = smem_desc_sw128(s0 + OFF_V, 16, 1024);
      const uint64_t dds_k = smem_desc_sw128(s0 + OFF_DS, 16, 1024);
      const uint64_t dds_mn = smem_desc_sw128(s0 + OFF_DS, 16384, 1024);
      // every lane waits; the verdict is made uniform so that the warp stays converged
      auto wait = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
        return __all_sync(0xffffffffu, mbar_wait(bar, parity, code, abort_flag)) != 0;
      };
      bool ok = true;
      // Sᵀ = K Q_iᵀ and dPᵀ = V dO_iᵀ of query tile `it`
      auto issue_scores = [&](int g, int n) -> bool {  // g: tiles of the CTA before this one, n: items
        const uint32_t kv = (n % KVS) * 2 * TILE_BYTES;
        const int st = g % QS;
        if (!wait(&q_full[st], (g / QS) & 1, 0x2300 | st)) return false;
        tc_fence_after();
        const uint64_t q_k = smem_desc_sw128(s0 + OFF_Q + st * TILE_BYTES, 16, 1024);
        const uint64_t do_k = smem_desc_sw128(s0 + OFF_DO + st * TILE_BYTES, 16, 1024);
#pragma unroll
        for (int s = 0; s < HD / 16; ++s) {
          const uint32_t off = s * 32;
          if (elect_one()) tc_mma_ss(tb + COL_S, desc_advance(dk_k, kv + off), desc_advance(q_k, off), idesc_s, s ? 1u : 0u);
        }
#pragma unroll
        for (int s = 0; s < HD / 16; ++s) {
          const uint32_t off = s * 32;
          if (elect_one()) tc_mma_ss(tb + COL_DP, desc_advance(dv_k, kv + off), desc_advance(do_k, off), idesc_s, s ? 1u : 0u);
        }
        if (elect_one()) tc_commit(s_full);
        return true;
      };
      // dV += Pᵀ dO_i, dK += dSᵀ Q_i, dQ_i = dS K
      auto issue_grads = [&](int g, int n, int it, bool last) -> bool {
        const uint32_t kv = (n % KVS) * 2 * TILE_BYTES;
        const int st = g % QS;
        const uint64_t q_mn = smem_desc_sw128(s0 + OFF_Q + st * TILE_BYTES, 16384, 1024);
        const uint64_t do_mn = smem_desc_sw128(s0 + OFF_DO + st * TILE_BYTES, 16384, 1024);
        // the dQ columns still hold the previous tile's dQ until the drain warps are done with it
        if (g > 0 && !wait(dq_free, (g - 1) & 1, 0x2400)) return false;
        tc_fence_after();
        const uint32_t acc = it ? 1u : 0u;
#pragma unroll
        for (int s = 0; s < FB_T / 16; ++s) {  // contraction over the 128 queries of this tile
          const uint32_t koff = (s / 4) * 16384 + (s % 4) * 32;  // K-major A: 16 queries = 32 B along the row
          const uint32_t moff = s * 2048;                         // MN-major B: 16 query rows of 128 B
          if (elect_one()) {
            tc_mma_ts(tb + COL_DV, tb + COL_PT + s * 8, desc_advance(do_mn, moff), idesc_kv, s ? 1u : acc);
            tc_mma_ss(tb + COL_DK, desc_advance(dds_k, koff), desc_advance(q_mn, moff), idesc_kv, s ? 1u : acc);
          }
        }
#pragma unroll
        for (int s = 0; s < FB_T / 16; ++s) {  // contraction over the 128 keys of this CTA
          const uint32_t moff = s * 2048;      // 16 key rows of 128 B in dSᵀ and in K
          if (elect_one()) tc_mma_ss(tb + COL_DQ, desc_advance(dds_mn, moff), desc_advance(dk_mn, kv + moff), idesc_q, s ? 1u : 0u);
        }
        if (elect_one()) {
          tc_commit(&q_empty[st]);
          tc_commit(dq_full);
          if (last) tc_commit(&kv_empty[n % KVS]);
        }
        return true;
      };
      Item w = item_of(blockIdx.x);
      int g = 0;
      ok = wait(&kv_full[0], 0, 0x2200) && issue_scores(0, 0);
      for (int n = 0; ok; ++n) {
        Item wn = w;
        bool more = false;
        for (int it = 0; it < nq - w.kt && ok; ++it, ++g) {
          const bool last = w.kt + it + 1 == nq;
          if (last) {
            more = next_of(n, wn, false);
            if (more && !wait(&kv_full[(n + 1) % KVS], ((n + 1) / KVS) & 1, 0x2200)) { ok = false; break; }
          }
          if (!last || more) {
            // The compute warps hand Sᵀ / dPᵀ back as soon as they hold them in registers, about half-way through
            // their work on the tile: the next tile's scores are issued then and have landed when the warps come
            // back for them.  (Issued only once Pᵀ / dSᵀ were ready, they cost a round trip of 1.5 k cycles per
            // tile that nothing hid: the score buffers cannot be doubled, tensor memory is full.)
            if (!wait(s_free, g & 1, 0x2550)) { ok = false; break; }
            if (!issue_scores(g + 1, last ? n + 1 : n)) { ok = false; break; }
          }
          if (!wait(pds_full, g & 1, 0x2500)) { ok = false; break; }
          // the first products of an item overwrite dV and dK of the one before
          if (it == 0 && n > 0 && !wait(acc_free, (n - 1) & 1, 0x2560)) { ok = false; break; }
          ok = issue_grads(g, n, it, last);
        }
        if (!more) break;
        w = wn;
      }
    }
    __syncwarp();
  }
  } else if (warp >= FB_FIRST_C) {
    // -------------------------------------------------------------------------- compute
    regs_up<FB_REGS_COMPUTE>();
    if (!dead) {
      const int cw = warp - FB_FIRST_C;  // 0..15
      const int qd = warp & 3;           // TMEM lane quarter
      const int cq = cw >> 2;            // which quarter (32) of the 128 query columns
      const int r = qd * 32 + lane;      // TMEM lane = key row
      const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
      const float c2 = p.scale * kLog2eB;
      const uint64_t c2p = f2_pack(c2, c2);
      uint8_t* sds = smem + OFF_DS;
      bool ok = true;
      // Per-query statistics of the warp's 32 query columns: lane l carries lse and delta of
      // column l, fetched one tile ahead (so the global-memory latency is not part of the tile) and handed to the
      // other lanes through a slice of shared memory that belongs to this warp: no barrier across the warps.
      auto load_stat = [&](const Item& w, int it, float& l2, float& dl) {
        const int i = (w.kt + it) * FB_T + cq * 32 + lane;
        const int64_t at = (int64_t)w.bh * p.T + i;
        l2 = i < p.T ? p.lse[at] : 0.f;  // converted to log2 units where it is used: nothing here may wait for the load
        dl = i < p.T ? p.delta[at] : 0.f;
      };
      float lse_next, delta_next;
      Item w = item_of(blockIdx.x), wp = w;  // wp: the item before
      load_stat(w, 0, lse_next, delta_next);
      // dV and dK of an item whose products have all retired
      auto store_item = [&](const Item& w) {
        tc_fence_after();
        const int j = w.kt * FB_T + r;
        T* dvp = reinterpret_cast<T*>(p.dv) + (w.bh / p.H) * p.sdv_b + (w.bh % p.H) * p.sdv_h + (int64_t)j * p.sdv_t;
        T* dkp = reinterpret_cast<T*>(p.dk) + (w.bh / p.H) * p.sdk_b + (w.bh % p.H) * p.sdk_h + (int64_t)j * p.sdk_t;
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {  // this warp's HD / 4 columns in steps of 8
          const int col0 = cq * (HD / 4) + c * 8;
          if (col0 >= p.hd) break;
          uint32_t v[8], u[8];
          tmem_ld8(lane_addr + COL_DV + col0, v);
          tmem_ld8(lane_addr + COL_DK + col0, u);
          tc_wait_ld();
          if (j < p.T) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[e]);
            *reinterpret_cast<uint4*>(dvp + col0) = pack8<T>(f);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(u[e]) * p.scale;
            *reinterpret_cast<uint4*>(dkp + col0) = pack8<T>(f);
          }
          __syncwarp();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_free);  // the next item's products may overwrite them
      };
      // With the next item's scores already there, an item is stored behind the arithmetic of the next one's first tile,
      // which hides its last products.
      int g = 0;  // tiles of the CTA before this one
      for (int n = 0;; ++n) {
      const AlibiLog2<BIAS> alibi(BIAS ? p.slopes[w.bh % p.H] : 0.f);
      const int j = w.kt * FB_T + r;     // this thread's key
      for (int it = 0; it < nq - w.kt; ++it, ++g) {
        const int i0 = (w.kt + it) * FB_T;
        // the warp's 32 x 32 block against the diagonal: < 0 masked, 0 cut, > 0 untouched
        const int rel = it * 4 + cq - qd;
        // this tile's statistics, double buffered by iteration parity: a lane that is already here may share
        // the warp with one that still reads the previous tile's slice
        float* s_lse2 = s_stat + ((g & 1) * FB_CWARPS + cw) * 64;
        float* s_delta = s_lse2 + 32;
        s_lse2[lane] = -lse_next * kLog2eB;
        s_delta[lane] = -delta_next;
        __syncwarp();
        if (it + 1 < nq - w.kt) load_stat(w, it + 1, lse_next, delta_next);  // after the warp barrier, which would wait for it
        if (ok) ok = mbar_wait(s_full, g & 1, 0x2600, abort_flag);
        uint32_t pk[16], dk_[16];  // this thread's 32 columns of Pᵀ and dSᵀ, packed 16-bit pairs
        if (ok) {
          tc_fence_after();
          if (rel < 0) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_free);
#pragma unroll
            for (int e = 0; e < 16; ++e) pk[e] = dk_[e] = 0u;
          } else {
            const int first = rel == 0 ? lane : 0;  // first of the warp's query columns that sees this thread's key
            // Four chunks of 8 query columns; the tensor-memory loads of a chunk are issued before the chunk ahead of
            // it is worked on (two register sets of 8 + 8 values), so only the first load's latency is exposed.
            // (Requesting a tile's first chunk at the end of the tile before it, ahead of the gradient products whose
            // burst makes the load wait 850 cycles, was tried: the wait for the next scores at that point cost more
            // than it saved, 230 against 210 us.  All 64 values at once do not fit the registers.)
            uint32_t sv_[2][8], dv_[2][8];
            tmem_ld8(lane_addr + COL_S + cq * 32, sv_[0]);
            tmem_ld8(lane_addr + COL_DP + cq * 32, dv_[0]);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const int col0 = cq * 32 + c * 8;
              const float d0 = (float)(i0 + col0 - j);  // distance of the chunk's first query to this thread's key
              tc_wait_ld();
              if (c + 1 < 4) {
                tmem_ld8(lane_addr + COL_S + col0 + 8, sv_[(c + 1) & 1]);
                tmem_ld8(lane_addr + COL_DP + col0 + 8, dv_[(c + 1) & 1]);
              } else {  // this warp's share of Sᵀ and dPᵀ is in registers
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_free);
              }
              const uint32_t *sv = sv_[c & 1], *dv = dv_[c & 1];
#pragma unroll
              for (int e4 = 0; e4 < 8; e4 += 4) {
                const float4 l4 = *reinterpret_cast<const float4*>(s_lse2 + c * 8 + e4);
                const float4 d4 = *reinterpret_cast<const float4*>(s_delta + c * 8 + e4);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  const int e = e4 + 2 * k;
                  uint64_t x = f2_fma(f2_pack(__uint_as_float(sv[e]), __uint_as_float(sv[e + 1])), c2p,
                                      k ? f2_pack(l4.z, l4.w) : f2_pack(l4.x, l4.y));
                  if (BIAS) x = alibi.sub_pair(x, d0 + (float)e, d0 + (float)(e + 1));
                  float x0, x1, s0, s1;
                  f2_unpack(x, x0, x1);
                  // (one exponential in four on the FMA pipe, as in the forward, changed nothing here)
                  x0 = c * 8 + e < first ? 0.f : ex2_approx_b(x0);
                  x1 = c * 8 + e + 1 < first ? 0.f : ex2_approx_b(x1);
                  const uint64_t d = f2_add(f2_pack(__uint_as_float(dv[e]), __uint_as_float(dv[e + 1])),
                                            k ? f2_pack(d4.z, d4.w) : f2_pack(d4.x, d4.y));
                  f2_unpack(f2_mul(f2_pack(x0, x1), d), s0, s1);
                  pk[c * 4 + e / 2] = pack2<T>(x0, x1);
                  dk_[c * 4 + e / 2] = pack2<T>(s0, s1);
                }
              }
            }
          }
          // Pᵀ / dSᵀ of the previous tile are still being read by its gradient products
          if (g > 0) ok = mbar_wait(dq_full, (g - 1) & 1, 0x2650, abort_flag);
        }
        // T is a multiple of 64, so a warp's 32 queries are all real or all past the sequence's end.  The latter get exact
        // zeros: what was worked out from the zero-filled rows is NaN where K or V holds an infinity.
        if (RAGGED && i0 + cq * 32 >= p.T) {
#pragma unroll
          for (int e = 0; e < 16; ++e) pk[e] = dk_[e] = 0u;
        }
        if (it == 0 && n > 0 && ok) store_item(wp);  // (the wait for dq_full above was for its last tile)
        if (ok) {
          tmem_st16(lane_addr + COL_PT + cq * 16, pk);  // this thread's 32 queries of Pᵀ
#pragma unroll
          for (int v4 = 0; v4 < 4; ++v4) {
            const int cc = cq * 4 + v4;  // 16-byte chunk index along the 128 queries
            const uint32_t off = (cc >> 3) * 16384 + r * 128 + (((cc & 7) ^ (r & 7)) << 4);
            *reinterpret_cast<uint4*>(sds + off) = make_uint4(dk_[v4 * 4], dk_[v4 * 4 + 1], dk_[v4 * 4 + 2], dk_[v4 * 4 + 3]);
          }
          tc_wait_st();
          tc_fence_before();
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(pds_full);
        }
      }
      Item wn = w;
      const bool more = __all_sync(0xffffffffu, ok) != 0 && next_of(n, wn, false);
      if (more) load_stat(wn, 0, lse_next, delta_next);  // on their way while this item is finished
      if (!more) {
        if (ok) ok = mbar_wait(dq_full, (g - 1) & 1, 0x2680, abort_flag);
        if (ok) store_item(w);
      }
      if (!more || !ok) break;
      wp = w;
      w = wn;
      }
    }
  } else {
    regs_down<FB_REGS_DRAIN>();
    if (!dead) {
    // ---------------------------------------------------------------------------- dQ drain
    // the second warpgroup: lanes are query rows here; each warp adds its 32 rows of dQ_i to the fp32 accumulator.
    // The rows go through swizzled shared-memory boxes and the TMA unit performs the
    // reduction (cp.reduce.async.bulk.tensor), which keeps the load/store path free for the compute warps.
    const int qd = warp & 3;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
    uint8_t* stage = smem + OFF_DQ + (warp - 4) * 4096;
    if (lane == 0) tma_prefetch_desc(&tmDQ);
    Item w = item_of(blockIdx.x);
    int g = 0;
    bool ok = true;
    for (int n = 0; ok; ++n) {
    const int bh = w.bh;
    for (int it = 0; it < nq - w.kt; ++it, ++g) {
      const int i0 = (w.kt + it) * FB_T;
      if (!mbar_wait(dq_full, g & 1, 0x2700, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const int row0 = (int)((int64_t)bh * p.T) + i0 + qd * 32;
#pragma unroll
      for (int c = 0; c < 2; ++c) {  // chunks of 32 columns
        uint32_t v[32];
        tmem_ld32(lane_addr + COL_DQ + c * 32, v);
        if (lane == 0) tma_store_wait_read();  // the box has been read by the TMA unit
        __syncwarp();
        tc_wait_ld();
        if (c == 1) {  // tensor memory is drained: the tensor core may overwrite dQ while the rows travel on
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_free);
        }
        if (c * 32 < p.hd) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {  // 16-byte chunks (4 floats) of this row
            const uint32_t off = lane * 128 + ((j ^ (lane & 7)) << 4);
            *reinterpret_cast<uint4*>(stage + off) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (!RAGGED || i0 + qd * 32 < p.T) tma_reduce_add_2d(&tmDQ, stage, c * 32, row0);  // the rows past the end are the next slice's
            tma_store_commit();
          }
        }
      }
    }
    ok = __all_sync(0xffffffffu, ok) != 0 && next_of(n, w, false);
    }
    if (lane == 0) tma_store_wait_all();  // every reduction has reached global memory
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int k = 0; k < 64; ++k) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// dq = round(scale * dq_acc), written with the caller's strides.  Bound by memory; one slice per grid row, vectors of eight
// columns, 1 << vshift of them per row (no 64-bit divisions to find a vector's row).  Backward before and with this and the delta pass
// of that time: B4 H16 T2048 hd64 fp16 191.5 -> 189.6 us, B3 H11 T1472 hd64 bf16 69.0 -> 67.0, B1 H12 T4096 hd128 226.5 -> 222.7.
constexpr int DQ_VECS = 2;  // of a thread
template <typename T>
__global__ void __launch_bounds__(256) attn_dq_convert_kernel(const float* __restrict__ acc, T* __restrict__ dq,
                                                              int64_t sb, int64_t sh, int64_t st, int H, int rows, int vshift,
                                                              float scale) {
  grid_dependency_wait();
  allow_dependents();
  const int bh = blockIdx.y, b = bh / H, h = bh % H;
  const int total = rows << vshift;
  const float4* src = reinterpret_cast<const float4*>(acc) + (int64_t)bh * total * 2;
  T* dst = dq + b * sb + h * sh;
  float4 x[DQ_VECS], y[DQ_VECS];
#pragma unroll
  for (int u = 0; u < DQ_VECS; ++u) {
    const int v = (blockIdx.x * DQ_VECS + u) * 256 + threadIdx.x;
    if (v < total) {
      x[u] = __ldcs(src + 2 * (int64_t)v);
      y[u] = __ldcs(src + 2 * (int64_t)v + 1);
    }
  }
#pragma unroll
  for (int u = 0; u < DQ_VECS; ++u) {
    const int v = (blockIdx.x * DQ_VECS + u) * 256 + threadIdx.x;
    if (v < total) {
      const float f[8] = {x[u].x * scale, x[u].y * scale, x[u].z * scale, x[u].w * scale,
                          y[u].x * scale, y[u].y * scale, y[u].z * scale, y[u].w * scale};
      *reinterpret_cast<uint4*>(dst + (int64_t)(v >> vshift) * st + (v & ((1 << vshift) - 1)) * 8) = pack8<T>(f);
    }
  }
}

// ------------------------------------------------------------------------------- host side

static int encode_bhtd(CUtensorMap* m, const void* ptr, const AttnStrides& s, int B, int H, int T, int hd, int dtype) {
  const uint64_t dims[4] = {(uint64_t)hd, (uint64_t)T, (uint64_t)H, (uint64_t)B};
  const uint64_t str[3] = {(uint64_t)s.t * 2, (uint64_t)s.h * 2, (uint64_t)s.b * 2};
  const uint32_t box[4] = {64, 128, 1, 1};
  return encode_tmap_sw128(m, ptr, dtype, 4, dims, str, box);
}

bool attn_tc05_bwd_eligible(const AttnArgs& a, int hd) {  // as in the forward
  return a.bias_mode != 3 && (attn_whole_tiles(a, hd) || (attn_strides_positive(a.sq) && attn_strides_positive(a.sk) &&
                                                          attn_strides_positive(a.sv) && attn_strides_positive(a.sdo)));
}

int attn_bwd128_tc05(const AttnArgs& a, int dtype, cudaStream_t st);
int attn_bwd128_fits(const AttnArgs& a, int dtype, bool& fit);

namespace {  // (not shared with another copy of the library in the process)
template <typename T, bool RAGGED>
struct Bwd64 {
  using Kernel = decltype(&attn_bwd_tc05_kernel<T, 0, RAGGED>);
  static inline std::atomic<uint64_t> smem_done[5] = {};
  static inline std::atomic<int> registers[5] = {};
  static Kernel kernel(int mode) {
    return mode == 0 ? attn_bwd_tc05_kernel<T, 0, RAGGED> : mode == 1 ? attn_bwd_tc05_kernel<T, 1, RAGGED>
         : mode == 2 ? attn_bwd_tc05_kernel<T, 2, RAGGED> : attn_bwd_tc05_kernel<T, 4, RAGGED>;
  }
  static int fits(const AttnArgs& a, bool& fit) {
    return registers_fit(kernel(a.bias_mode), FB_REGS, FB_REGS_COMPUTE, registers[a.bias_mode], "attention_bwd(tcgen05)", fit);
  }
};
}  // namespace

// Whether the kernel that would take the call has the registers that its split counts on.  If not, the mma.sync kernels take it.
int attn_tc05_bwd_fits(const AttnArgs& a, int hd, int dtype, bool& fit) {
  if (hd == 128) return attn_bwd128_fits(a, dtype, fit);
  TFB_DISPATCH_16(dtype, T, { return a.T % FB_T ? Bwd64<T, true>::fits(a, fit) : Bwd64<T, false>::fits(a, fit); })
}

template <typename T, bool RAGGED>
static int bwd64_launch(const AttnArgs& a, int hd, int dtype, cudaStream_t st) {
  int rc;
  CUtensorMap tq, tk, tv, tdo, tdq;
  {
    // fp32 dQ accumulator as a (HD, B*H*T) matrix, boxes of 32 floats x 32 rows
    const uint64_t dims[2] = {(uint64_t)hd, (uint64_t)a.B * a.H * a.T};
    const uint64_t str[1] = {(uint64_t)hd * 4};
    const uint32_t box[2] = {32, 32};
    if ((rc = encode_tmap_sw128(&tdq, a.dq_acc, TFB_F32, 2, dims, str, box))) return rc;
  }
  if ((rc = encode_bhtd(&tq, a.q, a.sq, a.B, a.H, a.T, hd, dtype))) return rc;
  if ((rc = encode_bhtd(&tk, a.k, a.sk, a.B, a.H, a.T, hd, dtype))) return rc;
  if ((rc = encode_bhtd(&tv, a.v, a.sv, a.B, a.H, a.T, hd, dtype))) return rc;
  if ((rc = encode_bhtd(&tdo, a.d_o, a.sdo, a.B, a.H, a.T, hd, dtype))) return rc;
  FbParams p;
  p.lse = a.lse; p.delta = a.delta; p.dk = a.dk; p.dv = a.dv;
  p.sdk_b = a.sdk.b; p.sdk_h = a.sdk.h; p.sdk_t = a.sdk.t;
  p.sdv_b = a.sdv.b; p.sdv_h = a.sdv.h; p.sdv_t = a.sdv.t;
  p.H = a.H; p.T = a.T; p.hd = hd; p.scale = a.scale; p.slopes = a.slopes;
  p.debug = g_attn_debug.load();
  p.status = dev_status_address();
  if (!p.status) return fail(TFB_ERR_LAUNCH, "attention_bwd(tcgen05): cannot find the status word");
  p.BH = a.B * a.H;
  p.group = attn_slices_per_group(a.B * a.H, a.T, HD);
  dim3 grid((unsigned)ceil_div(a.T, FB_T) * a.B * a.H);
  using Form = Bwd64<T, RAGGED>;
  const auto kernel = Form::kernel(a.bias_mode);
  if ((rc = ensure_dynamic_smem(kernel, SMEM_BYTES, Form::smem_done[a.bias_mode], "attention_bwd(tcgen05)"))) return rc;
  launch_overlapped(kernel, grid, dim3(FB_THREADS), SMEM_BYTES, st, tq, tk, tv, tdo, tdq, p);
  return launched("attention_bwd(tcgen05)");
}

template <typename T>
static int bwd_tc05_launch(const AttnArgs& a, int hd, int dtype, cudaStream_t st) {
  // the delta pass also clears the fp32 dQ accumulator (contiguous (B,H,T,hd), 16-byte aligned: checked by the
  // caller), so no fill sits between the kernels in the stream
  int rc = attn_delta(a, hd, dtype, st, a.dq_acc);
  if (!rc)
    rc = hd == 128 ? attn_bwd128_tc05(a, dtype, st)
                   : a.T % FB_T ? bwd64_launch<T, true>(a, hd, dtype, st) : bwd64_launch<T, false>(a, hd, dtype, st);
  if (rc) return rc;
  const int vshift = hd == 32 ? 2 : hd == 64 ? 3 : 4;
  const dim3 grid((unsigned)ceil_div((int64_t)a.T << vshift, 256 * DQ_VECS), (unsigned)(a.B * a.H));
  launch_overlapped(attn_dq_convert_kernel<T>, grid, dim3(256), 0, st, a.dq_acc, (T*)a.dq, a.sdq.b, a.sdq.h, a.sdq.t, a.H, a.T,
                    vshift, a.scale);
  return launched("attention_dq_convert");
}

int attn_tc05_bwd(const AttnArgs& a, int hd, int dtype, cudaStream_t st) {
  TFB_DISPATCH_16(dtype, T, {
    return bwd_tc05_launch<T>(a, hd, dtype, st);
  })
}

}  // namespace tfb
