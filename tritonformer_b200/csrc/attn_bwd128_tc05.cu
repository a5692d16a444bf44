// Causal flash attention backward on tcgen05 / TMEM for head_dim 128 (sm_100a): two sub-tiles of 64 queries in flight.
//
// The arithmetic is the one of attn_bwd_tc05.cu, transposed (rows = keys), in sub-tiles of 128 keys x 64 queries:
//   Sᵀ  = K Q_iᵀ                 dPᵀ = V dO_iᵀ                      (tensor cores -> TMEM)
//   Pᵀ  = 2^(Sᵀ·c + bias - lse)  dSᵀ = Pᵀ ∘ (dPᵀ - delta)            (compute warps -> TMEM / shared memory, 16 bit)
//   dV += Pᵀ dO_i     dK += dSᵀ Q_i     dQ_i = dS K                  (tensor cores -> TMEM)
// An item is a (128-key tile, batch*head); a CTA walks the sub-tiles at or below the diagonal.  dV and dK stay in TMEM for the
// whole walk; dQ_i is added to an fp32 global accumulator (TMA reduce-add), which a small kernel scales and rounds afterwards.
//
// What bounds it: the chain scores -> exponentials -> gradient products -> dQ read-out of a sub-tile, whose links use different
// parts of the SM (tensor core, SFU, shared memory, TMA unit) one after the other.  dV and dK take half of tensor memory; with
// tiles of 128 queries the scores of one tile fill the other half and the links add up.  With 64 queries there is
// room for TWO chains that fill each other's gaps: two slots of 128 columns that take the sub-tiles in turn, with eight
// compute warps each.  With the two small passes, against one tile of 128 queries at a time: B1 H12 T4096 fp16 253.7 -> 226.5 us,
// T4032 254 -> 221, B2 H16 T2048 bf16 with the rounded table 201 -> 180.
//
// TMEM columns of a slot: [0,64) Sᵀ, over it Pᵀ (16-bit, at the head of each warp's own score columns: the A operand of the dV
// product); [64,128) dPᵀ; over both dQ_i (M = 64: row 16 q + r sits in lane 32 q + r).  [256,384) dV, [384,512) dK.
// Roles: warp 0 TMA producer, warp 1 MMA issuer, from warp 4 on eight compute warps per slot: two per TMEM lane quarter, 32 query columns
// each; they also hand dQ to the TMA unit.
// A swizzled panel of 64 16-bit values per row is at the same time a K-major operand and an MN-major one, so each of K, V,
// Q_i, dO_i, dSᵀ sits in shared memory once and serves two products.
// Sequences are multiples of 64, so every sub-tile of queries is real; keys past the end are zero rows (TMA fill) that the
// causal mask keeps from every query.  A warp's 32 x 32 block is, as a whole, untouched by the mask, cut by the diagonal, or
// masked (nothing is computed).
#define TFB_STATUS_FROM_LAUNCH
#include "attn.cuh"
#include "tc05.cuh"
#include <type_traits>

namespace tfb {

extern std::atomic<int> g_attn_debug;

namespace {

constexpr float kLog2eB = 1.4426950408889634f;
constexpr int FB_K = 128;       // keys per item
constexpr int FB_Q = 64;        // queries per sub-tile
constexpr int FB_CWARPS = 8;    // compute warps per slot

constexpr int HD = 128;
constexpr int PANELS = 2;          // 64-element (128-byte) panels along head_dim
constexpr int SLOTS = 2;
// Warpgroups: TMA, MMA and two idle warps; the compute warps.  The block is launched with 96 registers a thread (five warps per
// scheduler); the first group hands most of its own on to the compute warps: B1 H12 T4096 fp16 222.7 -> 214.8 us, T4032 217 -> 210,
// B2 H16 T2048 bf16 with the rounded table 177 -> 170.
constexpr int FIRST_C = 4;         // first compute warp
constexpr int THREADS = 32 * (FIRST_C + FB_CWARPS * SLOTS);
constexpr int REGS = 96, REGS_ISSUE = 32, REGS_COMPUTE = 112;
static_assert(128 * REGS_ISSUE + 32 * FB_CWARPS * SLOTS * REGS_COMPUTE <= THREADS * REGS, "registers of the block");
constexpr int KV_BYTES = PANELS * FB_K * 128, Q_BYTES = PANELS * FB_Q * 128;
constexpr int QS = 2;              // Q / dO ring depth
constexpr int DS_BYTES = FB_K * FB_Q * 2;
constexpr int OFF_K = 0, OFF_V = KV_BYTES;
constexpr int OFF_Q = 2 * KV_BYTES;                          // [QS][Q, dO]
constexpr int OFF_DS = OFF_Q + QS * 2 * Q_BYTES;             // [SLOTS] dSᵀ 128 keys x 64 queries
constexpr int OFF_DQ = OFF_DS + SLOTS * DS_BYTES;            // [compute warps] box of 16 rows x 32 columns fp32
constexpr int OFF_STAT = OFF_DQ + SLOTS * FB_CWARPS * 2048;  // [2 parities][compute warps][-lse2[32], -delta[32]] fp32
constexpr int OFF_BAR = OFF_STAT + 2 * SLOTS * FB_CWARPS * 256;
constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
constexpr int COL_DV = SLOTS * 128, COL_DK = COL_DV + HD;

struct FbParams {
  int* status;    // the library's status word
  const float* lse;
  const float* delta;
  void *dk, *dv;
  int64_t sdk_b, sdk_h, sdk_t, sdv_b, sdv_h, sdv_t;
  int H, T;
  int BH, group;  // batch*heads; how many of them are walked together (their tiles share the L2)
  float scale;
  const float* slopes;
  int debug;      // bit 5: per-slice item order (test switch)
};

__device__ __forceinline__ float fb_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <typename T>
__device__ __forceinline__ uint32_t fb_pack(uint64_t v) {
  float a, b;
  f2_unpack(v, a, b);
  typename Num<T>::T2 h = Num<T>::from_f2(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

}  // namespace

template <typename T, int BIAS>
__global__ void __launch_bounds__(THREADS, 1)
    attn_bwd128_tc05_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                         const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                         const __grid_constant__ CUtensorMap tmDQ, const FbParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* s_stat = reinterpret_cast<float*>(smem + OFF_STAT);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* kv_full = bars + 0;         // K and V landed
  uint64_t* done = bars + 1;            // the last gradient products have retired
  uint64_t* q_full = bars + 2;          // [QS] Q_i and dO_i landed
  uint64_t* q_empty = q_full + QS;      // [QS] the products that read them have retired
  uint64_t* s_full = q_empty + QS;      // [SLOTS] Sᵀ in TMEM
  uint64_t* dp_full = s_full + SLOTS;   // [SLOTS] dPᵀ in TMEM
  uint64_t* pds_full = dp_full + SLOTS; // [SLOTS] Pᵀ and dSᵀ stored; Sᵀ and dPᵀ read
  uint64_t* dq_full = pds_full + SLOTS; // [SLOTS] dQ_i in TMEM
  uint64_t* dq_free = dq_full + SLOTS;  // [SLOTS] dQ_i read out
  uint64_t* box_free = dq_free + SLOTS; // [SLOTS][4 lane quarters] the TMA unit has read dQ_i out of the quarter's dSᵀ rows
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(box_free + 4 * SLOTS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Items are numbered longest walk first: within a group of batch*head slices the key tiles with the longest walk (tile 0)
  // of EVERY slice come first, so the tail of the kernel is made of short ones.
  const int nk = (p.T + FB_K - 1) / FB_K;
  int kt, bh;
  {
    const int block = (int)blockIdx.x;
    if (p.debug & 32) {  // per-slice order (test switch)
      kt = block % nk;
      bh = block / nk;
    } else {
      const int g = block / (nk * p.group), r = block % (nk * p.group);
      const int gsz = min(p.group, p.BH - g * p.group);
      kt = r / gsz;
      bh = g * p.group + r % gsz;
    }
  }
  const int b = bh / p.H, h = bh % p.H;
  const int i_first = kt * FB_K;                  // first query that sees a key of the tile
  const int n = (p.T - i_first) / FB_Q;           // sub-tiles of the walk; slot g % SLOTS takes the g-th

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(done, 1);
    for (int i = 0; i < QS; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < SLOTS; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&dp_full[i], 1);
      mbar_init(&pds_full[i], FB_CWARPS);
      mbar_init(&dq_full[i], 1);
      mbar_init(&dq_free[i], FB_CWARPS);
      for (int q = 0; q < 4; ++q) mbar_init(&box_free[i * 4 + q], 2);
    }
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

  if (warp < FIRST_C) {
  regs_down<REGS_ISSUE>();
  if (warp == 0) {
    // --------------------------------------------------------------------- TMA producer
    if (lane == 0 && !dead) {
      mbar_expect_tx(kv_full, 2 * KV_BYTES);
#pragma unroll
      for (int c = 0; c < PANELS; ++c) {
        tma_load_4d(smem + OFF_K + c * FB_K * 128, &tmK, c * 64, i_first, h, b, kv_full);
        tma_load_4d(smem + OFF_V + c * FB_K * 128, &tmV, c * 64, i_first, h, b, kv_full);
      }
      for (int g = 0; g < n; ++g) {
        const int st = g % QS;
        if (!mbar_wait(&q_empty[st], ((g / QS) & 1) ^ 1, 0x2100 | st, abort_flag)) break;
        uint8_t* dst = smem + OFF_Q + st * 2 * Q_BYTES;
        mbar_expect_tx(&q_full[st], 2 * Q_BYTES);
#pragma unroll
        for (int c = 0; c < PANELS; ++c) {
          tma_load_4d(dst + c * FB_Q * 128, &tmQ, c * 64, i_first + g * FB_Q, h, b, &q_full[st]);
          tma_load_4d(dst + Q_BYTES + c * FB_Q * 128, &tmDO, c * 64, i_first + g * FB_Q, h, b, &q_full[st]);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ----------------------------------------------------------------------- MMA issuer
    // The whole warp runs this code and one elected lane issues each tcgen05 instruction: warp-uniform code keeps the operand
    // descriptors in uniform registers, where the tensor core reads them (a single lane needed 80-120 cycles per instruction).
    if (!dead) {
      constexpr int fmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
      constexpr uint32_t idesc_s = instr_desc_f16(FB_K, FB_Q, fmt, 0, 0);   // Sᵀ, dPᵀ: both K-major
      constexpr uint32_t idesc_kv = instr_desc_f16(FB_K, HD, fmt, 0, 1);    // dV, dK : A K-major, B MN-major
      constexpr uint32_t idesc_q = instr_desc_f16(FB_Q, HD, fmt, 1, 1);     // dQ     : both MN-major
      const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);  // read from shared memory: tell the compiler it is uniform
      const uint32_t s0 = smem_u32(smem);
      // operand descriptors; each MMA only advances the start address (K-major: 8-row groups 1024 B apart, a panel per 64
      // elements of the contraction; MN-major: 8-row groups 1024 B apart, 64-element chunks one panel apart)
      const uint64_t k_k = smem_desc_sw128(s0 + OFF_K, 16, 1024), k_mn = smem_desc_sw128(s0 + OFF_K, FB_K * 128, 1024);
      const uint64_t v_k = smem_desc_sw128(s0 + OFF_V, 16, 1024);
      const uint64_t ds_k = smem_desc_sw128(s0 + OFF_DS, 16, 1024), ds_mn = smem_desc_sw128(s0 + OFF_DS, 16384, 1024);
      const uint64_t q_k0 = smem_desc_sw128(s0 + OFF_Q, 16, 1024), q_mn0 = smem_desc_sw128(s0 + OFF_Q, FB_Q * 128, 1024);
      auto wait = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
        return __all_sync(0xffffffffu, mbar_wait(bar, parity, code, abort_flag)) != 0;
      };
      auto scores = [&](int g) {  // Sᵀ(g); Q and dO of g have landed
        const uint64_t q = desc_advance(q_k0, (g % QS) * 2 * Q_BYTES);
        const uint32_t d = tb + (g % SLOTS) * 128;
#pragma unroll
        for (int s = 0; s < HD / 16; ++s)
          if (elect_one())
            tc_mma_ss(d, desc_advance(k_k, (s / 4) * (FB_K * 128) + (s % 4) * 32), desc_advance(q, (s / 4) * (FB_Q * 128) + (s % 4) * 32),
                      idesc_s, s ? 1u : 0u);
        if (elect_one()) tc_commit(&s_full[g % SLOTS]);
      };
      auto probs = [&](int g) {  // dPᵀ(g)
        const uint64_t d_o = desc_advance(q_k0, (g % QS) * 2 * Q_BYTES + Q_BYTES);
        const uint32_t d = tb + (g % SLOTS) * 128 + 64;
#pragma unroll
        for (int s = 0; s < HD / 16; ++s)
          if (elect_one())
            tc_mma_ss(d, desc_advance(v_k, (s / 4) * (FB_K * 128) + (s % 4) * 32), desc_advance(d_o, (s / 4) * (FB_Q * 128) + (s % 4) * 32),
                      idesc_s, s ? 1u : 0u);
        if (elect_one()) tc_commit(&dp_full[g % SLOTS]);
      };
      auto grad_v = [&](int g) {
        const uint64_t d_o = desc_advance(q_mn0, (g % QS) * 2 * Q_BYTES + Q_BYTES);
        const uint32_t pt = tb + (g % SLOTS) * 128;
#pragma unroll
        for (int s = 0; s < FB_Q / 16; ++s)  // 16 queries each; Pᵀ at columns 0-15 and 32-47
          if (elect_one())
            tc_mma_ts(tb + COL_DV, pt + (s >> 1) * 32 + (s & 1) * 8, desc_advance(d_o, s * 2048), idesc_kv, (g | s) ? 1u : 0u);
      };
      auto grad_q = [&](int g) {
        const uint64_t ds = desc_advance(ds_mn, (g % SLOTS) * DS_BYTES);
        const uint32_t d = tb + (g % SLOTS) * 128;
#pragma unroll
        for (int s = 0; s < FB_K / 16; ++s)  // 16 keys each
          if (elect_one()) tc_mma_ss(d, desc_advance(ds, s * 2048), desc_advance(k_mn, s * 2048), idesc_q, s ? 1u : 0u);
        if (elect_one()) tc_commit(&dq_full[g % SLOTS]);  // with it, all that read the sub-tile's dSᵀ
      };
      auto grad_k = [&](int g) {
        const uint64_t ds = desc_advance(ds_k, (g % SLOTS) * DS_BYTES), q = desc_advance(q_mn0, (g % QS) * 2 * Q_BYTES);
#pragma unroll
        for (int s = 0; s < FB_Q / 16; ++s)
          if (elect_one()) tc_mma_ss(tb + COL_DK, desc_advance(ds, s * 32), desc_advance(q, s * 2048), idesc_kv, (g | s) ? 1u : 0u);
      };
      bool ok = wait(kv_full, 0, 0x2200);
      {
        // Event loop over two cursors.  The scores of a slot go out once its dQ has been read out, gradient products once Pᵀ
        // and dSᵀ are stored.
        auto ready = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_test(bar, parity)) != 0; };
        int sg = 0, pg = 0;
        uint64_t t_idle = global_ns();
        while (ok && pg < n) {
          bool progress = false;
          if (sg < n && (sg < SLOTS || (sg - SLOTS < pg && ready(&dq_free[sg % SLOTS], (sg / SLOTS - 1) & 1))) &&
              ready(&q_full[sg % QS], (sg / QS) & 1)) {
            tc_fence_after();
            scores(sg);
            probs(sg);
            ++sg;
            progress = true;
          }
          if (pg < sg && ready(&pds_full[pg % SLOTS], (pg / SLOTS) & 1)) {
            tc_fence_after();
            grad_v(pg);
            grad_k(pg);
            grad_q(pg);
            if (elect_one()) tc_commit(&q_empty[pg % QS]);
            ++pg;
            if (pg == n && elect_one()) tc_commit(done);
            progress = true;
          }
          if (progress) {
            t_idle = global_ns();
          } else if (__any_sync(0xffffffffu, *abort_flag != 0)) {
            ok = false;
          } else if (__any_sync(0xffffffffu, global_ns() - t_idle > kWaitLimitNs)) {
            if (lane == 0) {
              *abort_flag = 1;
              atomicCAS(dev_status(), 0, 0x2550);
            }
            ok = false;
          } else {
            __nanosleep(20);
          }
        }
      }
    }
    __syncwarp();
  }
  } else {
    regs_up<REGS_COMPUTE>();
    if (!dead) {
    // -------------------------------------------------------------------------- compute
    const int cw = warp - FIRST_C;
    const int slot = cw / FB_CWARPS;
    const int qd = warp & 3;                 // TMEM lane quarter
    const int cq = (cw % FB_CWARPS) >> 2;    // which half (32) of the 64 query columns
    const int r = qd * 32 + lane;            // TMEM lane = key row
    const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t slot_addr = lane_addr + slot * 128;
    const float c2 = p.scale * kLog2eB;
    const uint64_t c2p = f2_pack(c2, c2);
    uint8_t* sds = smem + OFF_DS + slot * DS_BYTES + r * 128;
    uint8_t* const box[2] = {smem + OFF_DQ + cw * 2048, smem + OFF_DS + slot * DS_BYTES + qd * 4096 + cq * 2048};
    const AlibiLog2<BIAS> alibi(BIAS ? p.slopes[h] : 0.f);
    bool ok = true;
    if (lane == 0) tma_prefetch_desc(&tmDQ);
    // Statistics of the warp's 32 query columns: lane l carries those of column l, fetched one sub-tile ahead, and hands them
    // to the other lanes through a slice of shared memory that belongs to this warp.
    const float* lse_at = p.lse + (int64_t)bh * p.T + i_first + cq * 32 + lane;
    const float* delta_at = p.delta + (int64_t)bh * p.T + i_first + cq * 32 + lane;
    float lse_next = 0.f, delta_next = 0.f;
    if (slot < n) {
      lse_next = lse_at[slot * FB_Q];
      delta_next = delta_at[slot * FB_Q];
    }
    // dQ of sub-tile g: this warp's 16 rows and 64 columns, through two boxes of 32 columns, to the accumulator.  The second
    // box lies in the rows of dSᵀ that this warp and the other one of its lane quarter write: every product that reads
    // them has retired.  (Through one box after the other the read-out of a sub-tile took 2.1 k cycles instead of 0.6 k.)
    auto drain = [&](int g) {
      if (ok) ok = mbar_wait(&dq_full[slot], (g / SLOTS) & 1, 0x2700, abort_flag);
      if (!ok) return;
      tc_fence_after();
      uint32_t v[2][16];
#pragma unroll
      for (int c = 0; c < 2; ++c) tmem_ld_half32(slot_addr + cq * 64 + c * 32, v[c]);
      if (lane == 0) tma_store_wait_read();  // the first box has been read (the second one: box_free)
      __syncwarp();
      tc_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dq_free[slot]);
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // rows lane / 4 and lane / 4 + 8, two columns each
          uint8_t* at = box[c] + (lane >> 2) * 128 + (((j * 2 + ((lane & 3) >> 1)) ^ (lane >> 2)) << 4) + (lane & 1) * 8;
          *reinterpret_cast<uint2*>(at) = make_uint2(v[c][4 * j], v[c][4 * j + 1]);
          *reinterpret_cast<uint2*>(at + 1024) = make_uint2(v[c][4 * j + 2], v[c][4 * j + 3]);
        }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        const int row0 = (int)((int64_t)bh * p.T) + i_first + g * FB_Q + qd * 16;
#pragma unroll
        for (int c = 0; c < 2; ++c) tma_reduce_add_2d(&tmDQ, box[c], cq * 64 + c * 32, row0);
        tma_store_commit();
      }
    };
    for (int g = slot; g < n && ok; g += SLOTS) {
      const uint32_t ph = (g / SLOTS) & 1;
      float* s_lse = s_stat + (ph * (SLOTS * FB_CWARPS) + cw) * 64;
      s_lse[lane] = -lse_next * kLog2eB;
      s_lse[32 + lane] = -delta_next;
      __syncwarp();
      if (g + SLOTS < n) {
        lse_next = lse_at[(g + SLOTS) * FB_Q];
        delta_next = delta_at[(g + SLOTS) * FB_Q];
      }
      // the warp's 32 x 32 block against the diagonal: < 0 masked, 0 cut, > 0 untouched
      const int rel = g * 2 + cq - qd;
      ok = mbar_wait(&s_full[slot], ph, 0x2600, abort_flag);
      if (!ok) break;
      tc_fence_after();
      uint32_t sv[32];
      tmem_ld32(slot_addr + cq * 32, sv);
      tc_wait_ld();
      uint64_t pe[16];  // Pᵀ in fp32 until dPᵀ is there
      if (rel < 0) {
#pragma unroll
        for (int e = 0; e < 16; ++e) pe[e] = 0ull;
      } else {
        const float d0 = (float)(g * FB_Q + cq * 32 - r);  // distance of the first query column to this thread's key
#pragma unroll
        for (int e4 = 0; e4 < 8; ++e4) {
          const float4 l4 = *reinterpret_cast<const float4*>(s_lse + e4 * 4);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int e = e4 * 4 + 2 * k;
            uint64_t x = f2_fma(f2_pack(__uint_as_float(sv[e]), __uint_as_float(sv[e + 1])), c2p,
                                k ? f2_pack(l4.z, l4.w) : f2_pack(l4.x, l4.y));
            if (BIAS) x = alibi.sub_pair(x, d0 + (float)e, d0 + (float)(e + 1));
            float x0, x1;
            f2_unpack(x, x0, x1);
            x0 = fb_ex2(x0);
            x1 = fb_ex2(x1);
            pe[e / 2] = f2_pack(x0, x1);
          }
        }
        if (rel == 0) {  // query column c sees key row `lane` from c = lane on
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float x0, x1;
            f2_unpack(pe[e], x0, x1);
            pe[e] = f2_pack(2 * e < lane ? 0.f : x0, 2 * e + 1 < lane ? 0.f : x1);
          }
        }
      }
      {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) pk[e] = fb_pack<T>(pe[e]);
        tmem_st16(slot_addr + cq * 32, pk);  // over this warp's own scores, which it has read
      }
      if (g >= SLOTS && ok) {  // both warps' dQ of the slot's sub-tile before has left the rows of dSᵀ
        if (lane == 0) {
          tma_store_wait_read();
          mbar_arrive(&box_free[slot * 4 + qd]);
        }
        __syncwarp();
        ok = mbar_wait(&box_free[slot * 4 + qd], (g / SLOTS - 1) & 1, 0x2720, abort_flag);
      }
      if (ok) ok = mbar_wait(&dp_full[slot], ph, 0x2610, abort_flag);
      if (!ok) break;
      tc_fence_after();
      // dSᵀ.  The products of the slot's sub-tile before have read its buffer: they retired ahead of these scores.
      if (rel < 0) {
#pragma unroll
        for (int v = 0; v < 4; ++v) *reinterpret_cast<uint4*>(sds + (((cq * 4 + v) ^ (r & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
      } else {
        uint32_t dv[32];
        tmem_ld32(slot_addr + 64 + cq * 32, dv);
        tc_wait_ld();
#pragma unroll
        for (int v = 0; v < 4; ++v) {  // 16-byte chunks along the 64 queries
          uint32_t w[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int e = v * 8 + 2 * k;
            const float2 dl = *reinterpret_cast<const float2*>(s_lse + 32 + e);
            const uint64_t d = f2_add(f2_pack(__uint_as_float(dv[e]), __uint_as_float(dv[e + 1])), f2_pack(dl.x, dl.y));
            w[k] = fb_pack<T>(f2_mul(pe[e / 2], d));
          }
          *reinterpret_cast<uint4*>(sds + (((cq * 4 + v) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      tc_wait_st();
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pds_full[slot]);
      drain(g);
    }
    if (ok) ok = mbar_wait(done, 0, 0x2680, abort_flag);
    const int col0 = (cw >> 2) * 32;  // the four warps of a lane quarter share the columns of dV and dK
    if (ok) {
      tc_fence_after();
      const int j = i_first + r;
      T* dvp = reinterpret_cast<T*>(p.dv) + b * p.sdv_b + h * p.sdv_h + (int64_t)j * p.sdv_t + col0;
      T* dkp = reinterpret_cast<T*>(p.dk) + b * p.sdk_b + h * p.sdk_h + (int64_t)j * p.sdk_t + col0;
      uint32_t v[32], u[32];
      tmem_ld32(lane_addr + COL_DV + col0, v);
      tmem_ld32(lane_addr + COL_DK + col0, u);
      tc_wait_ld();
      if (j < p.T) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[c * 8 + e]);
          *reinterpret_cast<uint4*>(dvp + c * 8) = pack8<T>(f);
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(u[c * 8 + e]) * p.scale;
          *reinterpret_cast<uint4*>(dkp + c * 8) = pack8<T>(f);
        }
      }
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

// ------------------------------------------------------------------------------- host side
static int encode_rows(CUtensorMap* m, const void* ptr, const AttnStrides& s, const AttnArgs& a, int rows, int dtype) {
  const uint64_t dims[4] = {(uint64_t)HD, (uint64_t)a.T, (uint64_t)a.H, (uint64_t)a.B};
  const uint64_t str[3] = {(uint64_t)s.t * 2, (uint64_t)s.h * 2, (uint64_t)s.b * 2};
  const uint32_t box[4] = {64, (uint32_t)rows, 1, 1};
  return encode_tmap_sw128(m, ptr, dtype, 4, dims, str, box);
}

namespace {  // (not shared with another copy of the library in the process)
template <typename T>
struct Bwd128 {
  using Kernel = decltype(&attn_bwd128_tc05_kernel<T, 0>);
  static inline std::atomic<uint64_t> smem_done[5] = {};
  static inline std::atomic<int> registers[5] = {};
  static Kernel kernel(int mode) {
    return mode == 0 ? attn_bwd128_tc05_kernel<T, 0> : mode == 1 ? attn_bwd128_tc05_kernel<T, 1>
         : mode == 2 ? attn_bwd128_tc05_kernel<T, 2> : attn_bwd128_tc05_kernel<T, 4>;
  }
};
}  // namespace

int attn_bwd128_fits(const AttnArgs& a, int dtype, bool& fit) {
  TFB_DISPATCH_16(dtype, T, {
    return registers_fit(Bwd128<T>::kernel(a.bias_mode), REGS, REGS_COMPUTE, Bwd128<T>::registers[a.bias_mode],
                         "attention_bwd(tcgen05)", fit);
  })
}

// The walk over all items; the delta pass before it and the conversion of the dQ accumulator after it are the caller's.
template <typename T>
static int bwd128_launch(const AttnArgs& a, int dtype, cudaStream_t st) {
  int rc;
  CUtensorMap tq, tk, tv, tdo, tdq;
  {
    // fp32 dQ accumulator as a (128, B*H*T) matrix, boxes of 32 floats x 16 rows
    const uint64_t dims[2] = {(uint64_t)HD, (uint64_t)a.B * a.H * a.T};
    const uint64_t str[1] = {(uint64_t)HD * 4};
    const uint32_t box[2] = {32, 16};
    if ((rc = encode_tmap_sw128(&tdq, a.dq_acc, TFB_F32, 2, dims, str, box))) return rc;
  }
  if ((rc = encode_rows(&tq, a.q, a.sq, a, FB_Q, dtype))) return rc;
  if ((rc = encode_rows(&tk, a.k, a.sk, a, FB_K, dtype))) return rc;
  if ((rc = encode_rows(&tv, a.v, a.sv, a, FB_K, dtype))) return rc;
  if ((rc = encode_rows(&tdo, a.d_o, a.sdo, a, FB_Q, dtype))) return rc;
  FbParams p;
  p.lse = a.lse; p.delta = a.delta; p.dk = a.dk; p.dv = a.dv;
  p.sdk_b = a.sdk.b; p.sdk_h = a.sdk.h; p.sdk_t = a.sdk.t;
  p.sdv_b = a.sdv.b; p.sdv_h = a.sdv.h; p.sdv_t = a.sdv.t;
  p.H = a.H; p.T = a.T; p.scale = a.scale; p.slopes = a.slopes;
  p.debug = g_attn_debug.load();
  p.status = dev_status_address();
  if (!p.status) return fail(TFB_ERR_LAUNCH, "attention_bwd(tcgen05): cannot find the status word");
  p.BH = a.B * a.H;
  p.group = attn_slices_per_group(a.B * a.H, a.T, HD);
  const dim3 grid((unsigned)ceil_div(a.T, FB_K) * a.B * a.H);
  const auto kernel = Bwd128<T>::kernel(a.bias_mode);
  if ((rc = ensure_dynamic_smem(kernel, SMEM_BYTES, Bwd128<T>::smem_done[a.bias_mode], "attention_bwd(tcgen05)"))) return rc;
  launch_overlapped(kernel, grid, dim3(THREADS), SMEM_BYTES, st, tq, tk, tv, tdo, tdq, p);
  return launched("attention_bwd(tcgen05, head_dim 128)");
}

int attn_bwd128_tc05(const AttnArgs& a, int dtype, cudaStream_t st) {
  TFB_DISPATCH_16(dtype, T, { return bwd128_launch<T>(a, dtype, st); })
}

}  // namespace tfb
