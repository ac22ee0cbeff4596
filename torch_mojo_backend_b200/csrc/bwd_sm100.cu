// Backward flash attention for sm_100a: a preprocess pass and two tcgen05 kernels, one that
// owns dK/dV and one that owns dQ.
//
// Math (same as the reference's backward kernels,
// torch_mojo_backend/eager_flash_attention/fa4_bwd_kernel.mojo:1-44, 810-980, 1443-1444,
// 1634-1662, 1855), with c = scale*log2(e):
//   dpsum = rowsum(dO * O),  lse2 = lse*log2(e)              (preprocess; stored negated, so that
//                                                             both enter packed two-wide adds and FMAs)
//   P  = exp2(S*c - lse2),   dS = P * (dP - dpsum)
//   dV = P^T dO,   dK = scale * dS^T Q,   dQ = scale * dS K
//
// The reference accumulates dQ from every K/V tile into an fp32 buffer with bulk reduce-adds
// and converts it afterwards.  On B200 that accumulation is the bottleneck: fp32 reductions
// into L2 sustain 1.9-3.3 TB/s depending on the access pattern, and a 4k-token Llama-style
// backward needs 4.4 GB of them.  Here nothing is accumulated in global memory: the
// dK/dV kernel gives each CTA one 128-row K/V tile (S^T = K Q^T, dP^T = V dO^T, so P^T and
// dS^T land in tensor memory as the A operands of dV += P^T dO and dK += dS^T Q), and the dQ
// kernel gives each CTA one 128-row query tile (S = Q K^T, dP = dO V^T, dS in tensor memory
// as the A operand of dQ += dS K).  S and dP are computed twice (7 tile GEMMs per tile pair
// instead of 5), every accumulator lives in TMEM, and the results are deterministic.
//
// dK/dV kernel: warps 0-15 are four compute warpgroups that split the 128 score columns of a tile in
// quarters (thread <-> TMEM lane), warp 16 issues every MMA, warp 17 drives TMA.  dQ kernel: warps 0-3 and
// 4-7 split the columns in halves, warps 8 and 9 each issue one of two independent MMA chains, warp 10 drives TMA.
#include <mutex>

#include "common.cuh"
#include "philox.cuh"
#include "ptx.cuh"

namespace b200fa {
namespace {

constexpr int kTile = 128;
constexpr int kThreads = 384;        // dQ kernel: 8 compute warps + 4
constexpr int kDkdvThreads = 576;    // dK/dV kernel: 16 compute warps + 2
constexpr int kSubTileBytes = 128 * 128;

template <int kD>
struct BwdCfg {
  static constexpr int kTileBytes = kTile * kD * 2;
  static constexpr int kSub = kD / 64;
  // dK/dV kernel: the resident pair of tiles, the rings of streamed tiles, then the row statistics of two steps
  static constexpr int kQStages = kD == 128 ? 3 : 4, kDoStages = kD == 128 ? 2 : 4;
  static constexpr int kOffResident = 0;
  static constexpr int kOffQ = 2 * kTileBytes;
  static constexpr int kOffDo = kOffQ + kQStages * kTileBytes;
  static constexpr int kOffStat = kOffDo + kDoStages * kTileBytes;        // [step & 1][lse2|dpsum][128] fp32
  static constexpr int kOffBars = kOffStat + 2 * 2 * 128 * 4;
  static constexpr int kNumBars = 2 * kQStages + 2 * kDoStages + 15;
  // the dQ kernel keeps 2 resident + 3 K + 2 V tiles and no per-stage statistics
  static constexpr int kOffDqBars = 7 * kTileBytes;
  static constexpr int kSmemBytes =
      (kOffBars > kOffDqBars ? kOffBars : kOffDqBars) + kNumBars * 8 + 16;
};

#define B200FA_WAIT(bar, parity, site) \
  if (!mbar_wait((bar), (parity), abort_flag, p.status, (site), p.wait_budget)) goto teardown
#define B200FA_WAIT_WARP(bar, parity, site) \
  if (!mbar_wait_warp((bar), (parity), abort_flag, p.status, (site), p.wait_budget)) goto teardown

// two exponentials on the special function unit
__device__ __forceinline__ float2 exp2_mufu2(float2 x) { return make_float2(ex2_approx(x.x), ex2_approx(x.y)); }

// ------------------------------------------------------------------------------------------
// dK / dV kernel.  One CTA = one 128-row K/V tile of one (batch, kv head); it walks every
// query tile at or below the causal diagonal for every query head of the GQA group.
// TMEM columns: two work buffers of 128, in turn: S^T of a step, over which 16-bit P^T and dS^T go (the A operands of the
// dV and dK MMAs); then the dV and dK accumulators; dP^T at D = 64 in a third buffer, at D = 128 in the other step's.
// ------------------------------------------------------------------------------------------
template <int kD, bool kBf16, bool kCausal, bool kDropout>
__global__ void __launch_bounds__(kDkdvThreads, 1)
bwd_dkdv_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapDO,
                const __grid_constant__ CUtensorMap mapDK, const __grid_constant__ CUtensorMap mapDV,
                const BwdParams p, const int sched_group) {
  using Cfg = BwdCfg<kD>;
  // TMEM: two 128-column work buffers (step i has S^T in buffer i & 1, then P^T and dS^T, 16-bit, in its place),
  // the dV and dK accumulators, and at D = 64 a third buffer for dP^T; at D = 128 dP^T is in the other step's buffer.
  constexpr bool kOwnDp = kD == 64;
  constexpr int kTmemWork = 0, kTmemDV = 256, kTmemDK = 256 + kD, kTmemDP = 384;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem + Cfg::kOffResident;
  uint8_t* sV = sK + Cfg::kTileBytes;
  uint8_t* sQ = smem + Cfg::kOffQ;
  uint8_t* sDO = smem + Cfg::kOffDo;
  float* sStat = reinterpret_cast<float*>(smem + Cfg::kOffStat);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  uint64_t* k_full = bars;                         // [1]
  uint64_t* v_full = k_full + 1;                   // [1]
  uint64_t* q_full = v_full + 1;                   // [kQStages]
  uint64_t* q_empty = q_full + Cfg::kQStages;      // [kQStages]  dK MMA (and S^T before it) done
  uint64_t* do_full = q_empty + Cfg::kQStages;     // [kDoStages]
  uint64_t* do_empty = do_full + Cfg::kDoStages;   // [kDoStages]  dV MMA (and dP^T before it) done
  uint64_t* stat_full = do_empty + Cfg::kDoStages; // [2]  lse2 and dpsum of a step
  uint64_t* stat_empty = stat_full + 2;            // [2]
  uint64_t* s_full = stat_empty + 2;               // [2]  S^T ready in work buffer b
  uint64_t* dp_full = s_full + 2;                  // dP^T ready
  uint64_t* dp_free = dp_full + 1;                 // dP^T read into registers (16 warp arrivals)
  uint64_t* p_full = dp_free + 1;                  // [2]  P^T of step i written (16 warp arrivals; two, since at D = 64 a
                                                   //      warp may be done with P^T of the next step before another arrives)
  uint64_t* ds_full = p_full + 2;                  // dS^T written (16 warp arrivals)
  uint64_t* acc_full = ds_full + 1;                // dK, dV complete
  uint64_t* staged = acc_full + 1;                 // dV and dK tiles staged in shared memory (16 warp arrivals)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::kNumBars);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  // Block order: (batch, kv head) pairs are walked `sched_group` at a time, few enough that the
  // Q / dO rows they stream stay in L2, and inside such a group the K/V tiles with the most
  // causal work (the earliest) come first, so the last wave of CTAs is made of short ones.
  const int m_tiles = (p.S + kTile - 1) / kTile;      // query tiles
  const int n_tiles = (p.Sk + kTile - 1) / kTile;     // K/V tiles (== m_tiles when causal)
  int n_tile, hk, b;
  {
    const int pairs = p.B * p.Hkv;
    const int per_group = sched_group * n_tiles;
    const int g = static_cast<int>(blockIdx.x) / per_group;
    const int gsize = min(sched_group, pairs - g * sched_group);
    const int within = static_cast<int>(blockIdx.x) - g * per_group;
    n_tile = within / gsize;
    const int pair = g * sched_group + within % gsize;
    b = pair / p.Hkv;
    hk = pair - b * p.Hkv;
  }
  const int group = p.Hq / p.Hkv;
  const int n0 = n_tile * kTile;
  // query row i sees key column j iff j <= i + causal_off: the first query tile with a row that
  // sees a key of this tile (none: the tile's dK and dV are zero)
  const int m_start = kCausal ? min(m_tiles, max(0, n0 - p.causal_off) / kTile) : 0;
  const int per_head = m_tiles - m_start;
  const int steps = group * per_head;

  // A launch whose status word already reports a failed wait is not worth running; the swizzled
  // tiles assume a 1024-byte aligned shared-memory window.
  if (status_is_set(p.status)) {
    cudaGridDependencySynchronize();   // (no kernel of a backward ends before the ones launched ahead of it)
    return;
  }
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, kStatusOk, 0x414c0000u);
    cudaGridDependencySynchronize();
    return;
  }
  // Lane 0 of the producer warp sets up the barriers and at once issues the loads the first MMAs
  // wait for, so that their latency overlaps the TMEM allocation and the block-wide synchronisation.
  auto load_tile = [&](const CUtensorMap* map, uint8_t* dst, uint64_t* bar, int srow, int head) {
#pragma unroll
    for (int cs = 0; cs < Cfg::kSub; ++cs) tma_load_4d(dst + cs * kSubTileBytes, map, bar, cs * 64, srow, head, b);
  };
  // Q, dO and the row statistics of step i into their rings
  auto load_q = [&](int i) {
    const int stage = i % Cfg::kQStages;
    mbar_arrive_expect_tx(&q_full[stage], Cfg::kTileBytes);
    load_tile(&mapQ, sQ + stage * Cfg::kTileBytes, &q_full[stage], (m_start + i % per_head) * kTile, hk * group + i / per_head);
  };
  auto load_do = [&](int i) {
    const int stage = i % Cfg::kDoStages;
    mbar_arrive_expect_tx(&do_full[stage], Cfg::kTileBytes);
    load_tile(&mapDO, sDO + stage * Cfg::kTileBytes, &do_full[stage], (m_start + i % per_head) * kTile, hk * group + i / per_head);
  };
  auto load_stat = [&](int i) {
    const int64_t off = (static_cast<int64_t>(b) * p.Hq + hk * group + i / per_head) * p.Spad + (m_start + i % per_head) * kTile;
    float* st = sStat + (i & 1) * 256;
    mbar_arrive_expect_tx(&stat_full[i & 1], 1024);
    bulk_load_1d(st, p.lse_log2 + off, 512, &stat_full[i & 1]);
    bulk_load_1d(st + 128, p.dpsum + off, 512, &stat_full[i & 1]);
  };
  if (warp == 17 && lane == 0) {
    tma_prefetch_desc(&mapK);
    tma_prefetch_desc(&mapQ);
    tma_prefetch_desc(&mapDO);
    tma_prefetch_desc(&mapV);
    mbar_init(k_full, 1);
    mbar_init(v_full, 1);
    for (int i = 0; i < Cfg::kQStages; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < Cfg::kDoStages; ++i) {
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&stat_full[i], 1);
      mbar_init(&stat_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 16);   // one elected arrival per compute warp
    }
    mbar_init(dp_full, 1);
    mbar_init(dp_free, 16);
    mbar_init(ds_full, 16);
    mbar_init(acc_full, 1);
    mbar_init(staged, 16);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    if (steps > 0) {   // (else no MMA waits for a tile, and the block must not leave with copies in flight)
      mbar_arrive_expect_tx(k_full, Cfg::kTileBytes);
      load_tile(&mapK, sK, k_full, n0, hk);
      load_q(0);
      load_do(0);
      mbar_arrive_expect_tx(v_full, Cfg::kTileBytes);
      load_tile(&mapV, sV, v_full, n0, hk);
    }
    // This kernel may have started before the preprocess kernel was done; only the row statistics come from that one.
    // Once every block has them in reach the dQ kernel may start.
    let_the_dq_kernel_start();
    if (steps > 0) load_stat(0);
  }
  if (warp == 16) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp < 16) {
    // =========================== compute warps ===========================
    const int wg = warp >> 2;                       // which 32-column (query) quarter of the tile
    const int j = (warp & 3) * 32 + lane;           // key row inside the tile == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tWork = tmem_base + lane_off + kTmemWork + wg * 32;
    const float c = p.scale_log2;
    for (int i = 0; i < steps; ++i) {
      const int m_tile = m_start + i % per_head;
      const float4* lse2 = reinterpret_cast<const float4*>(sStat + (i & 1) * 256 + wg * 32);
      const float4* dps = lse2 + 32;
      // ---- P^T = exp2(S^T * c - lse2).  P^T and then dS^T (16-bit) take the columns of S^T that this warp has read
      const uint32_t tS = tWork + (i & 1) * 128, tDP = kOwnDp ? tWork + kTmemDP : tWork + ((i + 1) & 1) * 128;
      B200FA_WAIT(&s_full[i & 1], (i >> 1) & 1, 0x500);
      B200FA_WAIT(&stat_full[i & 1], (i >> 1) & 1, 0x501);
      tc_fence_after();
      float pf[32];
      tmem_ld32(tS, reinterpret_cast<uint32_t*>(pf));
      tmem_wait_ld();
      const float2 c2 = make_float2(c, c);
#pragma unroll
      for (int e4 = 0; e4 < 8; ++e4) {
        const float4 l4 = lse2[e4];   // minus lse2
        float2 x0 = __ffma2_rn(make_float2(pf[e4 * 4 + 0], pf[e4 * 4 + 1]), c2, make_float2(l4.x, l4.y));
        float2 x1 = __ffma2_rn(make_float2(pf[e4 * 4 + 2], pf[e4 * 4 + 3]), c2, make_float2(l4.z, l4.w));
        x0 = exp2_mufu2(x0);
        x1 = exp2_mufu2(x1);
        pf[e4 * 4 + 0] = x0.x; pf[e4 * 4 + 1] = x0.y; pf[e4 * 4 + 2] = x1.x; pf[e4 * 4 + 3] = x1.y;
      }
      if (kCausal && n0 + kTile - 1 > m_tile * kTile + p.causal_off) {
        // a tile the diagonal crosses: query column q sees key row j only if j <= q + causal_off
        const int first_q = n0 + j - p.causal_off - (m_tile * kTile + wg * 32);  // first column (of these 32) that sees key j
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          if (e < first_q) pf[e] = 0.f;
        }
      }
      // dropout: bit e of `keep` <-> query column e of these 32.  Lane L draws the bits of query
      // row L against this warp's 32 key rows (two Philox calls), and the warp transposes them.
      uint32_t keep = 0xffffffffu;
      if constexpr (kDropout) {
        const int h_now = hk * group + i / per_head;
        const int q_glob = m_tile * kTile + wg * 32 + lane;
        const int blk = (n0 + (warp & 3) * 32) >> 4;
        const uint32_t mine = dropout_bits16(p.drop, b * p.Hq + h_now, q_glob, blk) |
                              (dropout_bits16(p.drop, b * p.Hq + h_now, q_glob, blk + 1) << 16);
        keep = warp_transpose_bits(mine);
      }
      {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float p0 = pf[2 * e], p1 = pf[2 * e + 1];
          if constexpr (kDropout) {
            p0 = (keep >> (2 * e)) & 1u ? p0 * p.drop.inv_keep : 0.f;
            p1 = (keep >> (2 * e)) & 2u ? p1 * p.drop.inv_keep : 0.f;
          }
          pk[e] = pack2<kBf16>(p0, p1);
        }
        tmem_st16(tS, pk);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(&p_full[i & 1]);
      // ---- dS^T = P^T * (dP^T - dpsum)
      B200FA_WAIT(dp_full, i & 1, 0x510);
      tc_fence_after();
      {
        uint32_t d[32];
        tmem_ld32(tDP, d);
        tmem_wait_ld();
        if constexpr (!kOwnDp) {   // S^T of the next step goes there
          tc_fence_before();
          mbar_arrive_warp(dp_free);
        }
        const float* df = reinterpret_cast<const float*>(d);
        uint32_t pk[16];
#pragma unroll
        for (int e4 = 0; e4 < 8; ++e4) {
          const float4 d4 = dps[e4];
          float g0 = df[e4 * 4 + 0], g1 = df[e4 * 4 + 1], g2 = df[e4 * 4 + 2], g3 = df[e4 * 4 + 3];
          if constexpr (kDropout) {
            // the gradient reaches a probability only through the entries that were kept
            const uint32_t kb = keep >> (e4 * 4);
            g0 = (kb & 1u) ? g0 * p.drop.inv_keep : 0.f;
            g1 = (kb & 2u) ? g1 * p.drop.inv_keep : 0.f;
            g2 = (kb & 4u) ? g2 * p.drop.inv_keep : 0.f;
            g3 = (kb & 8u) ? g3 * p.drop.inv_keep : 0.f;
          }
          // d4 holds minus dpsum
          const float2 s0 = __fmul2_rn(make_float2(pf[e4 * 4 + 0], pf[e4 * 4 + 1]), __fadd2_rn(make_float2(g0, g1), make_float2(d4.x, d4.y)));
          const float2 s1 = __fmul2_rn(make_float2(pf[e4 * 4 + 2], pf[e4 * 4 + 3]), __fadd2_rn(make_float2(g2, g3), make_float2(d4.z, d4.w)));
          pk[e4 * 2] = pack2<kBf16>(s0.x, s0.y);
          pk[e4 * 2 + 1] = pack2<kBf16>(s1.x, s1.y);
        }
        tmem_st16(tS + 16, pk);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(ds_full);
    }
    // ---- epilogue: dV and dK (this warpgroup's quarter of the head dimension)
    B200FA_WAIT(acc_full, 0, 0x520);
    tc_fence_after();
    {
      // The 16-bit dV and dK tiles are staged in the Q ring (every MMA that read it has
      // completed) in the swizzled box layout and leave through TMA stores: whole 128-byte
      // lines, key rows past the end of the sequence clipped by the tensor map.
      constexpr int kQuarter = kD / 4;
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        uint8_t* stage = sQ + which * Cfg::kTileBytes;
        const uint32_t tacc = tmem_base + lane_off + (which == 0 ? kTmemDV : kTmemDK) + wg * kQuarter;
        const float mul = which == 0 ? 1.f : p.scale;
        uint32_t a[kQuarter];
        if (steps > 0) {
          if constexpr (kQuarter == 32) tmem_ld32(tacc, a); else tmem_ld16(tacc, a);
          tmem_wait_ld();
        } else {
          // no query row sees this K/V tile: nothing was accumulated, the gradients are zero
#pragma unroll
          for (int e = 0; e < kQuarter; ++e) a[e] = 0u;
        }
        const float* af = reinterpret_cast<const float*>(a);
#pragma unroll
        for (int v = 0; v < kQuarter / 8; ++v) {
          uint4 w;
          w.x = pack2<kBf16>(af[v * 8 + 0] * mul, af[v * 8 + 1] * mul);
          w.y = pack2<kBf16>(af[v * 8 + 2] * mul, af[v * 8 + 3] * mul);
          w.z = pack2<kBf16>(af[v * 8 + 4] * mul, af[v * 8 + 5] * mul);
          w.w = pack2<kBf16>(af[v * 8 + 6] * mul, af[v * 8 + 7] * mul);
          const int chunk = wg * (kQuarter / 8) + v;   // 16-byte chunk of the row
          *reinterpret_cast<uint4*>(stage + (chunk >> 3) * kSubTileBytes + j * 128 + (((chunk & 7) ^ (j & 7)) << 4)) = w;
        }
      }
      fence_proxy_async_smem();
      mbar_arrive_warp(staged);
      if (threadIdx.x == 0) {
        B200FA_WAIT(staged, 0, 0x521);
#pragma unroll
        for (int cs = 0; cs < Cfg::kSub; ++cs) {
          tma_store_4d(&mapDV, sQ + cs * kSubTileBytes, cs * 64, n0, hk, b);
          tma_store_4d(&mapDK, sQ + Cfg::kTileBytes + cs * kSubTileBytes, cs * 64, n0, hk, b);
        }
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  } else if (warp == 16) {
    // =========================== MMA issuer ===========================
    // One warp issues all four products, so that the order on the tensor pipe is the program's: what a later
    // product overwrites in tensor memory, the earlier ones have read.  It runs converged, with one elected lane
    // per MMA (behind an `if (lane == 0)` every MMA cost its lane 45 cycles of operand moves).
    // The bound at D = 128: a step's MMAs take 2048 cycles, and the 6 KB that shared memory moves per 64 of them (two
    // operands of S^T and dP^T, one of dV and dK, the tiles coming in) as long again.  P^T therefore goes to tensor
    // memory over the scores it came from, and not to a tile in shared memory (whose stores and reads took 768 cycles
    // more a step, and its 32 KB the place of a third Q stage); dP^T needs the other buffer for that, so S^T of the
    // next step starts when dP^T has been read.  At D = 64 tensor memory has room for a third buffer, and S^T runs a
    // step ahead.  B200, us, with P^T in shared memory / this: B4 Hq32 Hkv8 S4096 D128 bf16 causal 964 / 903,
    // B8 H16 S2048 D128 fp16 492 / 467, B8 H12 S1024 D64 bf16 causal 57.8 / 51.4, B8 H16 S4096 D64 fp16 1246 / 1033.
    constexpr uint32_t idesc_st = umma_idesc(kBf16, false, false, 128, 128);  // S^T, dP^T
    constexpr uint32_t idesc_acc = umma_idesc(kBf16, false, true, 128, kD);   // dV, dK (A in TMEM)
    const uint32_t tWork = tmem_base + kTmemWork, tDV = tmem_base + kTmemDV, tDK = tmem_base + kTmemDK;
    const UmmaDesc kK = umma_desc_split(smem_u32(sK), 16, 1024), kV = umma_desc_split(smem_u32(sV), 16, 1024);
    const UmmaDesc kQ = umma_desc_split(smem_u32(sQ), 16, 1024);                         // ring base, K-major
    const UmmaDesc kDO = umma_desc_split(smem_u32(sDO), 16, 1024);
    const UmmaDesc mQ = umma_desc_split(smem_u32(sQ), kSubTileBytes, 1024);              // ring base, MN-major
    const UmmaDesc mDO = umma_desc_split(smem_u32(sDO), kSubTileBytes, 1024);
    constexpr uint32_t kTileLo = umma_off(Cfg::kTileBytes);
    // acc[128 x 128] = A[128 x D] * B[128 x D]^T, both K-major
    auto issue_kmajor = [&](uint32_t d_tmem, const UmmaDesc& a, const UmmaDesc& bd, uint32_t b_stage_lo) {
#pragma unroll
      for (int kk = 0; kk < kD / 16; ++kk) {
        const uint32_t off = umma_off((kk >> 2) * kSubTileBytes + (kk & 3) * 32);
        umma_ss_elect(d_tmem, a.lo + off, a.hi, bd.lo + b_stage_lo + off, bd.hi, idesc_st, kk > 0);
      }
    };
    // acc[128 x D] += A[128 x 128] (16-bit, in TMEM from `a_tmem`: 16 columns of every 32) * B[128 x D]
    auto issue_acc = [&](uint32_t d_tmem, uint32_t a_tmem, const UmmaDesc& bd, uint32_t b_stage_lo, bool first) {
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_ts_elect(d_tmem, a_tmem + (kk >> 1) * 32 + (kk & 1) * 8, bd.lo + b_stage_lo + umma_off(kk * 2048), bd.hi, idesc_acc,
                      !(kk == 0 && first));
    };
    int q_next = 0, do_next = 0;               // ring stage that the next S^T, dP^T reads
    uint32_t q_phase = 0, do_phase = 0;
    int q_stage = 0, do_stage = 0;             // ring stage that the next dK, dV reads
#define B200FA_ISSUE_S(step)                                                  \
  do {                                                                        \
    B200FA_WAIT_WARP(&q_full[q_next], q_phase, 0x711);                        \
    tc_fence_after();                                                         \
    issue_kmajor(tWork + ((step) & 1) * 128, kK, kQ, q_next * kTileLo);       \
    umma_commit_elect(&s_full[(step) & 1]);                                   \
    if (++q_next == Cfg::kQStages) { q_next = 0; q_phase ^= 1; }              \
  } while (0)
#define B200FA_ISSUE_DP(step)                                                 \
  do {                                                                        \
    B200FA_WAIT_WARP(&do_full[do_next], do_phase, 0x713);                     \
    tc_fence_after();                                                         \
    issue_kmajor(kOwnDp ? tWork + kTmemDP : tWork + (((step) + 1) & 1) * 128, kV, kDO, do_next * kTileLo); \
    umma_commit_elect(dp_full);                                               \
    if (++do_next == Cfg::kDoStages) { do_next = 0; do_phase ^= 1; }          \
  } while (0)
    if (steps > 0) {
      B200FA_WAIT_WARP(k_full, 0, 0x700);
      B200FA_ISSUE_S(0);
      B200FA_WAIT_WARP(v_full, 0, 0x701);
      B200FA_ISSUE_DP(0);
      if (kOwnDp && steps > 1) B200FA_ISSUE_S(1);
    }
    for (int i = 0; i < steps; ++i) {
      const uint32_t tS = tWork + (i & 1) * 128;
      if (!kOwnDp && i + 1 < steps) {
        // S^T of the next step goes ahead of this one's dV: it is what the compute warps wait for
        B200FA_WAIT_WARP(dp_free, i & 1, 0x717);
        B200FA_ISSUE_S(i + 1);
      }
      B200FA_WAIT_WARP(&p_full[i & 1], (i >> 1) & 1, 0x710);
      tc_fence_after();
      issue_acc(tDV, tS, mDO, do_stage * kTileLo, i == 0);          // dV += P^T dO
      umma_commit_elect(&do_empty[do_stage]);
      B200FA_WAIT_WARP(ds_full, i & 1, 0x712);
      tc_fence_after();
      issue_acc(tDK, tS + 16, mQ, q_stage * kTileLo, i == 0);       // dK += dS^T Q
      umma_commit_elect(&q_empty[q_stage]);
      umma_commit_elect(&stat_empty[i & 1]);
      if (i + 1 < steps) B200FA_ISSUE_DP(i + 1);
      if (kOwnDp && i + 2 < steps) B200FA_ISSUE_S(i + 2);
      if (++q_stage == Cfg::kQStages) q_stage = 0;
      if (++do_stage == Cfg::kDoStages) do_stage = 0;
    }
    umma_commit_elect(acc_full);
#undef B200FA_ISSUE_S
#undef B200FA_ISSUE_DP
  } else if (warp == 17) {
    // =========================== TMA producer ===========================
    if (lane == 0) {
      // step 0 went out before the block-wide synchronisation
      for (int i = 1; i < steps; ++i) {
        if (i >= Cfg::kQStages) { B200FA_WAIT(&q_empty[i % Cfg::kQStages], ((i / Cfg::kQStages) - 1) & 1, 0x800); }
        load_q(i);
        if (i >= Cfg::kDoStages) { B200FA_WAIT(&do_empty[i % Cfg::kDoStages], ((i / Cfg::kDoStages) - 1) & 1, 0x801); }
        load_do(i);
        if (i >= 2) { B200FA_WAIT(&stat_empty[i & 1], ((i >> 1) - 1) & 1, 0x802); }
        load_stat(i);
      }
    }
  }

teardown:
  tc_fence_before();
  __syncthreads();
  settle_if_aborted(abort_flag);
  if (warp == 16) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------
// dQ kernel.  One CTA = one 128-row query tile of one (batch, query head); it walks the K/V
// tiles up to the causal diagonal.  Thread <-> query row, so lse2 and dpsum are per-thread
// scalars.  TMEM columns: S double-buffered at [0,128) and [128,256) (16-bit dS overwrites
// the buffer it was computed from), dP at [256,384), the dQ accumulator after that.
// ------------------------------------------------------------------------------------------
template <int kD, bool kBf16, bool kCausal, bool kDropout>
__global__ void __launch_bounds__(kThreads, 1)
bwd_dq_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
              const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapDO,
              const __grid_constant__ CUtensorMap mapDQ, const BwdParams p) {
  using Cfg = BwdCfg<kD>;
  constexpr int kTmemS = 0, kTmemDP = 256, kTmemDQ = 384;
  extern __shared__ __align__(1024) uint8_t smem[];
  // K_j is needed twice, a whole step apart (S_j, then dQ += dS_j K_j); V_j only once (dP_j).
  // Separate rings - three K slots, two V slots - keep a full step of TMA prefetch ahead of
  // the tensor pipe within the shared-memory budget.
  uint8_t* sQ = smem + Cfg::kOffResident;
  uint8_t* sDO = sQ + Cfg::kTileBytes;
  uint8_t* sK = smem + 2 * Cfg::kTileBytes;                   // [3] tiles
  uint8_t* sV = sK + 3 * Cfg::kTileBytes;                     // [2] tiles
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffDqBars);
  uint64_t* q_full = bars;                         // [1]  Q tile
  uint64_t* do_full = q_full + 1;                  // [1]  dO tile
  uint64_t* k_full = do_full + 1;                  // [3]
  uint64_t* k_empty = k_full + 3;                  // [3]
  uint64_t* v_full = k_empty + 3;                  // [2]
  uint64_t* v_empty = v_full + 2;                  // [2]
  uint64_t* s_full = v_empty + 2;                  // [2]  S buffer ready
  uint64_t* dp_full = s_full + 2;                  // dP ready
  uint64_t* ds_full = dp_full + 1;                 // dS written, dP consumed (8 warp arrivals)
  uint64_t* acc_full = ds_full + 1;                // dQ complete
  uint64_t* staged = acc_full + 1;                 // dQ tile staged in shared memory (8 warp arrivals)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::kNumBars);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const int m_tiles = (p.S + kTile - 1) / kTile;
  const int m_tile = m_tiles - 1 - static_cast<int>(blockIdx.x);  // heaviest (latest) causal tiles first
  const int h = blockIdx.y;
  const int b = blockIdx.z;
  const int hk = h / (p.Hq / p.Hkv);
  const int m0 = m_tile * kTile;
  // query row i sees key column j iff j <= i + causal_off: K/V tiles up to the one the tile's
  // last real row still sees (none: dQ of the tile is zero)
  const int nkv_total = (p.Sk + kTile - 1) / kTile;
  int n_tiles = nkv_total;
  if (kCausal) {
    const int last = min(m0 + kTile - 1, p.S - 1) + p.causal_off;
    n_tiles = last < 0 ? 0 : min(nkv_total, last / kTile + 1);
  }

  // This kernel may have started beside the dK/dV kernel.  It still ends after it: its last block waits for that, so
  // that what is ordered behind this kernel is ordered behind both.
  const bool last_block = blockIdx.x + 1 == gridDim.x && blockIdx.y + 1 == gridDim.y && blockIdx.z + 1 == gridDim.z;
  if (status_is_set(p.status)) {
    if (last_block) cudaGridDependencySynchronize();
    return;
  }
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, kStatusOk, 0x414c0001u);
    if (last_block) cudaGridDependencySynchronize();
    return;
  }
  // Lane 0 of the producer warp sets up the barriers and at once issues the loads the first MMAs
  // wait for (Q and K_0 for S_0 first), so that their latency overlaps the TMEM allocation and the
  // block-wide synchronisation.
  auto load_tile = [&](const CUtensorMap* map, uint8_t* dst, uint64_t* bar, int srow, int head) {
    mbar_arrive_expect_tx(bar, Cfg::kTileBytes);
#pragma unroll
    for (int cs = 0; cs < Cfg::kSub; ++cs) tma_load_4d(dst + cs * kSubTileBytes, map, bar, cs * 64, srow, head, b);
  };
  if (warp == 10 && lane == 0) {
    tma_prefetch_desc(&mapQ);
    tma_prefetch_desc(&mapK);
    tma_prefetch_desc(&mapDO);
    tma_prefetch_desc(&mapV);
    mbar_init(q_full, 1);
    mbar_init(do_full, 1);
    for (int i = 0; i < 3; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    mbar_init(&s_full[0], 1);
    mbar_init(&s_full[1], 1);
    mbar_init(dp_full, 1);
    mbar_init(ds_full, 8);
    mbar_init(acc_full, 1);
    mbar_init(staged, 8);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    if (n_tiles > 0) {
      load_tile(&mapQ, sQ, q_full, m0, h);
      load_tile(&mapK, sK, &k_full[0], 0, hk);
      load_tile(&mapDO, sDO, do_full, m0, h);
      load_tile(&mapV, sV, &v_full[0], 0, hk);
    }
  }
  if (warp == 8) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp < 8) {
    // =========================== compute warps ===========================
    const int wg = warp >> 2;                      // which 64-column (key) half of the tile
    const int r = (warp & 3) * 32 + lane;          // query row inside the tile == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tDP = tmem_base + lane_off + kTmemDP + wg * 64;
    const float c = p.scale_log2;
    const int64_t stat = (static_cast<int64_t>(b) * p.Hq + h) * p.Spad + m0 + r;  // padded rows exist
    const float nlse2 = __ldcg(p.lse_log2 + stat);   // minus lse2
    const float ndps = __ldcg(p.dpsum + stat);       // minus dpsum
    const float2 c2 = make_float2(c, c), nl2 = make_float2(nlse2, nlse2), nd2 = make_float2(ndps, ndps);
    for (int j = 0; j < n_tiles; ++j) {
      const int buf = j & 1;
      const uint32_t tS = tmem_base + lane_off + kTmemS + buf * 128 + wg * 64;
      B200FA_WAIT(&s_full[buf], (j >> 1) & 1, 0x900);
      tc_fence_after();
      float pf[64];
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        uint32_t s[32];
        tmem_ld32(tS + ch * 32, s);
        tmem_wait_ld();
        const float* sf = reinterpret_cast<const float*>(s);
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float2 x = __ffma2_rn(make_float2(sf[2 * e], sf[2 * e + 1]), c2, nl2);
          x = exp2_mufu2(x);
          pf[ch * 32 + 2 * e] = x.x;
          pf[ch * 32 + 2 * e + 1] = x.y;
        }
        // Columns to blank: beyond the causal diagonal, and beyond the last key.  K rows past Sk are
        // zero-filled, so their dS would be multiplied by zero, but with a very negative lse their
        // probability exp2(0 - lse2) overflows the 16-bit dS to inf, and inf * 0 is NaN.
        const bool diagonal = kCausal && j * kTile + kTile - 1 > m0 + p.causal_off;
        const bool past_end = (j + 1) * kTile > p.Sk;
        if (diagonal || past_end) {
          const int col0 = j * kTile + wg * 64 + ch * 32;
          int last_e = 31;   // last visible of these 32
          if (diagonal) last_e = m0 + r + p.causal_off - col0;   // query row r sees a key column only if column <= r + causal_off
          if (past_end) last_e = min(last_e, p.Sk - 1 - col0);
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            if (e > last_e) pf[ch * 32 + e] = 0.f;
          }
        }
      }
      uint32_t keep[2] = {0xffffffffu, 0xffffffffu};   // dropout: bit e of keep[ch] <-> key column ch*32 + e of this half
      if constexpr (kDropout) {
        const int blk = (j * kTile + wg * 64) >> 4;
        const int bh = b * p.Hq + h;
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          keep[ch] = dropout_bits16(p.drop, bh, m0 + r, blk + 2 * ch) |
                     (dropout_bits16(p.drop, bh, m0 + r, blk + 2 * ch + 1) << 16);
        }
      }
      B200FA_WAIT(dp_full, j & 1, 0x910);
      tc_fence_after();
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        uint32_t d[32];
        tmem_ld32(tDP + ch * 32, d);
        tmem_wait_ld();
        const float* df = reinterpret_cast<const float*>(d);
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float g0 = df[2 * e], g1 = df[2 * e + 1];
          if constexpr (kDropout) {
            const uint32_t kb = keep[ch] >> (2 * e);
            g0 = (kb & 1u) ? g0 * p.drop.inv_keep : 0.f;
            g1 = (kb & 2u) ? g1 * p.drop.inv_keep : 0.f;
          }
          const float2 a = __fmul2_rn(make_float2(pf[ch * 32 + 2 * e], pf[ch * 32 + 2 * e + 1]), __fadd2_rn(make_float2(g0, g1), nd2));
          pk[e] = pack2<kBf16>(a.x, a.y);
        }
        tmem_st16(tS + ch * 16, pk);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(ds_full);
    }
    // ---- epilogue: dQ (this warpgroup's half of the head dimension)
    B200FA_WAIT(acc_full, 0, 0x920);
    tc_fence_after();
    {
      // The scaled 16-bit dQ tile is staged in the Q buffer (every MMA that read it has
      // completed) in the swizzled box layout and leaves through TMA stores: whole 128-byte
      // lines, rows past the end of the sequence clipped by the tensor map, and nothing for
      // the CTA to wait on but the read of shared memory.
      constexpr int kHalf = kD / 2;
      const uint32_t tacc = tmem_base + lane_off + kTmemDQ + wg * kHalf;
#pragma unroll
      for (int ch = 0; ch < kHalf / 32; ++ch) {
        uint32_t a[32];
        if (n_tiles > 0) {
          tmem_ld32(tacc + ch * 32, a);
          tmem_wait_ld();
        } else {
          // no key is visible from this query tile: nothing was accumulated, dQ is zero
#pragma unroll
          for (int e = 0; e < 32; ++e) a[e] = 0u;
        }
        const float* af = reinterpret_cast<const float*>(a);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint4 w;
          w.x = pack2<kBf16>(af[v * 8 + 0] * p.scale, af[v * 8 + 1] * p.scale);
          w.y = pack2<kBf16>(af[v * 8 + 2] * p.scale, af[v * 8 + 3] * p.scale);
          w.z = pack2<kBf16>(af[v * 8 + 4] * p.scale, af[v * 8 + 5] * p.scale);
          w.w = pack2<kBf16>(af[v * 8 + 6] * p.scale, af[v * 8 + 7] * p.scale);
          const int chunk = (wg * kHalf + ch * 32) / 8 + v;   // 16-byte chunk of the row
          *reinterpret_cast<uint4*>(sQ + (chunk >> 3) * kSubTileBytes + r * 128 + (((chunk & 7) ^ (r & 7)) << 4)) = w;
        }
      }
      fence_proxy_async_smem();
      mbar_arrive_warp(staged);
      if (threadIdx.x == 0) {
        B200FA_WAIT(staged, 0, 0x921);
#pragma unroll
        for (int cs = 0; cs < Cfg::kSub; ++cs) tma_store_4d(&mapDQ, sQ + cs * kSubTileBytes, cs * 64, m0, h, b);
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  } else if (warp == 8 || warp == 9) {
    // =========================== MMA issuers ===========================
    // Warp 8: dQ += dS_j K_j, then S of tile j+2 into the buffer dS_j just left.
    // Warp 9: dP of tile j+1.  Separate warps so that neither chain stalls behind the other's
    // operands (an issuing warp is blocked while the tensor pipe is full).
    {
      constexpr uint32_t idesc_s = umma_idesc(kBf16, false, false, 128, 128);   // S, dP
      constexpr uint32_t idesc_dq = umma_idesc(kBf16, false, true, 128, kD);    // dQ (A from TMEM, K MN-major)
      const uint32_t tDP = tmem_base + kTmemDP, tDQ = tmem_base + kTmemDQ;
      const UmmaDesc kQ = umma_desc_split(smem_u32(sQ), 16, 1024), kDO = umma_desc_split(smem_u32(sDO), 16, 1024),
                     kK = umma_desc_split(smem_u32(sK), 16, 1024), kV = umma_desc_split(smem_u32(sV), 16, 1024);
      const UmmaDesc mK = umma_desc_split(smem_u32(sK), kSubTileBytes, 1024);
      auto issue_kmajor = [&](uint32_t d_tmem, const UmmaDesc& a, const UmmaDesc& bd, uint32_t b_slot_lo) {
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk) {
          const uint32_t off = umma_off((kk >> 2) * kSubTileBytes + (kk & 3) * 32);
          umma_ss_elect(d_tmem, a.lo + off, a.hi, bd.lo + b_slot_lo + off, bd.hi, idesc_s, kk > 0);
        }
      };
      constexpr uint32_t kTileLo = umma_off(Cfg::kTileBytes);
      if (warp == 8) {
        // prologue: S_0, S_1
        if (n_tiles > 0) {
          B200FA_WAIT_WARP(q_full, 0, 0xa00);
          B200FA_WAIT_WARP(&k_full[0], 0, 0xa01);
          tc_fence_after();
          issue_kmajor(tmem_base + kTmemS, kQ, kK, 0);
          umma_commit_elect(&s_full[0]);
        }
        if (n_tiles > 1) {
          B200FA_WAIT_WARP(&k_full[1], 0, 0xa02);
          tc_fence_after();
          issue_kmajor(tmem_base + kTmemS + 128, kQ, kK, kTileLo);
          umma_commit_elect(&s_full[1]);
        }
        int kslot = 0;  // ring slot of K_j
        for (int j = 0; j < n_tiles; ++j) {
          const int buf = j & 1;
          const uint32_t tSj = tmem_base + kTmemS + buf * 128;
          const int k2slot = (kslot == 0) ? 2 : kslot - 1;   // slot of K_{j+2} = (j + 2) % 3
          // compute has written dS_j over S_j
          B200FA_WAIT_WARP(ds_full, j & 1, 0xa10);
          tc_fence_after();
          // dQ += dS_j K_j   (A = 16-bit dS in the S_j columns, B = K_j rows as the contraction index)
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            const uint32_t a_col = (kk < 4) ? kk * 8 : 64 + (kk - 4) * 8;
            const uint32_t b_lo = mK.lo + kslot * kTileLo + umma_off(kk * 2048);
            umma_ts_elect(tDQ, tSj + a_col, b_lo, mK.hi, idesc_dq, !(kk == 0 && j == 0));
          }
          umma_commit_elect(&k_empty[kslot]);
          if (j + 2 < n_tiles) {
            // S of tile j+2 re-uses this S buffer
            B200FA_WAIT_WARP(&k_full[k2slot], static_cast<uint32_t>(((j + 2) / 3) & 1), 0xa11);
            tc_fence_after();
            issue_kmajor(tSj, kQ, kK, k2slot * kTileLo);
            umma_commit_elect(&s_full[buf]);
          }
          if (++kslot == 3) kslot = 0;
        }
        umma_commit_elect(acc_full);
      } else if (n_tiles > 0) {
        // dP_0, then dP_{j+1} whenever the compute warps have consumed dP_j
        B200FA_WAIT_WARP(do_full, 0, 0xa20);
        B200FA_WAIT_WARP(&v_full[0], 0, 0xa03);
        tc_fence_after();
        issue_kmajor(tDP, kDO, kV, 0);
        umma_commit_elect(dp_full);
        umma_commit_elect(&v_empty[0]);
        for (int j = 0; j + 1 < n_tiles; ++j) {
          const int vslot = (j + 1) & 1;
          B200FA_WAIT_WARP(&v_full[vslot], ((j + 1) >> 1) & 1, 0xa12);
          B200FA_WAIT_WARP(ds_full, j & 1, 0xa13);
          tc_fence_after();
          issue_kmajor(tDP, kDO, kV, vslot * kTileLo);
          umma_commit_elect(dp_full);
          umma_commit_elect(&v_empty[vslot]);
        }
      }
    }
  } else if (warp == 10) {
    // =========================== TMA producer ===========================
    if (lane == 0) {
      // K_0 and V_0 went out before the block-wide synchronisation
      int kslot = 1;
      for (int j = 1; j < n_tiles; ++j) {
        if (j >= 3) { B200FA_WAIT(&k_empty[kslot], static_cast<uint32_t>((j / 3 - 1) & 1), 0xb00); }
        load_tile(&mapK, sK + kslot * Cfg::kTileBytes, &k_full[kslot], j * kTile, hk);
        const int vslot = j & 1;
        if (j >= 2) { B200FA_WAIT(&v_empty[vslot], ((j >> 1) - 1) & 1, 0xb01); }
        load_tile(&mapV, sV + vslot * Cfg::kTileBytes, &v_full[vslot], j * kTile, hk);
        if (++kslot == 3) kslot = 0;
      }
    }
  }

teardown:
  tc_fence_before();
  __syncthreads();
  settle_if_aborted(abort_flag);
  if (warp == 8) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (last_block) cudaGridDependencySynchronize();
}
#undef B200FA_WAIT
#undef B200FA_WAIT_WARP

// ------------------------------------------------------------------------------------------
// preprocess: dpsum = rowsum(dO * O), lse2 = lse * log2(e), per (b, h, row), padded to a
// multiple of 128 rows, both stored negated.  Rows in [S, Spad) get -lse2 = -inf and dpsum = 0 so their
// probabilities vanish.  One row per group of D/8 lanes; every lane moves 16 bytes of O and dO.
// HBM-bound, if enough loads are in flight: a thread issues those of kRows rows before it adds any
// of them up, and a block lies inside one (b, h), so that only its index is divided.
// B200: B4 Hq32 S4096 D128 bf16 70 -> 47 us (0.88 of the copy rate), B8 H12 S1024 D64 8.2 -> 6.2; with one row
// per thread and 64-bit divisions per row it was at 0.6.  Eight rows per thread: 57.
// ------------------------------------------------------------------------------------------
template <int kD>
struct PreCfg {
  static constexpr int kLanesPerRow = kD / 8, kRowsPerWarp = 32 / kLanesPerRow;
  static constexpr int kRows = 4;                                  // rows of a thread
  static constexpr int kBlockRows = 8 * kRowsPerWarp * kRows;      // 64 (D = 128) or 128: divides Spad
};

template <int kD, bool kBf16>
__global__ void __launch_bounds__(256) bwd_preprocess_kernel(const BwdParams p) {
  using Cfg = PreCfg<kD>;
  cudaTriggerProgrammaticLaunchCompletion();
  const int lane = threadIdx.x & 31;
  const int li = lane % Cfg::kLanesPerRow;
  const int per_head = p.Spad / Cfg::kBlockRows;
  const int bh = static_cast<int>(blockIdx.x) / per_head;
  const int b = bh / p.Hq, h = bh - b * p.Hq;
  const int s0 = (static_cast<int>(blockIdx.x) - bh * per_head) * Cfg::kBlockRows +
                 (threadIdx.x >> 5) * Cfg::kRowsPerWarp * Cfg::kRows + lane / Cfg::kLanesPerRow;
  const uint16_t* o = reinterpret_cast<const uint16_t*>(p.out.ptr) + static_cast<int64_t>(b) * p.out.sb +
                      static_cast<int64_t>(h) * p.out.sh + li * 8;
  const uint16_t* d = reinterpret_cast<const uint16_t*>(p.dout.ptr) + static_cast<int64_t>(b) * p.dout.sb +
                      static_cast<int64_t>(h) * p.dout.sh + li * 8;
  uint4 ov[Cfg::kRows], dv[Cfg::kRows];
  float lse[Cfg::kRows];
#pragma unroll
  for (int u = 0; u < Cfg::kRows; ++u) {
    const int s = s0 + u * Cfg::kRowsPerWarp;
    ov[u] = dv[u] = make_uint4(0, 0, 0, 0);
    lse[u] = -INFINITY;
    if (s < p.S) {
      ov[u] = *reinterpret_cast<const uint4*>(o + static_cast<int64_t>(s) * p.out.ss);
      dv[u] = *reinterpret_cast<const uint4*>(d + static_cast<int64_t>(s) * p.dout.ss);
      if (li == 0) lse[u] = p.lse[static_cast<int64_t>(bh) * p.S + s];
    }
  }
#pragma unroll
  for (int u = 0; u < Cfg::kRows; ++u) {
    const uint32_t ow[4] = {ov[u].x, ov[u].y, ov[u].z, ov[u].w};
    const uint32_t dw[4] = {dv[u].x, dv[u].y, dv[u].z, dv[u].w};
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float o0, o1, d0, d1;
      if constexpr (kBf16) {
        o0 = __uint_as_float(ow[i] << 16); o1 = __uint_as_float(ow[i] & 0xffff0000u);
        d0 = __uint_as_float(dw[i] << 16); d1 = __uint_as_float(dw[i] & 0xffff0000u);
      } else {
        asm("{.reg .b16 lo, hi; mov.b32 {lo, hi}, %2; cvt.f32.f16 %0, lo; cvt.f32.f16 %1, hi;}"
            : "=f"(o0), "=f"(o1) : "r"(ow[i]));
        asm("{.reg .b16 lo, hi; mov.b32 {lo, hi}, %2; cvt.f32.f16 %0, lo; cvt.f32.f16 %1, hi;}"
            : "=f"(d0), "=f"(d1) : "r"(dw[i]));
      }
      acc = fmaf(o0, d0, acc);
      acc = fmaf(o1, d1, acc);
    }
#pragma unroll
    for (int off = Cfg::kLanesPerRow / 2; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (li == 0) {
      const int s = s0 + u * Cfg::kRowsPerWarp;
      const int64_t at = static_cast<int64_t>(bh) * p.Spad + s;
      p.dpsum[at] = (s < p.S) ? -acc : 0.f;
      // a row that saw no key (lse = -inf) gets -lse2 = -inf like the padding rows: its probabilities vanish
      p.lse_log2[at] = lse[u] != -INFINITY ? lse[u] * -1.4426950408889634f : -INFINITY;
    }
  }
}

// cudaFuncSetAttribute for one kernel, once per device, safe against concurrent first calls.
// `once` and `result` belong to the kernel (the caller keeps them as statics of the function
// template that names it: kernels of the same signature must not share them).
template <typename Kernel>
cudaError_t allow_dynamic_smem(Kernel kern, int bytes, std::once_flag (&once)[64], cudaError_t (&result)[64]) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  std::call_once(once[dev], [&] {
    result[dev] = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  });
  return result[dev];
}

template <int kD, bool kBf16, bool kCausal, bool kDropout>
cudaError_t launch_one(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo,
                       const CUtensorMap& mdq, const CUtensorMap& mdk, const CUtensorMap& mdv, const BwdParams& p,
                       cudaStream_t stream) {
  using Cfg = BwdCfg<kD>;
  cudaError_t e = cudaSuccess;
  auto k1 = bwd_dkdv_kernel<kD, kBf16, kCausal, kDropout>;
  auto k2 = bwd_dq_kernel<kD, kBf16, kCausal, kDropout>;
  static std::once_flag once1[64], once2[64];
  static cudaError_t result1[64], result2[64];
  if ((e = allow_dynamic_smem(k1, Cfg::kSmemBytes, once1, result1)) != cudaSuccess) return e;
  if ((e = allow_dynamic_smem(k2, Cfg::kSmemBytes, once2, result2)) != cudaSuccess) return e;
  if (p.parts & 1) {
    const int64_t pre_blocks = static_cast<int64_t>(p.B) * p.Hq * (p.Spad / PreCfg<kD>::kBlockRows);
    bwd_preprocess_kernel<kD, kBf16><<<static_cast<unsigned>(pre_blocks), 256, 0, stream>>>(p);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  const int tiles = (p.S + kTile - 1) / kTile;        // query tiles: the dQ kernel's grid
  const int kv_tiles = (p.Sk + kTile - 1) / kTile;    // K/V tiles: the dK/dV kernel's grid
  if (p.parts & 2) {
    // (batch, kv head) pairs whose streamed Q / dO rows (both, all query heads of the pair)
    // add up to about 48 MiB share a scheduling group
    const int64_t pair_bytes = static_cast<int64_t>(p.Hq / p.Hkv) * p.S * p.D * 2 * 2;
    int64_t sched_group = (48ll << 20) / (pair_bytes > 0 ? pair_bytes : 1);
    const int64_t pairs = static_cast<int64_t>(p.B) * p.Hkv;
    if (sched_group < 1) sched_group = 1;
    if (sched_group > pairs) sched_group = pairs;
    e = launch_early(k1, dim3(static_cast<unsigned>(kv_tiles * pairs)), kDkdvThreads, Cfg::kSmemBytes, stream, (p.parts & 1) != 0,
                     mq, mk, mv, mdo, mdk, mdv, p, static_cast<int>(sched_group));
  }
  if (e == cudaSuccess && (p.parts & 4)) {
    // The dQ kernel does not need the dK/dV kernel's results, only the row statistics, and fills the SMs that the last
    // blocks of that one leave idle.  B200, us, whole backward with the dQ kernel on a side stream behind events / each
    // kernel launched to start early: B1 H8 S512 D128 bf16 causal 30 / 23.5, B16 H8 S1000x77 D64 fp16 55 / 48, B2 H16 S1024
    // D128 51.6 / 47.7, B4 Hq32 Hkv8 S4096 D128 1494 / 1485, B8 H16 S2048 D128 unmasked (one after the other) 815 / 806.
    e = launch_early(k2, dim3(tiles, p.Hq, p.B), kThreads, Cfg::kSmemBytes, stream, (p.parts & 2) != 0, mq, mk, mv, mdo, mdq, p);
  }
  return e;
}

template <int kD, bool kBf16>
cudaError_t launch_mask(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo,
                        const CUtensorMap& mdq, const CUtensorMap& mdk, const CUtensorMap& mdv, const BwdParams& p,
                        cudaStream_t stream) {
  const bool drop = p.drop.threshold != 0;
  if (p.causal) {
    return drop ? launch_one<kD, kBf16, true, true>(mq, mk, mv, mdo, mdq, mdk, mdv, p, stream)
                : launch_one<kD, kBf16, true, false>(mq, mk, mv, mdo, mdq, mdk, mdv, p, stream);
  }
  return drop ? launch_one<kD, kBf16, false, true>(mq, mk, mv, mdo, mdq, mdk, mdv, p, stream)
              : launch_one<kD, kBf16, false, false>(mq, mk, mv, mdo, mdq, mdk, mdv, p, stream);
}

}  // namespace

cudaError_t launch_bwd_sm100(const BwdParams& p, int dtype, cudaStream_t stream, int* launches) {
  const bool bf16 = (dtype == kBF16);
  CUtensorMap mq, mk, mv, mdo, mdq, mdk, mdv;
  if (!encode_map_16bit(&mq, p.q, p.B, p.Hq, p.S, p.D, kTile, bf16)) return cudaErrorInvalidValue;
  if (!encode_map_16bit(&mk, p.k, p.B, p.Hkv, p.Sk, p.D, kTile, bf16)) return cudaErrorInvalidValue;
  if (!encode_map_16bit(&mv, p.v, p.B, p.Hkv, p.Sk, p.D, kTile, bf16)) return cudaErrorInvalidValue;
  if (!encode_map_16bit(&mdo, p.dout, p.B, p.Hq, p.S, p.D, kTile, bf16)) return cudaErrorInvalidValue;
  if (!encode_map_16bit(&mdq, p.dq, p.B, p.Hq, p.S, p.D, kTile, bf16)) return cudaErrorInvalidValue;
  if (!encode_map_16bit(&mdk, p.dk, p.B, p.Hkv, p.Sk, p.D, kTile, bf16)) return cudaErrorInvalidValue;
  if (!encode_map_16bit(&mdv, p.dv, p.B, p.Hkv, p.Sk, p.D, kTile, bf16)) return cudaErrorInvalidValue;
  cudaError_t e;
  if (p.D == 128) {
    e = bf16 ? launch_mask<128, true>(mq, mk, mv, mdo, mdq, mdk, mdv, p, stream)
             : launch_mask<128, false>(mq, mk, mv, mdo, mdq, mdk, mdv, p, stream);
  } else {
    e = bf16 ? launch_mask<64, true>(mq, mk, mv, mdo, mdq, mdk, mdv, p, stream)
             : launch_mask<64, false>(mq, mk, mv, mdo, mdq, mdk, mdv, p, stream);
  }
  if (e == cudaSuccess && launches) *launches += (p.parts & 1) + ((p.parts >> 1) & 1) + ((p.parts >> 2) & 1);
  return e;
}

}  // namespace b200fa
