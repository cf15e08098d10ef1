// Flash attention backward for sm_100a, as two deterministic kernels (no float atomics):
//
//   flash_bwd_q   one CTA per 128 query rows of a (batch, head): for each key block recompute
//                 S = Q K^T and dP = dO V^T into TMEM, form dS = P * (dP - delta) * scale in registers,
//                 stage it as a bf16 operand and accumulate dQ += dS K in TMEM.
//   flash_bwd_kv  one CTA per 128 keys of a (batch, kv head): for every query head of the group and every
//                 query block that can see these keys recompute S^T = K Q^T and dP^T = V dO^T (so a
//                 thread owns a key row), form P^T and dS^T, and accumulate dV += P^T dO and
//                 dK += dS^T Q in TMEM. Grouped-query heads are summed inside the CTA.
//   flash_delta   delta[b,h,s] = sum_d dO * O.
//
// Warp roles match the forward kernel: warp 0 feeds shared memory with TMA, warp 1 issues tcgen05.mma,
// warps 2..9 do the element-wise work, two threads per tile row with 64 of the block's 128 columns each (the row
// statistics come from the forward pass, so the halves are independent). dS (dQ) and P^T (dV) go back to tensor memory as
// bf16 and are read there as the A operand of the product they enter; only dS^T is staged in shared memory. That leaves
// room for two or three stages of every streamed tile at head size 128 too, so loads, products and element-wise steps of
// neighbouring blocks overlap. With everything staged in shared memory there was one stage of each, and a block's load,
// scores, element-wise step and accumulation ran one after the other. Measured, 8192 positions, 32 heads on 8, size 128,
// causal: dQ 1330 -> 747 us, dK / dV 1884 -> 1299 us; then with packed fp32 arithmetic 709 and 1263 us, and with one
// barrier arrival per warp and the scores issued before dP 690 and 1069 us. 8 x 1024, 12 heads, size 64: 49 -> 43 and
// 84 -> 74 us in all. What bounds them now is the chain of an element-wise step (two warps per scheduler, 64 columns per
// thread); the tensor pipe is busy 35 to 50 % of the time.
// A tile in shared memory serves as a K-major operand for one product and as an MN-major operand for the other, so nothing
// is transposed.
//
// Reference counterparts: flash_tc_bwd_q_d{64,128}, flash_tc_bwd_kv_d{64,128}, flash_tc_delta
// (src/Idrak.Gpu/Cuda/PtxKernels.FlashTensorCore.cs) and attn_bwd_{d,kv,q}_f32 (PtxKernels.Rows.cs:1222-1750).
#include "flash_common.cuh"

namespace idrak {

constexpr float kLog2e = 1.4426950408889634f;

constexpr int kBwdThreads = 320;      // TMA warp, MMA warp, eight element-wise warps (two threads per tile row)
__device__ __forceinline__ void softmax_bar_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// Write 32 consecutive columns [c*32, c*32+32) of row r of a 128x128 bf16 K-major operand tile.
__device__ __forceinline__ void store_operand_chunk(uint8_t* tile, int r, int c, const float (&v)[32]) {
  uint8_t* atom = tile + (c >> 1) * 16384 + r * 128;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int chunk = ((c & 1) * 4 + g) ^ (r & 7);
    uint4 o;
    o.x = pack_bf16x2(v[g * 8 + 0], v[g * 8 + 1]);
    o.y = pack_bf16x2(v[g * 8 + 2], v[g * 8 + 3]);
    o.z = pack_bf16x2(v[g * 8 + 4], v[g * 8 + 5]);
    o.w = pack_bf16x2(v[g * 8 + 6], v[g * 8 + 7]);
    *reinterpret_cast<uint4*>(atom + chunk * 16) = o;
  }
}

// K-major operand tile [128 rows][D]: descriptor for k-step kk (16 columns)
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t base, int kk) {
  return make_smem_desc_sw128(base + (kk >> 2) * 16384 + (kk & 3) * 32, 16, 1024);
}
// The same tile read as an MN-major operand (N = D, contraction over its 128 rows): k-step kk = 16 rows
__device__ __forceinline__ uint64_t mnmajor_desc(uint32_t base, int kk) {
  return make_smem_desc_sw128(base + kk * 2048, 16384, 1024);
}

// ---------------------------------------------------------------------------
// delta
// ---------------------------------------------------------------------------
__global__ void flash_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dO,
                                   float* __restrict__ delta, int B, int S, int H, int D) {
  // D/8 lanes share one (b, s, h) row, each with one 128-bit load of O and of dO; a warp covers 256/D rows
  const int lanes_per_row = D >> 3;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long w = t / lanes_per_row;
  const int sub = int(t - w * lanes_per_row);
  const long long total = (long long)B * S * H;
  float acc = 0.f;
  if (w < total) {
    const uint4 a = *reinterpret_cast<const uint4*>(o + w * D + sub * 8);
    const uint4 g = *reinterpret_cast<const uint4*>(dO + w * D + sub * 8);
    float2 x, y;
    x = unpack_bf16x2(a.x); y = unpack_bf16x2(g.x); acc += x.x * y.x + x.y * y.y;
    x = unpack_bf16x2(a.y); y = unpack_bf16x2(g.y); acc += x.x * y.x + x.y * y.y;
    x = unpack_bf16x2(a.z); y = unpack_bf16x2(g.z); acc += x.x * y.x + x.y * y.y;
    x = unpack_bf16x2(a.w); y = unpack_bf16x2(g.w); acc += x.x * y.x + x.y * y.y;
  }
  for (int o2 = lanes_per_row >> 1; o2 > 0; o2 >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o2);
  if (w < total && sub == 0) {
    const int h = int(w % H);
    const long long bs = w / H;
    const int s = int(bs % S);
    const int b = int(bs / S);
    delta[((long long)b * H + h) * S + s] = acc;
  }
}

// ---------------------------------------------------------------------------
// dQ
// ---------------------------------------------------------------------------
template <int D>
struct BwdQSmem {
  static constexpr int kTile = 128 * D * 2;
  // A key tile is freed only by the dQ product of its block, a value tile already by the dP product: with three and two
  // stages neither load (about 1500 cycles from L2) sits on the path from one block to the next. dS stays in tensor memory,
  // which is what makes the room for them at head size 128 (one stage of each before: every load, product and element-wise
  // step of a block waited for the one before).
  static constexpr int kKStages = 3, kVStages = 2;
  static constexpr int kQ = 0;
  static constexpr int kDO = kQ + kTile;
  static constexpr int kK = kDO + kTile;
  static constexpr int kV = kK + kKStages * kTile;
  static constexpr int kBar = kV + kVStages * kTile;
  static constexpr int kTotal = kBar + 256 + 1024;
};

// Persistent, like the dK / dV kernel below: one CTA per SM walks (query block, head, batch) units, heaviest first; the
// next unit's Q and dO load while the current unit's last block is in its element-wise and dQ steps, and the write-out of
// dQ overlaps the next unit's first score products.
// Unit `round` of this CTA. The units are sorted heaviest first; the CTAs take them in rounds, forwards in even rounds and
// backwards in odd ones, so a CTA that drew a heavier unit than its neighbours in one round draws a lighter one in the
// next (the static counterpart of handing units out one by one).
__device__ __forceinline__ int snake_unit(int round, int units) {
  const int g = int(gridDim.x), c = int(blockIdx.x);
  const int u = round * g + ((round & 1) ? (g - 1 - c) : c);
  return u < units ? u : -1;
}
__device__ __forceinline__ int snake_rounds(int units) { return (units + int(gridDim.x) - 1) / int(gridDim.x); }

struct QUnit {
  int qb, head, batch, kv_head, q0, jlo, nkv;
};

template <bool MODES>
__device__ __forceinline__ QUnit q_unit(const FlashParams& p, int u, int off, int nqt) {
  QUnit t;
  const int per_qb = p.H * p.B;
  const int slot = u / per_qb;
  t.qb = p.causal ? (nqt - 1 - slot) : slot;      // later query blocks see more keys: they go first
  const int rem = u - slot * per_qb;
  t.head = rem % p.H;
  t.batch = rem / p.H;
  t.kv_head = t.head / (p.H / p.Hkv);
  t.q0 = t.qb * 128;
  int nkv_end = (p.Skv + 127) / 128;
  if (p.causal) nkv_end = min(nkv_end, (t.q0 + 127 + off) / 128 + 1);
  if (nkv_end < 0) nkv_end = 0;
  // key blocks wholly below what the tile's first row may see are skipped (window / packed-sequence bounds)
  const bool bounded = MODES && p.causal && (p.window > 0 || p.row_start != nullptr);
  t.jlo = bounded ? min(nkv_end, max(0, flash_row_lo(p, t.batch, min(t.q0, p.Sq - 1), off)) / 128) : 0;
  t.nkv = nkv_end - t.jlo;      // key block of iteration j is jlo + j
  return t;
}

template <int D, bool MODES>
__global__ void __launch_bounds__(kBwdThreads, 1)
flash_bwd_q_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                   const FlashParams p) {
  using L = BwdQSmem<D>;
  constexpr int KS = L::kKStages, VS = L::kVStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* qdo_full = bars + 0;
  uint64_t* k_full = bars + 1;      // [3]
  uint64_t* k_empty = bars + 4;     // [3]
  uint64_t* v_full = bars + 7;      // [2]
  uint64_t* v_empty = bars + 9;     // [2]
  uint64_t* sdp_full = bars + 11;
  uint64_t* ds_ready = bars + 12;   // [2]: one per dS buffer, as of P in the forward pass
  uint64_t* dq_done = bars + 14;    // [2]: one per dS buffer
  uint64_t* sdp_taken = bars + 16;  // the element-wise warps hold S and dP of the block in registers: TMEM may be rewritten
  uint64_t* qdo_free = bars + 17;   // the unit's last score products have read Q and dO: the next unit's may land
  uint64_t* dq_free = bars + 18;    // dQ of the unit sits in registers: the next unit may accumulate
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int off = p.Skv - p.Sq;
  const int nqt = (p.Sq + 127) / 128;
  const int units = nqt * p.H * p.B;
  const bool bounded = MODES && p.causal && (p.window > 0 || p.row_start != nullptr);

  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1);
    for (int s = 0; s < KS; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < VS; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    mbar_init(sdp_full, 1);
    mbar_init(&ds_ready[0], 8);
    mbar_init(&ds_ready[1], 8);
    mbar_init(&dq_done[0], 1);
    mbar_init(&dq_done[1], 1);
    mbar_init(sdp_taken, 8);
    mbar_init(qdo_free, 1);
    mbar_init(dq_free, 8);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  constexpr uint32_t kTmemCols = 512;   // S [0,128) | dP [128,256) | dS 2 x 64 [256,384) | dQ [384, 384+D)
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base, tmem_dP = tmem_base + 128, tmem_dS = tmem_base + 256, tmem_dQ = tmem_base + 384;

  // Every role walks the same units and counts alike: n = units with work so far, g = key blocks so far over all units.
  if (warp == 0) {
    if (lane == 0) {
      int n = 0, g = 0;
      bool ok = true;
      for (int round = 0; round < snake_rounds(units) && ok; ++round) {
        const int u = snake_unit(round, units);
        if (u < 0) continue;
        const QUnit t = q_unit<MODES>(p, u, off, nqt);
        if (t.nkv <= 0) continue;
        if (n > 0 && !mbar_wait(qdo_free, (n - 1) & 1, abort_flag, p.st, kTimeoutSmemEmpty, (3u << 16) | 14)) break;
        mbar_expect_tx(qdo_full, 2 * L::kTile);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          tma_load_4d(smem + L::kQ + c * 16384, &tmQ, qdo_full, c * 64, t.q0, t.head, t.batch);
          tma_load_4d(smem + L::kDO + c * 16384, &tmDO, qdo_full, c * 64, t.q0, t.head, t.batch);
        }
        for (int j = 0; j < t.nkv; ++j, ++g) {
          const int ks = g % KS, vs = g % VS;
          const int key0 = (t.jlo + j) * 128;
          if (!mbar_wait(&k_empty[ks], ((g / KS) & 1) ^ 1, abort_flag, p.st, kTimeoutSmemEmpty, (3u << 16) | ks)) { ok = false; break; }
          mbar_expect_tx(&k_full[ks], L::kTile);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(smem + L::kK + ks * L::kTile + c * 16384, &tmK, &k_full[ks], c * 64, key0, t.kv_head, t.batch);
          if (!mbar_wait(&v_empty[vs], ((g / VS) & 1) ^ 1, abort_flag, p.st, kTimeoutSmemEmpty, (3u << 16) | (4 + vs))) { ok = false; break; }
          mbar_expect_tx(&v_full[vs], L::kTile);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(smem + L::kV + vs * L::kTile + c * 16384, &tmV, &v_full[vs], c * 64, key0, t.kv_head, t.batch);
        }
        ++n;
      }
      if (*abort_flag) __nanosleep(50000);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_f16(128, 128, 0, 0, 1);
      constexpr uint32_t idesc_dq = make_idesc_f16(128, D, 0, 1, 1);
      const uint32_t sq = smem_u32(smem + L::kQ), sdo = smem_u32(smem + L::kDO);
      int n = 0, g0 = 0;
      bool ok = true;
      // S and dP of global block g; within a unit they are issued one block ahead, as soon as the element-wise warps
      // have taken the previous block's S and dP into registers
      auto issue_scores = [&](int g) -> bool {
        const int ks = g % KS, vs = g % VS;
        if (!mbar_wait(&k_full[ks], (g / KS) & 1, abort_flag, p.st, kTimeoutSmemFull, (3u << 16) | ks)) return false;
        if (!mbar_wait(&v_full[vs], (g / VS) & 1, abort_flag, p.st, kTimeoutSmemFull, (3u << 16) | (4 + vs))) return false;
        if (g > 0 && !mbar_wait(sdp_taken, (g - 1) & 1, abort_flag, p.st, kTimeoutTmemEmpty, (3u << 16) | 13)) return false;
        tc_fence_after();
        const uint32_t sk = smem_u32(smem + L::kK + ks * L::kTile), sv = smem_u32(smem + L::kV + vs * L::kTile);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          tc_mma_f16_ss(tmem_S, kmajor_desc(sq, kk), kmajor_desc(sk, kk), idesc_s, kk > 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          tc_mma_f16_ss(tmem_dP, kmajor_desc(sdo, kk), kmajor_desc(sv, kk), idesc_s, kk > 0 ? 1u : 0u);
        tc_commit(sdp_full);
        tc_commit(&v_empty[vs]);
        return true;
      };
      for (int round = 0; round < snake_rounds(units) && ok; ++round) {
        const int u = snake_unit(round, units);
        if (u < 0) continue;
        const QUnit t = q_unit<MODES>(p, u, off, nqt);
        if (t.nkv <= 0) continue;
        if (!mbar_wait(qdo_full, n & 1, abort_flag, p.st, kTimeoutSmemFull, (3u << 16) | 8)) break;
        ok = issue_scores(g0);
        if (ok && t.nkv == 1) tc_commit(qdo_free);
        for (int j = 0; j < t.nkv && ok; ++j) {
          const int g = g0 + j;
          const int ks = g % KS;
          if (j + 1 < t.nkv) {
            if (!issue_scores(g + 1)) { ok = false; break; }
            if (j + 2 == t.nkv) tc_commit(qdo_free);        // the unit's last score products are on their way
          }
          if (!mbar_wait(&ds_ready[g & 1], uint32_t(g >> 1) & 1u, abort_flag, p.st, kTimeoutGeneric, (3u << 16) | 9)) { ok = false; break; }
          if (j == 0 && n > 0) {
            // dQ of the previous unit must have been read out before this unit starts its own sum
            if (!mbar_wait(dq_free, (n - 1) & 1, abort_flag, p.st, kTimeoutTmemEmpty, (3u << 16) | 15)) { ok = false; break; }
          }
          tc_fence_after();
          const uint32_t sk = smem_u32(smem + L::kK + ks * L::kTile);
          const uint32_t ds_b = tmem_dS + (g & 1) * 64;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma_f16_ts(tmem_dQ, ds_b + kk * 8, mnmajor_desc(sk, kk), idesc_dq, (j > 0 || kk > 0) ? 1u : 0u);
          tc_commit(&k_empty[ks]);
          tc_commit(&dq_done[g & 1]);
        }
        g0 += t.nkv;
        ++n;
      }
    }
  } else {
    // Two threads per query row: warps 2..5 take key columns [0, 64) of a block, warps 6..9 columns [64, 128); the
    // row's statistics come from the forward pass, so the halves are independent.
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
    const bool capped = MODES && p.softcap > 0.f;
    const bool special = bounded || capped;
    const float cap_in = capped ? p.scale / p.softcap : 0.f;
    const float cap_l2 = p.softcap * kLog2e;
    constexpr int kOC = D / 2;               // each half writes D / 2 columns of the row
    int g0 = 0;
    bool ok = true;
    for (int round = 0; round < snake_rounds(units) && ok; ++round) {
      const int u = snake_unit(round, units);
      if (u < 0) continue;
      const QUnit t = q_unit<MODES>(p, u, off, nqt);
      const int row = t.q0 + r;
      __nv_bfloat16* drow = p.dQ + (size_t(t.batch) * p.Sq + row) * p.dq_row_stride + size_t(t.head) * D + half * kOC;
      if (t.nkv <= 0) {
        if (row < p.Sq)
          for (int i = 0; i < kOC; i += 8) *reinterpret_cast<uint4*>(drow + i) = make_uint4(0, 0, 0, 0);
        continue;
      }
      float lse2 = INFINITY, dlt = 0.f;
      if (row < p.Sq) {
        const size_t idx = (size_t(t.batch) * p.H + t.head) * p.Sq + row;
        const float l = p.lse[idx];
        lse2 = (l == -INFINITY) ? INFINITY : l * kLog2e;
        dlt = p.delta[idx];
      }
      const float dlt_s = dlt * p.scale;       // dS = P * (dP * scale - delta * scale)
      const int row_lo = bounded ? flash_row_lo(p, t.batch, row, off) : 0;
      for (int j = 0; j < t.nkv && ok; ++j) {
        const int g = g0 + j;
        if (!warp_wait(sdp_full, g & 1, abort_flag, p.st, kTimeoutTmemFull, (3u << 16) | 10)) { ok = false; break; }
        tc_fence_after();
        const int k0 = (t.jlo + j) * 128 + half * 64;          // first key of this thread's 64 columns
        int lim = p.Skv - k0;
        if (p.causal) lim = min(lim, row + off - k0 + 1);
        lim = max(0, min(64, lim));
        const int lo = max(0, min(64, row_lo - k0));           // keys below the row's window / sequence start
        // four loads in flight and one wait; once every thread holds its part the MMA warp may overwrite S and dP with
        // the next block's
        uint32_t s[2][32], dp[2][32];
        tmem_ld_32x32b_x32(tmem_S + lane_addr + half * 64, s[0]);
        tmem_ld_32x32b_x32(tmem_S + lane_addr + half * 64 + 32, s[1]);
        tmem_ld_32x32b_x32(tmem_dP + lane_addr + half * 64, dp[0]);
        tmem_ld_32x32b_x32(tmem_dP + lane_addr + half * 64 + 32, dp[1]);
        tmem_ld_wait();
        tc_fence_before();
        warp_arrive(sdp_taken);
        uint32_t packed[32];
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          float ds[32];
          if (!special) {
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const float2 x = fma2(as_float2(s[cc][i], s[cc][i + 1]), make_float2(p.scale_log2, p.scale_log2), make_float2(-lse2, -lse2));
              const float2 d = fma2(as_float2(dp[cc][i], dp[cc][i + 1]), make_float2(p.scale, p.scale), make_float2(-dlt_s, -dlt_s));
              const float2 v = mul2(make_float2(fast_exp2(x.x), fast_exp2(x.y)), d);
              ds[i] = v.x;
              ds[i + 1] = v.y;
            }
          } else {
            // lower key bound and / or soft-capped scores: u = cap * tanh(s * scale / cap), du/ds = scale * (1 - tanh^2)
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              float sc = __uint_as_float(s[cc][i]), gr = 1.f;
              if (capped) {
                const float th = tanh_fast(sc * cap_in);
                sc = th * cap_l2;
                gr -= th * th;
              } else {
                sc *= p.scale_log2;
              }
              const float pr = fast_exp2(sc - lse2);
              ds[i] = pr * (__uint_as_float(dp[cc][i]) * p.scale - dlt_s) * gr;
            }
          }
          if (lim < 64 || lo > 0) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (cc * 32 + i >= lim || cc * 32 + i < lo) ds[i] = 0.f;
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) packed[cc * 16 + i] = pack_bf16x2(ds[2 * i], ds[2 * i + 1]);
        }
        if (g >= 2) {
          // the dQ product that last read this dS buffer (block g - 2) must be complete
          if (!warp_wait(&dq_done[g & 1], uint32_t((g >> 1) - 1) & 1u, abort_flag, p.st, kTimeoutTmemFull, (3u << 16) | 11)) {
            ok = false;
            break;
          }
          tc_fence_after();
        }
        tmem_st_32x32b_x32(tmem_dS + (g & 1) * 64 + lane_addr + half * 32, packed);
        tmem_st_wait();
        tc_fence_before();
        warp_arrive(&ds_ready[g & 1]);
      }
      if (!ok) break;
      const int last = g0 + t.nkv - 1;
      if (!warp_wait(&dq_done[last & 1], uint32_t(last >> 1) & 1u, abort_flag, p.st, kTimeoutTmemFull, (3u << 16) | 12)) {
        ok = false;
        break;
      }
      tc_fence_after();
      // dQ leaves tensor memory first, so the next unit may start accumulating while the row is packed and stored
      uint32_t o[kOC];
#pragma unroll
      for (int c = 0; c < kOC / 32; ++c)
        tmem_ld_32x32b_x32(tmem_dQ + lane_addr + half * kOC + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&o[c * 32]));
      tmem_ld_wait();
      tc_fence_before();
      warp_arrive(dq_free);
      if (row < p.Sq) {
#pragma unroll
        for (int gq = 0; gq < kOC / 8; ++gq) {
          uint4 w;
          w.x = pack_bf16x2(__uint_as_float(o[gq * 8 + 0]), __uint_as_float(o[gq * 8 + 1]));
          w.y = pack_bf16x2(__uint_as_float(o[gq * 8 + 2]), __uint_as_float(o[gq * 8 + 3]));
          w.z = pack_bf16x2(__uint_as_float(o[gq * 8 + 4]), __uint_as_float(o[gq * 8 + 5]));
          w.w = pack_bf16x2(__uint_as_float(o[gq * 8 + 6]), __uint_as_float(o[gq * 8 + 7]));
          *reinterpret_cast<uint4*>(drow + gq * 8) = w;
        }
      }
      g0 += t.nkv;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------------------
// dK, dV
// ---------------------------------------------------------------------------
template <int D>
struct BwdKVSmem {
  static constexpr int kTile = 128 * D * 2;
  static constexpr int kStages = 2;                         // Q and dO: the next block's load during this one's products
  static constexpr int kK = 0;
  static constexpr int kV = kK + kTile;
  static constexpr int kQ = kV + kTile;
  static constexpr int kDO = kQ + kStages * kTile;
  // P^T is an operand in tensor memory; only dS^T is staged here, in two buffers at head size 64 and in the one that fits
  // beside two Q / dO stages at head size 128 (227 KB in all)
  static constexpr int kDSBufs = (D == 64) ? 2 : 1;
  static constexpr int kDST = kDO + kStages * kTile;
  static constexpr int kStat = kDST + kDSBufs * 32768;      // -lse * log2(e) [128], -delta * scale [128], lo[128]
  static constexpr int kBar = kStat + 1536;
  static constexpr int kTotal = kBar + 256 + 1024;
};

// Persistent: the grid is one CTA per SM and every CTA walks a list of (key block, kv head, batch) units, heaviest
// first. Barriers, tensor memory and the Q / dO ring are set up once; the next unit's K and V load while the last block of
// the current unit is still in its element-wise and accumulation steps, and the write-out of dK / dV overlaps the first
// score products of the next unit. With one launch of 1536 short CTAs the set-up, first-load and write-out latencies
// (about 12 k cycles per CTA) ran unhidden, a third of the time at 1024 tokens.
struct KvUnit {
  int kb, kv_head, batch, part, head0, k0, i_min, per_head, iters;
};

template <bool MODES>
__device__ __forceinline__ KvUnit kv_unit(const FlashParams& p, int u, int off, int nq) {
  KvUnit t;
  const int per_kb = p.Hkv * p.B * p.kv_parts;
  t.kb = u / per_kb;                         // ascending key block = most query blocks first under a causal mask
  int rem = u - t.kb * per_kb;
  t.part = rem % p.kv_parts;
  rem /= p.kv_parts;
  t.kv_head = rem % p.Hkv;
  t.batch = rem / p.Hkv;
  const int group = p.H / p.Hkv;
  const int heads = group / p.kv_parts;      // query heads of this unit
  t.head0 = t.kv_head * group + t.part * heads;
  t.k0 = t.kb * 128;
  t.i_min = p.causal ? max(0, (t.k0 - off) / 128) : 0;
  // query blocks past the last one that can see these keys are skipped too: a sliding window bounds them directly,
  // packed sequences by the first block whose first row already starts beyond this key block
  int i_end = nq;
  if (MODES && p.causal && (p.window > 0 || p.row_start != nullptr)) {
    if (p.window > 0) i_end = min(i_end, (t.k0 + 127 + p.window - 1 - off) / 128 + 1);
    if (p.row_start) {
      int i = t.i_min;
      while (i < i_end && p.row_start[size_t(t.batch) * p.Sq + min(i * 128, p.Sq - 1)] <= t.k0 + 127) ++i;
      i_end = i;
    }
    i_end = max(i_end, t.i_min);
  }
  t.per_head = max(0, i_end - t.i_min);
  t.iters = t.per_head * heads;
  return t;
}

template <int D, bool MODES>
__global__ void __launch_bounds__(kBwdThreads, 1)
flash_bwd_kv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                    const FlashParams p) {
  using L = BwdKVSmem<D>;
  constexpr int NS = L::kStages;
  constexpr int DB = L::kDSBufs;
  constexpr bool kAlias = D == 128;    // P^T lies over the scores it was made from (tensor memory is full)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* kv_full = bars + 0;
  uint64_t* qdo_full = bars + 1;    // [2]
  uint64_t* qdo_empty = bars + 3;   // [2]
  uint64_t* s_full = bars + 5;
  uint64_t* dp_full = bars + 6;
  uint64_t* s_taken = bars + 7;     // S^T / dP^T of the block are in registers: TMEM may be rewritten
  uint64_t* dp_taken = bars + 8;
  uint64_t* p_ready = bars + 9;     // P^T is in tensor memory
  uint64_t* ds_ready = bars + 10;   // [2]: dS^T is in shared memory, one per buffer
  uint64_t* dv_done = bars + 12;    // the dV product has read P^T
  uint64_t* dk_done = bars + 13;    // [2]: one per dS^T buffer
  uint64_t* kv_free = bars + 15;    // the unit's last score products have read K and V: the next unit's may land
  uint64_t* acc_free = bars + 16;   // dV and dK of the unit sit in registers: the next unit may accumulate
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* s_lse2 = reinterpret_cast<float*>(smem + L::kStat);
  float* s_delta = s_lse2 + 128;
  int* s_lo = reinterpret_cast<int*>(s_delta + 128);      // first key each query of the block may see

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int off = p.Skv - p.Sq;
  const int nq = (p.Sq + 127) / 128;
  const int units = ((p.Skv + 127) / 128) * p.Hkv * p.B * p.kv_parts;
  const bool bounded = MODES && p.causal && (p.window > 0 || p.row_start != nullptr);

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&qdo_full[s], 1);
      mbar_init(&qdo_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(s_taken, 8);
    mbar_init(dp_taken, 8);
    mbar_init(p_ready, 8);
    mbar_init(&ds_ready[0], 8);
    mbar_init(&ds_ready[1], 8);
    mbar_init(dv_done, 1);
    mbar_init(&dk_done[0], 1);
    mbar_init(&dk_done[1], 1);
    mbar_init(kv_free, 1);
    mbar_init(acc_free, 8);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  // S^T [0,128) | dP^T [128,256) | dV [256,256+D) | dK [256+D, 256+2D) | P^T: 64 more columns at D = 64; at D = 128 over
  // the scores, each half of the queries in the first 32 columns of its own half
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kPHalf = kAlias ? 64 : 32;      // columns from the first 64 queries' part of P^T to the second's
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_ST = tmem_base, tmem_dPT = tmem_base + 128, tmem_dV = tmem_base + 256,
                 tmem_dK = tmem_base + 256 + D, tmem_PT = kAlias ? tmem_base : tmem_base + 256 + 2 * D;

  // Every role walks the same units and counts the same things: n = units with work so far (parity of the per-unit
  // barriers), g = query blocks so far over all units (stage and parity of the per-block barriers).
  if (warp == 0) {
    if (lane == 0) {
      int n = 0, g = 0;
      bool ok = true;
      for (int round = 0; round < snake_rounds(units) && ok; ++round) {
        const int u = snake_unit(round, units);
        if (u < 0) continue;
        const KvUnit t = kv_unit<MODES>(p, u, off, nq);
        if (t.iters == 0) continue;
        // K and V of this unit: once the previous unit's last score products have read theirs
        if (n > 0 && !mbar_wait(kv_free, (n - 1) & 1, abort_flag, p.st, kTimeoutSmemEmpty, (4u << 16) | 14)) break;
        mbar_expect_tx(kv_full, 2 * L::kTile);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          tma_load_4d(smem + L::kK + c * 16384, &tmK, kv_full, c * 64, t.k0, t.kv_head, t.batch);
          tma_load_4d(smem + L::kV + c * 16384, &tmV, kv_full, c * 64, t.k0, t.kv_head, t.batch);
        }
        int head = t.head0, qi = t.i_min;
        for (int it = 0; it < t.iters; ++it, ++g) {
          const int st = g % NS;
          const uint32_t ph = (g / NS) & 1;
          if (!mbar_wait(&qdo_empty[st], ph ^ 1, abort_flag, p.st, kTimeoutSmemEmpty, (4u << 16) | st)) { ok = false; break; }
          mbar_expect_tx(&qdo_full[st], 2 * L::kTile);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) {
            tma_load_4d(smem + L::kQ + st * L::kTile + c * 16384, &tmQ, &qdo_full[st], c * 64, qi * 128, head, t.batch);
            tma_load_4d(smem + L::kDO + st * L::kTile + c * 16384, &tmDO, &qdo_full[st], c * 64, qi * 128, head, t.batch);
          }
          if (++qi == t.i_min + t.per_head) {
            qi = t.i_min;
            ++head;
          }
        }
        ++n;
      }
      if (*abort_flag) __nanosleep(50000);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_f16(128, 128, 0, 0, 1);
      constexpr uint32_t idesc_acc = make_idesc_f16(128, D, 0, 1, 1);
      const uint32_t sk = smem_u32(smem + L::kK), sv = smem_u32(smem + L::kV);
      const uint32_t sdst = smem_u32(smem + L::kDST);
      int n = 0, g0 = 0;
      bool ok = true;
      auto load_wait = [&](int g) -> bool {
        const int st = g % NS;
        return mbar_wait(&qdo_full[st], (g / NS) & 1, abort_flag, p.st, kTimeoutSmemFull, (4u << 16) | st);
      };
      // Scores of global block g, once their place is free: S^T of the block before was taken into registers or, where P^T
      // lies over it, the dV product that reads P^T is complete.
      auto issue_s = [&](int g) -> bool {
        if (!load_wait(g)) return false;
        if (g > 0 && !mbar_wait(kAlias ? dv_done : s_taken, (g - 1) & 1, abort_flag, p.st, kTimeoutTmemEmpty, (4u << 16) | 13))
          return false;
        tc_fence_after();
        const uint32_t sq = smem_u32(smem + L::kQ + (g % NS) * L::kTile);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          tc_mma_f16_ss(tmem_ST, kmajor_desc(sk, kk), kmajor_desc(sq, kk), idesc_s, kk > 0 ? 1u : 0u);
        tc_commit(s_full);
        return true;
      };
      auto issue_dp = [&](int g) -> bool {
        if (!load_wait(g)) return false;
        if (g > 0 && !mbar_wait(dp_taken, (g - 1) & 1, abort_flag, p.st, kTimeoutTmemEmpty, (4u << 16) | 16)) return false;
        tc_fence_after();
        const uint32_t sdo = smem_u32(smem + L::kDO + (g % NS) * L::kTile);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          tc_mma_f16_ss(tmem_dPT, kmajor_desc(sv, kk), kmajor_desc(sdo, kk), idesc_s, kk > 0 ? 1u : 0u);
        tc_commit(dp_full);
        return true;
      };
      for (int round = 0; round < snake_rounds(units) && ok; ++round) {
        const int u = snake_unit(round, units);
        if (u < 0) continue;
        const KvUnit t = kv_unit<MODES>(p, u, off, nq);
        if (t.iters == 0) continue;
        if (!mbar_wait(kv_full, n & 1, abort_flag, p.st, kTimeoutSmemFull, (4u << 16) | 8)) break;
        ok = issue_s(g0) && issue_dp(g0);
        if (ok && t.iters == 1) tc_commit(kv_free);
        for (int it = 0; it < t.iters && ok; ++it) {
          const int g = g0 + it;
          const int st = g % NS;
          const bool more = it + 1 < t.iters;
          // The next block's scores and dP go out between this block's two accumulations, so the element-wise warps find
          // them when they are done with this block: the scores first, which their next step starts from (with a place of
          // their own even before dV).
          if (more && !kAlias && !issue_s(g + 1)) { ok = false; break; }
          if (!mbar_wait(p_ready, g & 1, abort_flag, p.st, kTimeoutGeneric, (4u << 16) | 9)) { ok = false; break; }
          if (it == 0 && n > 0) {
            // dV and dK of the previous unit must have been read out before this unit starts its own sums
            if (!mbar_wait(acc_free, (n - 1) & 1, abort_flag, p.st, kTimeoutTmemEmpty, (4u << 16) | 15)) { ok = false; break; }
          }
          tc_fence_after();
          const uint32_t sq = smem_u32(smem + L::kQ + st * L::kTile), sdo = smem_u32(smem + L::kDO + st * L::kTile);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma_f16_ts(tmem_dV, tmem_PT + (kk >> 2) * kPHalf + (kk & 3) * 8, mnmajor_desc(sdo, kk), idesc_acc,
                          (it > 0 || kk > 0) ? 1u : 0u);
          tc_commit(dv_done);
          if (more && kAlias && !issue_s(g + 1)) { ok = false; break; }
          if (more && !issue_dp(g + 1)) { ok = false; break; }
          if (it + 2 == t.iters) tc_commit(kv_free);               // the unit's last score products are on their way
          if (!mbar_wait(&ds_ready[g % DB], uint32_t(g / DB) & 1u, abort_flag, p.st, kTimeoutGeneric, (4u << 16) | 17)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sdst_b = sdst + (g % DB) * 32768;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma_f16_ss(tmem_dK, kmajor_desc(sdst_b, kk), mnmajor_desc(sq, kk), idesc_acc, (it > 0 || kk > 0) ? 1u : 0u);
          tc_commit(&qdo_empty[st]);
          tc_commit(&dk_done[g % DB]);
        }
        g0 += t.iters;
        ++n;
      }
    }
  } else {
    // Two threads per key row: warps 2..5 take query columns [0, 64) of the block, warps 6..9 columns [64, 128). The
    // columns are independent here (the row statistics come from the forward pass), so the halves never talk.
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;       // key row within the block
    const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
    bool ok = true;
    const bool capped = MODES && p.softcap > 0.f;
    const float cap_in = capped ? p.scale / p.softcap : 0.f;
    const float cap_l2 = p.softcap * kLog2e;
    int n = 0, g0 = 0;
    // A thread whose wait gave up keeps walking units and blocks without touching tensor memory: the block-wide barrier
    // of the element-wise warps has no time limit of its own, so nobody may leave early.
    for (int round = 0; round < snake_rounds(units); ++round) {
      const int u = snake_unit(round, units);
      if (u < 0) continue;
      const KvUnit t = kv_unit<MODES>(p, u, off, nq);
      const int key = t.k0 + r;
      if (t.iters > 0) {
        // lse and delta of one row of query block qi, as they are in memory: they are converted only where they are staged
        auto load_stats = [&](int head, int qi, float& l, float& dl, int& lo) {
          const int qr = qi * 128 + r;
          l = -INFINITY;
          dl = 0.f;
          if (qr < p.Sq) {
            const size_t idx = (size_t(t.batch) * p.H + head) * p.Sq + qr;
            l = p.lse[idx];
            dl = p.delta[idx];
          }
          lo = bounded ? flash_row_lo(p, t.batch, qr, off) : 0;
        };
        // both negated: the addends of the fused multiply-adds below
        auto staged_lse = [](float l) { return (l == -INFINITY) ? -INFINITY : -(l * kLog2e); };
        int head = t.head0, qi = t.i_min;             // of the current block, counted along
        // the previous unit's last block ended with a barrier after its statistics were last read
        if (half == 0) {
          float l, dl;
          int lo;
          load_stats(head, qi, l, dl, lo);
          s_lse2[r] = staged_lse(l);
          s_lo[r] = lo;
          s_delta[r] = -(dl * p.scale);
        }
        softmax_bar_sync();
        for (int it = 0; it < t.iters; ++it) {
          const int g = g0 + it;
          const int qrow0 = qi * 128;
          if (++qi == t.i_min + t.per_head) {
            qi = t.i_min;
            ++head;
          }
          // The statistics of the next query block are fetched now. Its lse replaces this block's once the probabilities
          // are formed, its delta once dS is: each is written after one of the block's two barriers and read after the
          // other, so neither barrier stands alone in the chain.
          float n_l = -INFINITY, n_dl = 0.f;
          int n_lo = 0;
          const bool fetch = half == 0 && it + 1 < t.iters;
          if (fetch) load_stats(head, qi, n_l, n_dl, n_lo);
          if (ok && !warp_wait(s_full, g & 1, abort_flag, p.st, kTimeoutTmemFull, (4u << 16) | 10)) ok = false;
          tc_fence_after();
          // query q (column) sees this key iff key <= q + off  <=>  q >= key - off
          const int first_q = p.causal ? (key - off - qrow0) : 0;    // columns below this are masked
          const bool diagonal = p.causal && t.k0 + 127 - off > qrow0;
          float pr[2][32], gr[MODES ? 2 : 1][MODES ? 32 : 1];
          {
            uint32_t s[2][32], packed[32];
            if (ok) {
              tmem_ld_32x32b_x32(tmem_ST + lane_addr + half * 64, s[0]);
              tmem_ld_32x32b_x32(tmem_ST + lane_addr + half * 64 + 32, s[1]);
              tmem_ld_wait();
              tc_fence_before();
              if (!kAlias) warp_arrive(s_taken);
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) s[0][i] = s[1][i] = 0u;
            }
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
              const int c0 = half * 64 + cc * 32;
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                const float4 l4 = *reinterpret_cast<const float4*>(&s_lse2[c0 + i]);
                const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                  const float2 l2 = make_float2(l[e], l[e + 1]);
                  float2 x;
                  if (MODES && capped) {
                    // u = cap * tanh(s * scale / cap), du/ds = scale * (1 - tanh^2)
                    const float t0 = tanh_fast(__uint_as_float(s[cc][i + e]) * cap_in), t1 = tanh_fast(__uint_as_float(s[cc][i + e + 1]) * cap_in);
                    x = fma2(make_float2(t0, t1), make_float2(cap_l2, cap_l2), l2);
                    gr[MODES ? cc : 0][MODES ? i + e : 0] = 1.f - t0 * t0;
                    gr[MODES ? cc : 0][MODES ? i + e + 1 : 0] = 1.f - t1 * t1;
                  } else {
                    x = fma2(as_float2(s[cc][i + e], s[cc][i + e + 1]), make_float2(p.scale_log2, p.scale_log2), l2);
                  }
                  pr[cc][i + e] = fast_exp2(x.x);
                  pr[cc][i + e + 1] = fast_exp2(x.y);
                }
              }
              if (diagonal) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (c0 + i < first_q) pr[cc][i] = 0.f;
              }
              if (bounded) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (key < s_lo[c0 + i]) pr[cc][i] = 0.f;
              }
#pragma unroll
              for (int i = 0; i < 16; ++i) packed[cc * 16 + i] = pack_bf16x2(pr[cc][2 * i], pr[cc][2 * i + 1]);
            }
            if (!kAlias && ok && g > 0) {
              // the dV product of the block before has read P^T (over the scores: they came after it)
              if (!warp_wait(dv_done, (g - 1) & 1, abort_flag, p.st, kTimeoutTmemFull, (4u << 16) | 18)) ok = false;
              tc_fence_after();
            }
            if (ok) {
              tmem_st_32x32b_x32(tmem_PT + lane_addr + half * kPHalf, packed);
              tmem_st_wait();
              tc_fence_before();
              warp_arrive(p_ready);
            }
          }
          softmax_bar_sync();    // this block's lse is no longer read; its delta is visible
          if (fetch) {
            s_lse2[r] = staged_lse(n_l);
            s_lo[r] = n_lo;
          }
          if (ok && !warp_wait(dp_full, g & 1, abort_flag, p.st, kTimeoutTmemFull, (4u << 16) | 19)) ok = false;
          tc_fence_after();
          uint8_t* sDST = smem + L::kDST + (g % DB) * 32768;
          if (ok && g >= DB) {
            // the dK product that last read this dS^T buffer (block g - DB) must be complete
            if (!warp_wait(&dk_done[g % DB], (uint32_t(g / DB) - 1u) & 1u, abort_flag, p.st, kTimeoutTmemFull, (4u << 16) | 11)) ok = false;
          }
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            const int c0 = half * 64 + cc * 32;
            uint32_t dp[32];                       // 32 at a time: beside the 64 probabilities they stay in registers
            if (ok) {
              tmem_ld_32x32b_x32(tmem_dPT + lane_addr + c0, dp);
              tmem_ld_wait();
              if (cc == 1) {
                tc_fence_before();
                warp_arrive(dp_taken);
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) dp[i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const float4 d4 = *reinterpret_cast<const float4*>(&s_delta[c0 + i]);
              const float d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
              for (int e = 0; e < 4; e += 2) {
                float2 v = fma2(as_float2(dp[i + e], dp[i + e + 1]), make_float2(p.scale, p.scale), make_float2(d[e], d[e + 1]));
                v = mul2(make_float2(pr[cc][i + e], pr[cc][i + e + 1]), v);
                if (MODES && capped) v = mul2(v, make_float2(gr[MODES ? cc : 0][MODES ? i + e : 0], gr[MODES ? cc : 0][MODES ? i + e + 1 : 0]));
                pr[cc][i + e] = v.x;
                pr[cc][i + e + 1] = v.y;
              }
            }
            if (ok) store_operand_chunk(sDST, r, half * 2 + cc, pr[cc]);
          }
          if (ok) {
            fence_proxy_async_smem();
            tc_fence_before();
            __syncwarp();
            warp_arrive(&ds_ready[g % DB]);
          }
          softmax_bar_sync();    // this block's delta is no longer read; the next block's lse is visible
          if (fetch) s_delta[r] = -(n_dl * p.scale);
        }
        if (ok) {
          const int last = g0 + t.iters - 1;
          if (!warp_wait(&dk_done[last % DB], uint32_t(last / DB) & 1u, abort_flag, p.st, kTimeoutTmemFull, (4u << 16) | 12))
            ok = false;
        }
        tc_fence_after();
      }
      // write-out: the first half of the threads takes dV, the second dK; the sums leave tensor memory first so that the
      // next unit may start accumulating while the rows are packed and stored
      uint32_t o[D];
      if (t.iters > 0 && ok) {
        const uint32_t acc = half ? tmem_dK : tmem_dV;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) tmem_ld_32x32b_x32(acc + lane_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&o[c * 32]));
        tmem_ld_wait();
        tc_fence_before();
        warp_arrive(acc_free);
      } else {
#pragma unroll
        for (int i = 0; i < D; ++i) o[i] = 0u;
      }
      if ((ok || t.iters == 0) && key < p.Skv && p.kv_parts > 1) {
        float* row = p.kv_partial + ((((size_t(t.part) * 2 + half) * p.B + t.batch) * p.Skv + key) * p.Hkv + t.kv_head) * D;
#pragma unroll
        for (int i = 0; i < D / 4; ++i) *reinterpret_cast<uint4*>(row + i * 4) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
      } else if ((ok || t.iters == 0) && key < p.Skv) {
        __nv_bfloat16* drow = (half ? p.dK + (size_t(t.batch) * p.Skv + key) * p.dk_row_stride
                                    : p.dV + (size_t(t.batch) * p.Skv + key) * p.dv_row_stride) + size_t(t.kv_head) * D;
#pragma unroll
        for (int gq = 0; gq < D / 8; ++gq) {
          uint4 w;
          w.x = pack_bf16x2(__uint_as_float(o[gq * 8 + 0]), __uint_as_float(o[gq * 8 + 1]));
          w.y = pack_bf16x2(__uint_as_float(o[gq * 8 + 2]), __uint_as_float(o[gq * 8 + 3]));
          w.z = pack_bf16x2(__uint_as_float(o[gq * 8 + 4]), __uint_as_float(o[gq * 8 + 5]));
          w.w = pack_bf16x2(__uint_as_float(o[gq * 8 + 6]), __uint_as_float(o[gq * 8 + 7]));
          *reinterpret_cast<uint4*>(drow + gq * 8) = w;
        }
      }
      if (t.iters > 0) {
        g0 += t.iters;
        ++n;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Sums the parts of dV and dK in part order: one thread per eight columns of a (batch, key, kv head) row.
__global__ void __launch_bounds__(256) flash_kv_parts_kernel(const FlashParams p, int D) {
  const int per_row = D / 8;
  const long long rows = (long long)p.B * p.Skv * p.Hkv, n = rows * per_row;
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (i >= n) return;
  const bool is_k = blockIdx.y == 1;
  const size_t plane = size_t(rows) * D;
  float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int part = 0; part < p.kv_parts; ++part) {
    const float4* v = reinterpret_cast<const float4*>(p.kv_partial + (size_t(part) * 2 + is_k) * plane + size_t(i) * 8);
    const float4 x = v[0], y = v[1];
    a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w;
    a[4] += y.x; a[5] += y.y; a[6] += y.z; a[7] += y.w;
  }
  const long long row = i / per_row;
  const int head = int(row % p.Hkv);
  const long long pos = row / p.Hkv;          // batch * Skv + key
  __nv_bfloat16* dst = (is_k ? p.dK + pos * p.dk_row_stride : p.dV + pos * p.dv_row_stride) + size_t(head) * D + (i - row * per_row) * 8;
  *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]), pack_bf16x2(a[4], a[5]), pack_bf16x2(a[6], a[7]));
}

// Query blocks that key block kb meets, as kv_unit walks them.
static int kv_seen(int kb, int nq, int off, int causal, int window) {
  const int first = causal ? max(0, (kb * 128 - off) / 128) : 0;
  int last = nq;
  if (causal && window > 0) last = min(last, (kb * 128 + 127 + window - 1 - off) / 128 + 1);
  return max(0, last - first);
}

// Into how many units the query heads of a key head are dealt. One unit walks every query head of its key block, so with
// grouped heads there are few units and the first key block's, which under a causal mask every query block sees, is longer
// than a CTA's fair share: 3 x 999 tokens with 16 heads on 4 has 96 units of up to 32 blocks for 148 SMs, against 12 blocks
// a SM if they were even. Measured, causal, size 64: 2 x 2048 tokens, 16 heads on 4: 142 -> 78 + 4 us for the sum; with 8192
// tokens the units are even enough and stay whole.
//
// The most parts worth a look: the smallest divisor of the group that brings the longest unit to a quarter over the fair share.
static int kv_parts_bound(int B, int H, int Hkv, int Sq, int Skv, int causal) {
  const int group = H / Hkv, nq = (Sq + 127) / 128, nkb = (Skv + 127) / 128, off = Skv - Sq;
  long long blocks = 0;
  int longest = 0;
  for (int kb = 0; kb < nkb; ++kb) {
    const int seen = kv_seen(kb, nq, off, causal, 0);
    blocks += seen;
    longest = max(longest, seen);
  }
  if (longest * group < 4) return 1;
  const double share = double(blocks) * H * B / sm_count();
  int parts = 1;
  while (parts < group && double(longest) * (group / parts) > 1.25 * max(share, 1.0)) {
    do ++parts; while (group % parts);
  }
  return parts;
}
// Of the divisors up to that, the one with the least estimated time: 2.1 us for each block of the busiest CTA as the units are
// handed out and, for more than one part, 0.4 us per MB of fp32 sums written and read again and 4.5 us for the launch that adds
// them up. Fitted to 140 shapes of 130 to 8192 tokens, head sizes 64 and 128, with and without windows: the choices come within
// 0.2 % of the best parts on average, and are never more than 4 % slower than whole units (the bound alone: up to 48 %).
// Measured, us, dealt / whole: 8 x 130 tokens, 32 heads on 8, size 128: 71 / 62, 4 x 256 queries on 700 keys, 8 on 4: 62 / 44, a
// window of 256 over 2048, 32 on 8: 130 / 110 (whole by the estimate); 2048 tokens, 16 on 4: 114 / 202, with the window 79 / 85.
// Sequences packed into a row make units shorter by what only the device knows: dealt only where the estimate for one sequence
// is a third of the whole one, from where on nothing measured slower. Eight sequences in 2048 tokens, 32 on 8, size 128:
// 108 / 87, in 8192, 8 on 1: 198 / 271.
static int kv_parts_of(int B, int H, int Hkv, int Sq, int Skv, int D, int causal, int window, bool packed) {
  const int bound = kv_parts_bound(B, H, Hkv, Sq, Skv, causal);
  if (bound == 1) return 1;
  const int group = H / Hkv, nq = (Sq + 127) / 128, nkb = (Skv + 127) / 128, off = Skv - Sq, sms = sm_count();
  int best = 1;
  double best_us = 0.0, whole_us = 0.0;
  for (int parts = 1; parts <= bound; ++parts) {
    if (group % parts) continue;
    const int per_kb = Hkv * B * parts;
    const long long units = (long long)nkb * per_kb;
    const int ctas = int(units < sms ? units : sms);
    long long busiest = 0;
    for (int c = 0; c < ctas; ++c) {                                       // snake_unit
      long long mine = 0;
      for (long long round = 0; round * ctas < units; ++round) {
        const long long u = round * ctas + ((round & 1) ? (ctas - 1 - c) : c);
        if (u < units) mine += kv_seen(int(u / per_kb), nq, off, causal, window);
      }
      busiest = max(busiest, mine);
    }
    double us = double(busiest) * (group / parts) * 2.1;
    if (parts == 1) whole_us = us;
    else us += 4.5 + 0.4e-6 * 8.0 * parts * B * Skv * Hkv * D;
    if (parts == 1 || us < best_us) {
      best = parts;
      best_us = us;
    }
  }
  return packed && 3.0 * best_us > whole_us ? 1 : best;
}

template <int D, bool MODES>
static int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                      const FlashParams& p, cudaStream_t stream) {
  auto kq = flash_bwd_q_kernel<D, MODES>;
  auto kkv = flash_bwd_kv_kernel<D, MODES>;
  static DeviceOnce configured;
  if (int e = configured.run([&] {
        cudaError_t e1 = cudaFuncSetAttribute(kq, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdQSmem<D>::kTotal);
        if (e1 != cudaSuccess) return int(e1);
        return int(cudaFuncSetAttribute(kkv, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdKVSmem<D>::kTotal));
      }))
    return e;
  const int q_units = ((p.Sq + 127) / 128) * p.H * p.B;
  kq<<<min(q_units, sm_count()), kBwdThreads, BwdQSmem<D>::kTotal, stream>>>(tq, tk, tv, tdo, p);
  note_launches(1);
  int rc = int(cudaGetLastError());
  if (rc) return rc;
  const int kv_units = ((p.Skv + 127) / 128) * p.Hkv * p.B * p.kv_parts;
  kkv<<<min(kv_units, sm_count()), kBwdThreads, BwdKVSmem<D>::kTotal, stream>>>(tq, tk, tv, tdo, p);
  note_launches(1);
  rc = int(cudaGetLastError());
  if (rc || p.kv_parts == 1) return rc;
  const long long vecs = (long long)p.B * p.Skv * p.Hkv * (D / 8);
  flash_kv_parts_kernel<<<dim3(unsigned((vecs + 255) / 256), 2), 256, 0, stream>>>(p, D);
  note_launches(1);
  return int(cudaGetLastError());
}

}  // namespace idrak

using namespace idrak;

// fp32 elements of workspace a backward call of these sizes needs (0: none); packed: with row_start. The form without a window
// is enough for any.
IDRAK_API long long idrak_flash_bwd_workspace_ex(int B, int H, int Hkv, int Sq, int Skv, int D, int causal, int window, int packed) {
  if (B <= 0 || Hkv <= 0 || H <= 0 || H % Hkv) return 0;
  const int parts = kv_parts_of(B, H, Hkv, Sq, Skv, D, causal, window, packed != 0);
  return parts > 1 ? 2LL * parts * B * Skv * Hkv * D : 0;
}
IDRAK_API long long idrak_flash_bwd_workspace(int B, int H, int Hkv, int Sq, int Skv, int D, int causal) {
  if (B <= 0 || Hkv <= 0 || H <= 0 || H % Hkv) return 0;
  const int parts = kv_parts_bound(B, H, Hkv, Sq, Skv, causal);
  return parts > 1 ? 2LL * parts * B * Skv * Hkv * D : 0;
}

// out / dout: contiguous [B, Sq, H, D]; lse, delta [B,H,Sq]. dq / dk / dv rows hold heads packed [heads, D] with
// the given row strides in elements (0 = contiguous), so they may be slices of one fused d(QKV) buffer;
// their batch stride is rows * row stride.
// window > 0 and row_start (one int per query row, [B, Sq]) restrict the keys a query sees exactly as in the forward
// entry point; both need `causal`. `softcap` > 0 differentiates through the tanh cap of the forward.
// workspace: idrak_flash_bwd_workspace_ex fp32 elements on a 16-byte boundary, or null (the heads of a group then stay together).
IDRAK_API int idrak_flash_bwd_ex(const void* q, const void* k, const void* v, const void* out, const void* dout,
                                 const float* lse, float* delta, void* dq, void* dk, void* dv, int B, int H, int Hkv,
                                 int Sq, int Skv, int D, long long q_row_stride, long long k_row_stride,
                                 long long v_row_stride, long long q_batch_stride, long long k_batch_stride,
                                 long long v_batch_stride, long long dq_row_stride, long long dk_row_stride,
                                 long long dv_row_stride, float scale, int causal, int window, const int* row_start,
                                 float softcap, float* workspace, void* stream_) {
  if (D != 64 && D != 128) return -2;
  if (H % Hkv) return -3;
  if ((window > 0 || row_start) && !causal) return -4;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  {
    const long long rows = (long long)B * Sq * H;
    const int threads = 256;
    const long long blocks = (rows * (D / 8) + threads - 1) / threads;
    flash_delta_kernel<<<unsigned(blocks), threads, 0, stream>>>(static_cast<const __nv_bfloat16*>(out),
                                                                 static_cast<const __nv_bfloat16*>(dout), delta, B,
                                                                 Sq, H, D);
    note_launches(1);
    int rc = int(cudaGetLastError());
    if (rc) return rc;
  }
  FlashParams p;
  p.kv_parts = workspace ? kv_parts_of(B, H, Hkv, Sq, Skv, D, causal, window, row_start != nullptr) : 1;
  p.kv_partial = workspace;
  p.O = nullptr;
  p.o_row_stride = 0;
  p.lse = const_cast<float*>(lse);
  p.delta = delta;
  p.B = B; p.H = H; p.Hkv = Hkv; p.Sq = Sq; p.Skv = Skv;
  p.scale = scale;
  p.scale_log2 = scale * kLog2e;
  p.causal = causal;
  p.window = window > 0 ? window : 0;
  p.row_start = row_start;
  p.softcap = softcap > 0.f ? softcap : 0.f;
  p.st = status_device_ptr();
  p.dQ = static_cast<__nv_bfloat16*>(dq);
  p.dK = static_cast<__nv_bfloat16*>(dk);
  p.dV = static_cast<__nv_bfloat16*>(dv);
  p.dq_row_stride = dq_row_stride > 0 ? dq_row_stride : (long long)H * D;
  p.dk_row_stride = dk_row_stride > 0 ? dk_row_stride : (long long)Hkv * D;
  p.dv_row_stride = dv_row_stride > 0 ? dv_row_stride : (long long)Hkv * D;
  CUtensorMap tq, tk, tv, tdo;
  if (make_head_map(&tq, q, D, Sq, H, B, q_row_stride, q_batch_stride)) return -10;
  if (make_head_map(&tk, k, D, Skv, Hkv, B, k_row_stride, k_batch_stride)) return -11;
  if (make_head_map(&tv, v, D, Skv, Hkv, B, v_row_stride, v_batch_stride)) return -12;
  if (make_head_map(&tdo, dout, D, Sq, H, B, (long long)H * D, (long long)Sq * H * D)) return -13;
  if (p.window > 0 || p.row_start || p.softcap > 0.f)
    return D == 64 ? launch_bwd<64, true>(tq, tk, tv, tdo, p, stream) : launch_bwd<128, true>(tq, tk, tv, tdo, p, stream);
  return D == 64 ? launch_bwd<64, false>(tq, tk, tv, tdo, p, stream) : launch_bwd<128, false>(tq, tk, tv, tdo, p, stream);
}

IDRAK_API int idrak_flash_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout,
                              const float* lse, float* delta, void* dq, void* dk, void* dv, int B, int H, int Hkv,
                              int Sq, int Skv, int D, long long q_row_stride, long long k_row_stride,
                              long long v_row_stride, long long q_batch_stride, long long k_batch_stride,
                              long long v_batch_stride, long long dq_row_stride, long long dk_row_stride,
                              long long dv_row_stride, float scale, int causal, void* stream_) {
  return idrak_flash_bwd_ex(q, k, v, out, dout, lse, delta, dq, dk, dv, B, H, Hkv, Sq, Skv, D, q_row_stride,
                            k_row_stride, v_row_stride, q_batch_stride, k_batch_stride, v_batch_stride, dq_row_stride,
                            dk_row_stride, dv_row_stride, scale, causal, 0, nullptr, 0.f, nullptr, stream_);
}
