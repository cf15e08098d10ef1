// Flash attention forward for sm_100a, two query tiles per CTA: causal or full, grouped heads, head size 128.
//
// One CTA owns 256 query rows of one (batch, head) as two tiles of 128 and walks the keys in blocks of 128 for both:
//   warp 0       TMA producer: both Q tiles, then K and V blocks in turn through one ring of four stages
//   warp 1       MMA issuer: per block and tile O += P V, then the tile's next S = Q K^T
//   warps 4..11  softmax of tile 0, warps 12..19 of tile 1: two threads per row with 64 of the block's 128 scores each
// While one tile's scores are in the exponential unit, the tensor core has the other tile's products. With one tile per CTA
// (flash_fwd.cu, the tensor pipe busy a third of the time) a block is a chain of scores, row maximum, exponentials, P and
// accumulation, 2800 cycles for 1024 of MMA and 1024 of exponentials. A thread per row, which needs no exchange of maxima, is a
// chain of 3200 cycles by itself: with one warp of a tile to a scheduler nothing fills its latencies (8192 positions, 32 heads on
// 8: 597 us).
//
// Tensor memory is full: S of both tiles, O of both tiles. P is written over the scores it was made from, so a tile's next scores
// wait for the accumulation that reads P - and a tile whose scores have come may rescale its accumulator at once.
//
// The arithmetic of a row is that of flash_fwd.cu in the same order (sums of a block's two halves apart), so a row has the
// same bits on either kernel but for the moment a warp's rows are rescaled together.
//
// Measured, us, two threads per row and one tile / this: 1 x 8192, 32 heads on 8, 666, 549 (700 before the row blocks were put in order
// over all heads); 4 x 2048 231, 184; 1 x 4096, 16 heads 97, 80. What bounds it is still the chain of a tile's block: the tensor pipe and
// the exponential unit are busy 43 % of the time each.
//
// Reference counterparts: flash_tc_fwd_d{64,128} (src/Idrak.Gpu/Cuda/PtxKernels.FlashTensorCore.cs:318-321).
#include "flash_common.cuh"
#include "flash_fwd_pair.h"

namespace idrak {

constexpr int kPairFwdThreads = 640;      // producer warpgroup (TMA warp, MMA warp, two idle), two softmax warpgroups per tile
// registers: 640 x 96 at launch, 128 x 40 + 512 x 104 afterwards
constexpr int kPairFwdStages = 4;

template <int D>
struct PairFwdSmem {
  static constexpr int kTile = 128 * D * 2;
  static constexpr int kQ = 0;                               // two tiles
  static constexpr int kRing = kQ + 2 * kTile;
  static constexpr int kXch = kRing + kPairFwdStages * kTile;   // row maxima and sums: [tile][parity][half][128 rows]
  static constexpr int kBar = kXch + 4096;
  static constexpr int kTotal = kBar + 256 + 1024;
  static_assert(kTotal <= 232448, "shared memory per CTA");
};

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <int D>
__global__ void __launch_bounds__(kPairFwdThreads, 1)
flash_fwd_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const FlashParams p) {
  using L = PairFwdSmem<D>;
  constexpr int NS = kPairFwdStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* q_full = bars;             // [2]
  uint64_t* full = bars + 2;           // [stages]
  uint64_t* empty = bars + 7;          // [stages]
  uint64_t* s_full = bars + 12;        // [2] the tile's scores are in tensor memory
  uint64_t* p_full = bars + 14;        // [2] its probabilities are
  uint64_t* o_done = bars + 16;        // [2] the accumulation that read them is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const FwdUnit unit = fwd_unit(p, 256);
  const int qb = unit.qb, head = unit.head, batch = unit.batch;
  const int kv_head = head / (p.H / p.Hkv);
  const int q0 = qb * 256;
  const int off = p.Skv - p.Sq;        // causal: query row r sees keys <= r + off
  int nkv[2];                          // key blocks of each tile
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    int n = (p.Skv + 127) / 128;
    const int first = q0 + t * 128;
    if (p.causal) n = min(n, (first + 127 + off) / 128 + 1);
    nkv[t] = first < p.Sq ? max(n, 0) : 0;
  }
  const int blocks = max(nkv[0], nkv[1]);

  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1);
      mbar_init(&s_full[t], 1);
      mbar_init(&p_full[t], 8);
      mbar_init(&o_done[t], 1);
    }
    for (int s = 0; s < NS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  // S of the tiles [0, 128) and [128, 256), O at [256, 256 + D) and [256 + D, 256 + 2 D); P in the first 64 columns of its S
  constexpr uint32_t kTmemCols = 512;
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_O = tmem_base + 256;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 0 && lane == 0 && blocks > 0) {
      bool ok = true;
      auto load = [&](int i, const CUtensorMap* tm, int block) {       // the i-th tile of the ring
        const int st = i % NS;
        if (!mbar_wait(&empty[st], uint32_t((i / NS) & 1) ^ 1u, abort_flag, p.st, kTimeoutSmemEmpty, (10u << 16) | st)) return false;
        mbar_expect_tx(&full[st], L::kTile);
#pragma unroll
        for (int c = 0; c < D / 64; ++c)
          tma_load_4d(smem + L::kRing + st * L::kTile + c * 16384, tm, &full[st], c * 64, block * 128, kv_head, batch);
        return true;
      };
      for (int t = 0; t < 2; ++t) {
        if (nkv[t] > 0) {
          mbar_expect_tx(&q_full[t], L::kTile);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(smem + L::kQ + t * L::kTile + c * 16384, &tmQ, &q_full[t], c * 64, q0 + t * 128, head, batch);
        }
        if (t == 0) ok = load(0, &tmK, 0);
      }
      for (int j = 0; j < blocks && ok; ++j) {
        if (j > 0) ok = load(2 * j, &tmK, j);
        ok = ok && load(2 * j + 1, &tmV, j);
      }
      if (!ok || *abort_flag) {          // let the copies on their way land before shared memory is released
        const uint64_t from = global_timer_ns();
        while (global_timer_ns() - from < 200000ull) { }
      }
    } else if (warp == 1 && lane == 0 && blocks > 0) {
      constexpr uint32_t idesc_s = make_idesc_f16(128, 128, 0, 0, 1);
      constexpr uint32_t idesc_o = make_idesc_f16(128, D, 0, 1, 1);
      // scores of block j for tile t
      auto scores = [&](int t, int j) {
        const int st = (2 * j) % NS;
        if (!mbar_wait(&full[st], uint32_t((2 * j) / NS) & 1u, abort_flag, p.st, kTimeoutSmemFull, (10u << 16) | (8 + st))) return false;
        // P of the block before lies there until its accumulation has read it
        if (j > 0 && !mbar_wait(&o_done[t], uint32_t(j - 1) & 1u, abort_flag, p.st, kTimeoutTmemEmpty, (10u << 16) | (16 + t))) return false;
        tc_fence_after();
        const uint32_t sq = smem_u32(smem + L::kQ + t * L::kTile), sk = smem_u32(smem + L::kRing + st * L::kTile);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t o = (kk >> 2) * 16384 + (kk & 3) * 32;
          tc_mma_f16_ss(tmem_base + t * 128, make_smem_desc_sw128(sq + o, 16, 1024), make_smem_desc_sw128(sk + o, 16, 1024), idesc_s,
                        kk > 0 ? 1u : 0u);
        }
        tc_commit(&s_full[t]);
        return true;
      };
      bool ok = true;
      for (int t = 0; t < 2 && ok; ++t)
        if (nkv[t] > 0)
          ok = mbar_wait(&q_full[t], 0, abort_flag, p.st, kTimeoutSmemFull, (10u << 16) | (20 + t)) && scores(t, 0);
      if (ok) tc_commit(&empty[0]);
      for (int j = 0; j < blocks && ok; ++j) {
        const int sv_st = (2 * j + 1) % NS;
        for (int t = 0; t < 2 && ok; ++t) {
          if (j < nkv[t]) {
            ok = mbar_wait(&full[sv_st], uint32_t((2 * j + 1) / NS) & 1u, abort_flag, p.st, kTimeoutSmemFull, (10u << 16) | (24 + sv_st)) &&
                 mbar_wait(&p_full[t], uint32_t(j) & 1u, abort_flag, p.st, kTimeoutGeneric, (10u << 16) | (30 + t));
            if (!ok) break;
            tc_fence_after();
            const uint32_t sv = smem_u32(smem + L::kRing + sv_st * L::kTile);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              tc_mma_f16_ts(tmem_O + t * D, tmem_base + t * 128 + kk * 8, make_smem_desc_sw128(sv + kk * 2048, 16384, 1024), idesc_o,
                            (j > 0 || kk > 0) ? 1u : 0u);
            tc_commit(&o_done[t]);
          }
          if (t == 1) tc_commit(&empty[sv_st]);
          if (j + 1 < nkv[t]) ok = scores(t, j + 1);
        }
        if (ok && j + 1 < blocks) tc_commit(&empty[(2 * (j + 1)) % NS]);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    const int t = (warp - 4) >> 3;               // the tile
    const int quarter = warp & 3;
    const int half = ((warp - 4) >> 2) & 1;      // which 64 columns of the block
    const int r = quarter * 32 + lane;           // row within the tile == TMEM lane
    const int row = q0 + t * 128 + r;            // query position
    const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
    constexpr int kOC = D / 2;                   // accumulator columns this thread rescales and stores
    const uint32_t s_addr = tmem_base + t * 128 + lane_addr, o_addr = tmem_O + t * D + lane_addr + half * kOC;
    float* xch = reinterpret_cast<float*>(smem + L::kXch) + t * 512;
    const uint32_t pair_bar = 1 + t * 4 + quarter;
    const float sl2 = p.scale_log2;
    const int n = nkv[t];
    float m_used = -INFINITY;                    // max the accumulator and the running sum are scaled by
    float l = 0.f;                               // this thread's part of the row sum
    bool ok = n > 0;
    // A thread whose wait gave up keeps walking the loop without touching tensor memory: its partner meets it at the pair's barrier
    // in every block, and that barrier has no time limit of its own.
    for (int j = 0; j < n; ++j) {
      if (ok && !warp_wait(&s_full[t], uint32_t(j) & 1u, abort_flag, p.st, kTimeoutTmemFull, (10u << 16) | (32 + t))) ok = false;
      tc_fence_after();
      uint32_t s[2][32];
      if (ok) {
        tmem_ld_32x32b_x32(s_addr + half * 64, s[0]);
        tmem_ld_32x32b_x32(s_addr + half * 64 + 32, s[1]);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) s[0][i] = s[1][i] = 0u;
      }
      // keys visible to this row among its 64: [0, lim)
      int lim = p.Skv - j * 128 - half * 64;
      if (p.causal) lim = min(lim, row + off - j * 128 - half * 64 + 1);
      const bool masked = __any_sync(0xffffffffu, lim < 64);
      tmem_ld_wait();
      float m2[4];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (masked) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i >= lim) s[c][i] = 0xff800000u;        // -inf
        }
        float a = max3(__uint_as_float(s[c][0]), __uint_as_float(s[c][1]), __uint_as_float(s[c][2])), b = __uint_as_float(s[c][3]);
#pragma unroll
        for (int i = 4; i < 32; i += 4) {
          a = max3(a, __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
          b = max3(b, __uint_as_float(s[c][i + 2]), __uint_as_float(s[c][i + 3]));
        }
        m2[2 * c] = a;
        m2[2 * c + 1] = b;
      }
      // the row maximum over both halves; behind the barrier both hold their scores, so P may be written over them
      float* slot = xch + (j & 1) * 256;
      slot[half * 128 + r] = fmaxf(max3(m2[0], m2[1], m2[2]), m2[3]);
      flash_bar_sync(pair_bar, 64);
      const float m_new = fmaxf(m_used, fmaxf(slot[r], slot[128 + r]) * sl2);
      // the accumulator is rescaled only when some row of this warp moved its max by more than 2^8 (both warps of a quarter hold the
      // same rows and so decide alike). The accumulation of the block before is complete: this block's scores were issued after it
      const bool rescale = __any_sync(0xffffffffu, j > 0 && m_new - m_used > 8.0f);
      if (j == 0) {
        m_used = m_new;
      } else if (rescale) {
        const float alpha = (m_new == -INFINITY) ? 1.f : exp2f(m_used - m_new);
        m_used = m_new;
        l *= alpha;
        if (ok) {
#pragma unroll 1
          for (int c = 0; c < kOC / 16; ++c) {          // 16 columns at a time: the scores stay in registers beside them
            uint32_t o[16];
            tmem_ld_32x32b_x16(o_addr + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32b_x16(o_addr + c * 16, o);
          }
        }
      }
      const float m_sub = (m_used == -INFINITY) ? 0.f : m_used;
      // probabilities -> bf16 A operand of the P V product, two columns of the row per 32-bit column. A masked score is -inf and
      // its probability 0
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float2 l01 = make_float2(0.f, 0.f), l23 = l01;
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float2 x = fma2(as_float2(s[c][i], s[c][i + 1]), make_float2(sl2, sl2), make_float2(-m_sub, -m_sub));
          const float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
          if (i & 2) l23 = add2(l23, e);
          else l01 = add2(l01, e);
          packed[i / 2] = pack_bf16x2(e.x, e.y);
        }
        if (ok) tmem_st_32x32b_x16(s_addr + half * 32 + c * 16, packed);
        l += (l01.x + l01.y) + (l23.x + l23.y);
      }
      if (ok) {
        tmem_st_wait();
        tc_fence_before();
        warp_arrive(&p_full[t]);
      }
    }
    if (ok && n > 0 && !warp_wait(&o_done[t], uint32_t(n - 1) & 1u, abort_flag, p.st, kTimeoutTmemFull, (10u << 16) | (34 + t))) ok = false;
    tc_fence_after();
    // the row sum over both halves
    float* slot = xch + (n & 1) * 256;
    slot[half * 128 + r] = l;
    flash_bar_sync(pair_bar, 64);
    const float l_row = slot[r] + slot[128 + r];
    __nv_bfloat16* orow = p.O + (size_t(batch) * p.Sq + row) * p.o_row_stride + size_t(head) * D + half * kOC;
    if (n <= 0) {
      // no visible key: output zeros, lse = -inf
      if (row < p.Sq) {
        for (int i = 0; i < kOC; i += 8) *reinterpret_cast<uint4*>(orow + i) = make_uint4(0, 0, 0, 0);
        if (p.lse && half == 0) p.lse[(size_t(batch) * p.H + head) * p.Sq + row] = -INFINITY;
      }
    } else if (ok) {
      const float inv = l_row > 0.f ? 1.f / l_row : 0.f;
#pragma unroll
      for (int c = 0; c < kOC / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(o_addr + c * 32, o);
        tmem_ld_wait();
        if (row < p.Sq) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(o[g * 8 + 0]) * inv, __uint_as_float(o[g * 8 + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(o[g * 8 + 2]) * inv, __uint_as_float(o[g * 8 + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(o[g * 8 + 4]) * inv, __uint_as_float(o[g * 8 + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(o[g * 8 + 6]) * inv, __uint_as_float(o[g * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c * 32 + g * 8) = w;
          }
        }
      }
      if (row < p.Sq && p.lse && half == 0) {
        // natural-log LSE of the scaled scores
        p.lse[(size_t(batch) * p.H + head) * p.Sq + row] = (l_row > 0.f) ? (m_used + log2f(l_row)) * 0.6931471805599453f : -INFINITY;
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

// Whether a plain call (no window, packed sequences or soft cap) goes to two query tiles per CTA. (A score that is masked is set to
// -inf before it is scaled, so the scale has to be positive.) Only where they are a CTA for every SM at least: us, one tile and two,
// 32 heads on 8, at 768 positions (96 CTAs of two tiles) 17.4, 21.5, at 1024 (128) 22.8, 25.6, at 1536 (192) 40.4, 34.8, at 2048 (256)
// 61.2, 49.1; 1 x 4096, 16 heads 97.0, 80.1, 8 heads (128) 49.4, 78.1.
bool flash_fwd_pair_wanted(const FlashParams& p, int D) {
  const long long ctas = (long long)((p.Sq + 255) / 256) * p.H * p.B;
  return D == 128 && p.scale > 0.f && ctas >= sm_count() && ctas < (1ll << 30);
}

int flash_fwd_pair_launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashParams& p, cudaStream_t stream) {
  using L = PairFwdSmem<128>;
  auto kern = flash_fwd_pair_kernel<128>;
  static DeviceOnce configured;
  if (int e = configured.run([&] { return int(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal)); }))
    return e;
  kern<<<unsigned((p.Sq + 255) / 256 * p.H * p.B), kPairFwdThreads, L::kTotal, stream>>>(tq, tk, tv, p);
  note_launches(1);
  return int(cudaGetLastError());
}

}  // namespace idrak
