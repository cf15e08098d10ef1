// Few-row products for decoding: C[M, N] = X[M, K] W[N, K]^T with M <= 64 tokens, bound by streaming W once.
//
// The product is computed transposed, so the weights fill the 128-row side of the tensor-core tile and the tokens the
// narrow side: D[128 features, NT tokens] += W_tile[128, 64] X_tile[NT, 64]^T per K block (tcgen05.mma M = 128,
// N = NT in {16, 32, 64}, fp32 accumulator in TMEM). One tile of 128 output features belongs to a CLUSTER of 1 to 8 CTAs
// that split K between them, which is what fills the machine when N / 128 is below the SM count (a 4096-wide projection
// is 32 tiles). Each CTA:
//   warp 0      TMA producer: its K range of the W tile (16 KB per block) and of X (NT x 64) through a ring of stages
//   warp 1      MMA issuer
//   warps 2..9  meanwhile sum the squares of this CTA's K range of X (only when the RMS norm is folded in) or expand the
//               codes of a packed weight, then move the accumulator into shared memory
// then the cluster meets and CTA r finishes the tokens r, r + c, r + 2c, ...: it sums the c partial tiles of its tokens
// through distributed shared memory in rank order - deterministic, no second kernel, no fp32 workspace in HBM - and
// runs the epilogue on them:
//   norm fold   y *= rsqrt(mean_k x^2 + eps): with the norm weight multiplied into W's columns beforehand this is
//               RMSNorm(x) W^T without a norm launch or a normalised copy of x
//   bias, residual add
//   gated       W holds [gate rows; up rows]; a tile pairs 64 gate features with their 64 up features and writes
//               act(gate) * up: no [M, 2 ff] round trip, no activation launch
// The reduction is split by tokens, not by features, so that c can be any number up to 8 (6144 features are 48 tiles of
// 5 CTAs: 240 of the 296 that fit), and only the M real tokens are summed. Shared memory is 112 KB per CTA so two CTAs
// share an SM.
//
// Packed weights (int8 codes with one scale per output, int4 codes with one scale per 32 inputs and output) are stored
// [inputs, outputs] and read in that layout, from 17 tokens on (below that: skinny_packed.cu): the eight warps turn each
// block of codes into an MN-major bf16 operand tile in a ring of its own while the next blocks are in flight, one 16-byte
// chunk per eight codes of one input. int8 codes enter the tensor core as exact numbers and their scale multiplies the
// sum; int4 codes are multiplied by their group's scale in fp32 and rounded to bf16 once, the same value as unpacking the
// weight first.
//
// Launched with programmatic serialization: while the kernels ahead still run, a CTA sets up and asks for its first
// weight blocks to be brought into L2, so the weight stream does not stop between products. A prefetch into L2 reads
// nothing into the kernel, so weights that the kernels ahead still write are read as they left them.
//
// Measured with a small norm kernel before each product and weights that no cache holds, us at 64 tokens / 1 token
// (before: feature-split reduction over 1, 2, 4 or 8 CTAs, four epilogue warps, no prefetch; floor at 6544 GB/s):
//   6144 x 4096    13.5 / 11.3  (19.1 / 14.4; 7.7)       4096 x 4096     11.5 / 8.8   (17 to 29 / 10.8; 5.1)
//   4096 x 14336   24.3 / 20.5  (32 / 24; 17.9)          28672 x 4096    44.9 / 39.0  (73.9 / -; 35.9)
//
// Every mbarrier wait is bounded (status word + abort flag); every thread reaches both cluster barriers whatever
// happened before, so no CTA leaves while a peer still reads its shared memory.
//
// Reference counterparts: the few-row GEMV family with fused epilogues (src/Idrak.Gpu/Cuda/PtxKernels.Quantized.cs:13,
// 454-495: *_gemv_multi, _multi_act, _addnorm, _normaddnorm) and PtxKernels.Rows.cs:2047-2060.
#include "skinny_common.cuh"

namespace idrak {

constexpr int kSkFeat = 128;     // output features per tile (MMA M)
constexpr int kSkBK = 64;        // K elements per stage
constexpr int kSkWarps = 8;      // epilogue warps
constexpr int kSkThreads = 64 + kSkWarps * 32;

struct SkinnyParams {
  const __nv_bfloat16* X;        // [M, ldx]
  int ldx, K;
  SkinnyOut o;
  const __half* scales;          // int8: [outputs]; int4: [groups, scale_ld]
  int scale_ld;
  float norm_eps;                // >= 0: multiply row m by rsqrt(sum_k x[m,k]^2 / K + eps)
  int csize;                     // CTAs per cluster = K splits
  Status* st;
};

template <int NT, int kBits>
struct SkinnySmem {
  static constexpr int kX = NT * kSkBK * 2;
  static constexpr int kW = kSkFeat * kSkBK * kBits / 8;  // a block of W as it is stored
  static constexpr int kStage = kW + kX;
  static constexpr int kOps = kBits == 16 ? 0 : 3;        // operand tiles of a packed weight
  static constexpr int kOp = kSkFeat * kSkBK * 2;
  static constexpr int kFixed = 64 * 4 * 2 + 512 + 1024;  // sums of squares, barriers, alignment
  static constexpr int kBudget = 112 * 1024;              // two CTAs per SM
  static constexpr int kFit = (kBudget - kFixed - kOps * kOp) / kStage;
  static constexpr int kStages = kFit < 12 ? kFit : 12;
  static constexpr int kRing = kOps * kOp;                // where the stages start
  // after the main loop everything before kSs is reused for the partial tile [NT][128] fp32
  static constexpr int kSs = kRing + kStages * kStage;
  static constexpr int kBar = kSs + 64 * 4 * 2;
  static constexpr int kTotal = kBar + 512 + 1024;
  static_assert(kStages >= 3 && NT * kSkFeat * 4 <= kSs, "ring too small");
};

// Four int8 codes of consecutive features per word -> bf16 code / 64, exactly: an unsigned integer u < 256 in a 16-bit lane
// is, read as bf16, u * 2^-133; one fused multiply-add takes it to (u - 128) / 64 (the 64 goes into the scale).
__device__ __forceinline__ uint32_t sk_int8_pair(uint32_t t) {
  const uint32_t mul = 0x7F007F00u, add = 0xC000C000u;
  const __nv_bfloat162 v = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&t), *reinterpret_cast<const __nv_bfloat162*>(&mul),
                                   *reinterpret_cast<const __nv_bfloat162*>(&add));
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint4 sk_int8_words(uint32_t a, uint32_t b) {
  a ^= 0x80808080u;
  b ^= 0x80808080u;
  return make_uint4(sk_int8_pair(__byte_perm(a, 0, 0x4140)), sk_int8_pair(__byte_perm(a, 0, 0x4342)),
                    sk_int8_pair(__byte_perm(b, 0, 0x4140)), sk_int8_pair(__byte_perm(b, 0, 0x4342)));
}

// Eight int4 codes of one word times their scales -> four bf16 pairs. s[i] holds scale i times 16^-(i & 3): the nibble is
// dropped where it stands into the mantissa of 2^23, so that subtracting 2^23 + 8 * 16^(i & 3) leaves code * 16^(i & 3)
// exactly, and the product with s[i] is code * scale exactly (4 x 11 bits) before the one rounding to bf16.
__device__ __forceinline__ uint4 sk_int4_word(uint32_t word, const float (&s)[8]) {
  const uint32_t x = word ^ 0x88888888u, y = x >> 16;
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int sh = 4 * (i & 3);
    const uint32_t bits = ((i < 4 ? x : y) & (0xFu << sh)) | 0x4B000000u;
    v[i] = (__uint_as_float(bits) - (8388608.f + float(8 << sh))) * s[i];
  }
  return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}

template <int NT, int kBits>
__global__ void __launch_bounds__(kSkThreads, 2)
skinny_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SkinnyParams p) {
  using L = SkinnySmem<NT, kBits>;
  constexpr int kStages = L::kStages;
  constexpr int FT = kSkFeat;
  constexpr int kTmemCols = NT < 32 ? 32 : NT;
  constexpr int kHalf = FT / 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* part = reinterpret_cast<float*>(smem);
  float* ss_part = reinterpret_cast<float*>(smem + L::kSs);
  float* ss = ss_part + 64;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* empty = full + kStages;
  uint64_t* op_full = empty + kStages;                 // [kOps], packed weights only
  uint64_t* op_empty = op_full + L::kOps;
  uint64_t* acc_full = op_empty + L::kOps;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int csize = p.csize;
  const int rank = int(sk_cluster_rank());
  const int tile = blockIdx.x / csize;
  const bool gated = p.o.gate_kind >= 0;
  const int kblocks = (p.K + kSkBK - 1) / kSkBK;
  const int kb0 = int((long long)kblocks * rank / csize), kb1 = int((long long)kblocks * (rank + 1) / csize);

  pdl_launch_dependents();
  // first output of half h of the tile: its outputs [0, FT / 2) and [FT / 2, FT), or the gate and the up features
  auto half_row = [&](int h) { return gated ? h * p.o.up_offset + tile * kHalf : tile * FT + h * kHalf; };
  auto issue = [&](int kb, int stage) {
    uint8_t* sw = smem + L::kRing + stage * L::kStage;
    mbar_expect_tx(&full[stage], L::kStage);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (kBits == 16) tma_load_2d(sw + h * (L::kW / 2), &tmW, &full[stage], kb * kSkBK, half_row(h));
      else tma_load_2d(sw + h * (L::kW / 2), &tmW, &full[stage], half_row(h) * kBits / 8, kb * kSkBK);
    }
    tma_load_2d(sw + L::kW, &tmX, &full[stage], kb * kSkBK, 0);
  };
  const int first = min(kStages, kb1 - kb0);            // stages filled before the CTA-wide sync (all are free then)
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    for (int i = 0; i < first; ++i) {                    // see the head of the file
      for (int h = 0; h < 2; ++h) {
        if (kBits == 16) sk_prefetch_2d(&tmW, (kb0 + i) * kSkBK, half_row(h));
        else sk_prefetch_2d(&tmW, half_row(h) * kBits / 8, (kb0 + i) * kSkBK);
      }
    }
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < L::kOps; ++s) {
      mbar_init(&op_full[s], kSkWarps);
      mbar_init(&op_empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    fence_barrier_init();
    pdl_wait();                                          // the kernels before this one have written the token rows
    for (int i = 0; i < first; ++i) issue(kb0 + i, i);   // in flight while tensor memory is allocated below
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();                                            // every thread that reads global memory (rows, bias, residual)
  const uint32_t tmem_acc = *tmem_slot;
  bool ok = true;

  if (warp == 0) {
    if (lane == 0) {
      int stage = first % kStages;
      uint32_t phase = first == kStages ? 1u : 0u;
      uint32_t issued_mask = (1u << first) - 1u, issued_phase = 0;
      for (int kb = kb0 + first; kb < kb1 && ok; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.st, kTimeoutSmemEmpty, (7u << 16) | stage)) {
          ok = false;
          break;
        }
        issue(kb, stage);
        issued_mask |= 1u << stage;
        issued_phase = (issued_phase & ~(1u << stage)) | (phase << stage);
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
      if (!ok || *abort_flag) {
        for (int s = 0; s < kStages; ++s) {
          if (issued_mask & (1u << s)) {
            const uint32_t par = (issued_phase >> s) & 1u;
            for (int i = 0; i < (1 << 20); ++i)
              if (mbar_try_wait(&full[s], par)) break;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // bf16 weights are K-major rows; an expanded tile is MN-major (two blocks of 64 features)
      constexpr uint32_t idesc = make_idesc_f16(128, NT, kBits == 16 ? 0 : 1, 0, 1);
      int stage = 0, ob = 0;
      uint32_t phase = 0, op_phase = 0;
      for (int kb = kb0; kb < kb1 && ok; ++kb) {
        if (!mbar_wait(&full[stage], phase, abort_flag, p.st, kTimeoutSmemFull, (7u << 16) | (16 + stage)) ||
            (kBits != 16 && !mbar_wait(&op_full[ob], op_phase, abort_flag, p.st, kTimeoutSmemFull, (7u << 16) | (32 + ob)))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t ring = smem_u32(smem + L::kRing + stage * L::kStage);
        const uint32_t sw = kBits == 16 ? ring : smem_u32(smem + ob * L::kOp);
        const uint32_t sx = ring + L::kW;
#pragma unroll
        for (int kk = 0; kk < kSkBK / 16; ++kk) {
          const uint64_t da = kBits == 16 ? make_smem_desc_sw128(sw + kk * 32, 16, 1024)
                                          : make_smem_desc_sw128(sw + kk * 2048, 8192, 1024);
          const uint64_t db = make_smem_desc_sw128(sx + kk * 32, 16, 1024);
          tc_mma_f16_ss(tmem_acc, da, db, idesc, (kb > kb0 || kk > 0) ? 1u : 0u);
        }
        tc_commit(&empty[stage]);
        if (kBits != 16) {
          tc_commit(&op_empty[ob]);
          if (++ob == L::kOps) { ob = 0; op_phase ^= 1; }
        }
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
      if (ok) tc_commit(acc_full);
    }
  } else {
    if constexpr (kBits != 16) {
      // ---------------------------------------------------------------- codes -> bf16 operand tiles
      // a thread owns one unit of eight features and a run of kRows inputs (inside one group of 32) of every block
      constexpr int kUnits = FT / 8, kHalfUnits = kUnits / 2;
      constexpr int kRows = kSkBK * kUnits / (kSkWarps * 32);
      constexpr int kRowBytes = kHalf * kBits / 8;         // one input of one half of the tile
      const int t = threadIdx.x - 64;
      const int u = t % kUnits, r0 = (t / kUnits) * kRows, h = u / kHalfUnits;
      const uint8_t* src = smem + L::kRing + h * (L::kW / 2) + (u - h * kHalfUnits) * kBits;
      const int dst_block = (u >> 3) * 8192, chunk = u & 7;
      const int col = half_row(h) + (u - h * kHalfUnits) * 8;
      auto scales_of = [&](int kb) {
        const int group = (kb * kSkBK + r0) >> 5;
        if (kBits != 4 || group >= (p.K + 31) / 32 || col + 8 > p.scale_ld) return make_uint4(0, 0, 0, 0);
        return __ldg(reinterpret_cast<const uint4*>(p.scales + size_t(group) * p.scale_ld + col));
      };
      uint4 next_scales = kb0 < kb1 ? scales_of(kb0) : make_uint4(0, 0, 0, 0);
      int stage = 0, ob = 0;
      uint32_t phase = 0, op_phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        float s[8];
        if (kBits == 4) {
          const uint32_t sw[4] = {next_scales.x, next_scales.y, next_scales.z, next_scales.w};
          constexpr float kPow[4] = {1.f, 0.0625f, 0.00390625f, 0.000244140625f};
#pragma unroll
          for (int i = 0; i < 8; ++i)
            s[i] = __half2float(__ushort_as_half((unsigned short)((sw[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu))) * kPow[i & 3];
          if (kb + 1 < kb1) next_scales = scales_of(kb + 1);
        }
        bool go = mbar_wait(&op_empty[ob], op_phase ^ 1, abort_flag, p.st, kTimeoutSmemEmpty, (7u << 16) | (36 + ob));
        go = go && mbar_wait(&full[stage], phase, abort_flag, p.st, kTimeoutSmemFull, (7u << 16) | (40 + stage));
        if (!__all_sync(0xffffffffu, go)) { ok = false; break; }
        uint8_t* dst = smem + ob * L::kOp + dst_block;
        const uint8_t* codes = src + stage * L::kStage;
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const int r = r0 + (i ^ h);                      // the halves start on the same banks: their rows are read crossed
          uint4 o;
          if (kBits == 8) {
            const uint2 w = *reinterpret_cast<const uint2*>(codes + r * kRowBytes);
            o = sk_int8_words(w.x, w.y);
          } else {
            o = sk_int4_word(*reinterpret_cast<const uint32_t*>(codes + r * kRowBytes), s);
          }
          *reinterpret_cast<uint4*>(dst + r * 128 + ((chunk ^ (r & 7)) << 4)) = o;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&op_full[ob]);
        if (++stage == kStages) { stage = 0; phase ^= 1; }
        if (++ob == L::kOps) { ob = 0; op_phase ^= 1; }
      }
    } else if (p.norm_eps >= 0.f) {
      // sum of squares of this CTA's K range, one warp per token row
      const int k_lo = kb0 * kSkBK, k_hi = min(p.K, kb1 * kSkBK);
      for (int m = warp - 2; m < NT; m += kSkWarps) {
        float acc = 0.f;
        if (m < p.o.M) {
          const __nv_bfloat16* row = p.X + size_t(m) * p.ldx;
          for (int k = k_lo + lane * 8; k < k_hi; k += 256) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(row + k));
            float2 f;
            f = unpack_bf16x2(v.x); acc += f.x * f.x + f.y * f.y;
            f = unpack_bf16x2(v.y); acc += f.x * f.x + f.y * f.y;
            f = unpack_bf16x2(v.z); acc += f.x * f.x + f.y * f.y;
            f = unpack_bf16x2(v.w); acc += f.x * f.x + f.y * f.y;
          }
        }
        acc = warp_sum(acc);
        if (lane == 0) ss_part[m] = acc;
      }
    }
    // ---------------------------------------------------------------- accumulator -> shared memory
    const bool have = kb1 > kb0;
    if (have && ok) ok = mbar_wait(acc_full, 0, abort_flag, p.st, kTimeoutTmemFull, (7u << 16) | 60);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    const int q = warp & 3;                              // the TMEM lane quarter this warp may read
    const int set = (warp - 2) >> 2;                     // which half of the tokens it moves
    const int f = q * 32 + lane;
    constexpr int kCols = NT >= 32 ? NT / 2 : NT;
    const int c_first = set * kCols;
    if (c_first < NT) {
      if (have && ok) {
#pragma unroll
        for (int c = 0; c < kCols / 16; ++c) {
          uint32_t v[16];
          const int col0 = c_first + c * 16;
          tmem_ld_32x32b_x16(tmem_acc + (uint32_t(q * 32) << 16) + col0, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) part[(col0 + i) * FT + f] = __uint_as_float(v[i]);
        }
      } else {
        for (int m = 0; m < kCols; ++m) part[(c_first + m) * FT + f] = 0.f;      // no K blocks here, or gave up
      }
    }
  }

  // every thread of every CTA of the cluster: partial tiles (and partial sums of squares) are complete and visible
  tc_fence_before();
  __syncwarp();
  sk_cluster_sync();

  if (warp >= 2) {
    const int t = threadIdx.x - 64;
    if (kBits == 16 && p.norm_eps >= 0.f) {
      const uint32_t ssp_addr = smem_u32(ss_part);
      if (t < (p.o.M - rank + csize - 1) / csize) {
        const int m = rank + t * csize;
        float a = 0.f;
        for (int r = 0; r < csize; ++r) a += sk_ld_cluster(sk_map_rank(ssp_addr + m * 4, r));
        ss[m] = rsqrtf(a / float(p.K) + p.norm_eps);
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    sk_finish<FT, FT>(p.o, part, csize, rank, tile, t, [&](int m, int n) {
      if (kBits == 8) return __half2float(p.scales[n]) * 64.f;
      return kBits == 16 && p.norm_eps >= 0.f ? ss[m] : 1.f;
    });
  }

  // nobody leaves while a peer may still read its shared memory
  __syncwarp();
  sk_cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_acc, kTmemCols);
  }
}

// CTAs per cluster, the ways K is split: as many (up to 8) as fit on the device together, two per SM, with a margin of one
// in seven for the SMs that whole clusters cannot fill; a product with more tiles than that is not split. Measured at 64
// tokens, us: 6144 x 4096 (48 tiles) c = 2 / 4 / 5 / 6 (288 CTAs, no longer together) 16.1 / 13.7 / 13.1 / 18.8; 4096 x 4096
// (32 tiles) c = 2 / 4 / 8 14.8 / 10.7 / 11.0; 4096 x 14336 c = 4 / 7 / 8 27.2 / 24.3 / 24.4; 28672 x 4096 (224 tiles)
// c = 1 / 2 / 4 45.2 / 46.5 / 54.6; int8 codes 6144 x 4096 c = 2 / 4 / 5 / 8 21.8 / 16.3 / 14.7 / 20.4.
template <int NT, int kBits>
static int launch_skinny(const CUtensorMap& tmW, const CUtensorMap& tmX, SkinnyParams& p, cudaStream_t stream, bool one_pass = false) {
  using L = SkinnySmem<NT, kBits>;
  auto kern = skinny_gemm_kernel<NT, kBits>;
  static DeviceOnce configured;
  if (int e = configured.run([&] {
        return int(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal));
      }))
    return e;
  const int half = kSkFeat / 2, kblocks = (p.K + kSkBK - 1) / kSkBK;
  const int tiles = p.o.gate_kind >= 0 ? (p.o.N + half - 1) / half : (p.o.N + kSkFeat - 1) / kSkFeat;
  int c = one_pass ? 1 : skinny_forced_splits();
  if (!c)
    for (c = 8; c > 1 && tiles * c > sm_count() * 2 * 6 / 7;) --c;
  p.csize = c < kblocks ? c : kblocks;
  return skinny_launch(kern, tiles * p.csize, p.csize, kSkThreads, L::kTotal, stream, tmW, tmX, p);
}

static int encode_tokens(CUtensorMap* tm, const void* X, int ldx, int M, int K, int NT) {
  uint64_t dims[2] = {uint64_t(K), uint64_t(M)};
  uint64_t strides[1] = {uint64_t(ldx) * 2};
  uint32_t box[2] = {uint32_t(kSkBK), uint32_t(NT)};
  return encode_tensor_map(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(X), dims, strides, box,
                           CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace idrak

using namespace idrak;

// C[M, N] = epilogue(X[M, K] W^T), M <= 64. W is [N, K] (ldw elements per row), or with gate_kind >= 0 the stacked
// [gate; up] matrix of 2 * N rows and C = act(x Wg^T) * (x Wu^T). norm_eps >= 0 folds an RMS norm over K in (the norm
// weight must already be multiplied into W's columns). one_pass: K is not cut, an element has the bits of the dense kernel's
// uncut sum. K % 8 == 0, rows 16-byte aligned. Returns 0, a CUDA error, or a negative argument error.
IDRAK_API int idrak_skinny_gemm(const void* X, int ldx, const void* W, int ldw, void* C, int ldc, int M, int N, int K,
                                const void* bias, const void* residual, int ldr, int gate_kind, float norm_eps,
                                int one_pass, void* stream_) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > 64) return -2;
  if ((K & 7) || (ldx & 7) || (ldw & 7)) return -3;
  if ((reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(W) & 15)) return -4;
  if (gate_kind > 2) return -5;
  const bool gated = gate_kind >= 0;
  if (gated && (N % 8)) return -6;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  SkinnyParams p{};
  p.X = static_cast<const __nv_bfloat16*>(X); p.ldx = ldx; p.K = K;
  p.o = {static_cast<__nv_bfloat16*>(C), ldc, static_cast<const __nv_bfloat16*>(bias),
         static_cast<const __nv_bfloat16*>(residual), ldr, M, N, gated ? gate_kind : -1, gated ? N : 0, gated ? N : 0};
  p.norm_eps = norm_eps;
  p.st = status_device_ptr();
  const int NT = M <= 16 ? 16 : (M <= 32 ? 32 : 64);
  CUtensorMap tmW, tmX;
  uint64_t dims[2] = {uint64_t(K), uint64_t(gated ? 2 * N : N)};
  uint64_t strides[1] = {uint64_t(ldw) * 2};
  uint32_t box[2] = {uint32_t(kSkBK), uint32_t(kSkFeat / 2)};
  if (encode_tensor_map(&tmW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(W), dims, strides, box,
                        CU_TENSOR_MAP_SWIZZLE_128B))
    return -10;
  if (encode_tokens(&tmX, X, ldx, M, K, NT)) return -11;
  if (NT == 16) return launch_skinny<16, 16>(tmW, tmX, p, stream, one_pass);
  if (NT == 32) return launch_skinny<32, 16>(tmW, tmX, p, stream, one_pass);
  return launch_skinny<64, 16>(tmW, tmX, p, stream, one_pass);
}

// C[M, N] = epilogue(X[M, K] W) over a packed weight stored [K inputs, outputs] (gated: outputs = [gate | up], 2 * N of
// them, and C = act(x Wg) * (x Wu)): bits = 8, one code per byte (ld bytes per row) and one fp16 scale per output, or
// bits = 4, eight codes per 32-bit word (ld bytes per row) and one fp16 scale per 32 inputs and output (scale_ld per group
// row). M <= 64, K a multiple of 16 (int8) or 32 (int4); rows of X, codes and int4 scales start on 16-byte boundaries, and
// so does a gated weight's up half, which starts at column up_col of the codes: N, or for int8 codes whose halves are padded
// a multiple of 16 past it (scales and bias are not padded). Returns 0, a CUDA error, or a negative argument error.
//
// Up to 16 tokens the register kernel (skinny_packed.cu) is the faster one, above them this file's, whose tensor cores take
// 64 tokens at the price of 16: 4096 x 28672 int8, us, register / this kernel at 16 tokens 33 / 57, at 64 tokens 97 / 61.
IDRAK_API int idrak_skinny_packed(const void* X, int ldx, const void* codes, int ld, const void* scales, int scale_ld,
                                  int bits, void* C, int ldc, int M, int N, int K, const void* bias, const void* residual,
                                  int ldr, int gate_kind, int up_col, void* stream_) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > 64) return -2;
  if (bits != 8 && bits != 4) return -7;
  if ((ldx & 7) || (ld & 15) || (K % (bits == 8 ? 16 : 32))) return -3;
  if ((reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(codes) & 15)) return -4;
  if (gate_kind > 2) return -5;
  const bool gated = gate_kind >= 0;
  const int outputs = gated ? 2 * N : N;
  if (gated && (up_col % (bits == 8 ? 16 : 32) || up_col < N || (bits == 4 && up_col != N))) return -6;
  if ((long long)ld * (8 / bits) < (gated ? up_col + N : N) || scale_ld < outputs) return -8;
  if (bits == 4 && ((scale_ld & 7) || (reinterpret_cast<uintptr_t>(scales) & 15))) return -9;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const SkinnyOut o = {static_cast<__nv_bfloat16*>(C), ldc, static_cast<const __nv_bfloat16*>(bias),
                       static_cast<const __nv_bfloat16*>(residual), ldr, M, N, gated ? gate_kind : -1, gated ? up_col : 0,
                       gated ? N : 0};
  if (M <= kSkinnyRegisterRows)
    return skinny_packed_registers(static_cast<const __nv_bfloat16*>(X), ldx, codes, ld, static_cast<const __half*>(scales),
                                   scale_ld, bits, K, o, stream);
  SkinnyParams p{};
  p.X = static_cast<const __nv_bfloat16*>(X); p.ldx = ldx; p.K = K;
  p.o = o;
  p.scales = static_cast<const __half*>(scales); p.scale_ld = scale_ld;
  p.norm_eps = -1.f;
  p.st = status_device_ptr();
  const int NT = M <= 32 ? 32 : 64;
  CUtensorMap tmW, tmX;
  uint64_t dims[2] = {uint64_t(ld), uint64_t(K)};
  uint64_t strides[1] = {uint64_t(ld)};
  uint32_t box[2] = {uint32_t(kSkFeat / 2 * bits / 8), uint32_t(kSkBK)};
  if (encode_tensor_map(&tmW, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(codes), dims, strides, box,
                        CU_TENSOR_MAP_SWIZZLE_NONE))
    return -10;
  if (encode_tokens(&tmX, X, ldx, M, K, NT)) return -11;
  if (bits == 8) return NT == 32 ? launch_skinny<32, 8>(tmW, tmX, p, stream) : launch_skinny<64, 8>(tmW, tmX, p, stream);
  return NT == 32 ? launch_skinny<32, 4>(tmW, tmX, p, stream) : launch_skinny<64, 4>(tmW, tmX, p, stream);
}
