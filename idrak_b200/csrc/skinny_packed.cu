// Few-row products over packed weights: C[M, N] = X[M, K] W[K, N], M <= 16 tokens, W as it is stored: int8 codes with one
// fp16 scale per output, or int4 codes with one fp16 scale per 32 inputs and output. Bound by streaming the codes once,
// a half or a quarter of the bytes of bf16, as long as turning them into operands keeps up.
//
// That turning is the kernel. A tcgen05 operand lives in shared memory: every code would be written there by TMA, read,
// written back as two bytes of bf16 and read again by the tensor core, and each block would pass a barrier from the
// converting warps to the MMA and back (57 us for 4096 x 28672 int8 codes at 16 tokens, three times the stream). Here a
// warp's MMAs take their operands from registers (mma.sync m16n8k16, the weights as the 16-row side; at 8 or 16 tokens the
// legacy tensor pipe is an eighth to a quarter busy): a warp's own ring of TMA boxes brings blocks of 32 inputs x 128 features, its lanes
// read the codes, expand them in registers and multiply; no CTA-wide barrier until the sums. The order of the MMA's k
// index and of its rows is free as long as both operands agree, so a lane takes eight consecutive inputs of 16
// consecutive features: its part of X is one 16-byte load per token.
//
//   int8   code pairs (k, k + 1) of a feature become exact bf16 numbers; the scale multiplies the sum in the epilogue
//   int4   the same, and the scale multiplies each group's partial sum in fp32: weights are never rounded
//
// A CTA is 8 warps: FW side by side along the features (1; 2 for a gated pair, gate beside up), 8 / FW taking every
// (8 / FW)-th block of inputs. Their partial tiles are summed in a fixed tree through shared memory, the CTAs of a cluster
// (which split K further) in rank order through distributed shared memory, and the epilogue (skinny_common.cuh) runs on
// the sum.
//
// What bounds it (counters, 4096 x 28672): no single unit. The integer pipe, which turns the codes (two instructions per pair,
// half rate), is the busiest at half of its peak (int8, 16 tokens 50 %, int4, 7 tokens 47 %; tensor pipe 24 and 14 %), DRAM at
// 37 and 23 %. 224 CTAs share 148 SMs, two on some and one on the others, so 12 of the 16 warps that an SM could hold are
// there on average, and they wait: for loads of X and scales, for the pipe, for the fixed latency of dependent instructions.
// At 4096 x 4096 (one CTA per SM) the integer pipe is a quarter busy and the barriers of the sums weigh as much as the loads.
//
// Measured, us, 16 tokens int8 / 7 tokens int4 (before: tensor-core tiles expanded by four warps from a K-major copy of the
// codes / unpacking to bf16 and a dense product): 4096 x 6144 12.0 / 10.6 (15.7 / 35.4), 4096 x 4096 9.0 / 7.9 (12.2 / 28.9),
// 14336 x 4096 17.6 / 15.8 (24.9 / 75.1), 4096 x 28672 33.0 / 30.7 (48.8 / 145.5).
//
// Launched with programmatic serialization: the first blocks are prefetched into L2 (which reads nothing into the
// kernel) while the kernels ahead finish. Waits are bounded; every thread reaches both cluster barriers.
//
// Reference counterparts: int8_gemv_f32 / int4_gemv_f32 and their fused forms
// (src/Idrak.Gpu/Cuda/PtxKernels.Quantized.cs:13,454-495).
#include "skinny_common.cuh"

namespace idrak {

constexpr int kSpThreads = 256;
constexpr int kSpNF = 128;       // features per warp
constexpr int kSpU = 16;         // features per lane

struct SkinnyPackedParams {
  const __nv_bfloat16* X;        // [M, ldx]
  int ldx, K;
  const __half* scales;          // int8: [outputs]; int4: [K / 32, scale_ld]
  int scale_ld;
  SkinnyOut o;
  int csize;
  Status* st;
};

template <int kBits, int NT, int FW>
struct SkinnyPackedShape {
  static constexpr int KW = 8 / FW;
  static constexpr int F = kSpNF * FW;                     // features per CTA
  static constexpr int kRow = kSpNF * kBits / 8;           // bytes of one input of the warp's features
  static constexpr int kStage = 32 * kRow;                 // a block: 32 inputs
  static constexpr int kStages = kBits == 8 ? 3 : 5;
  static constexpr int kRing = 8 * kStages * kStage;
  static constexpr int kAcc = 8 * (NT / 8) * 4;            // accumulators per lane
  static constexpr int kTree = (KW / 2) * FW * kAcc * 32 * 4;
  static constexpr int kLd = F + 4;                        // floats per token of the partial tile
  static constexpr int kPart = NT * kLd * 4;
  static_assert(kTree <= kRing && kPart <= kRing, "the ring is reused by the sums");
  static constexpr int kTotal = kRing + 8 * kStages * 8 + 64 + 1024;
};

__device__ __forceinline__ void sp_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void sp_lds(uint32_t (&w)[4], uint32_t addr) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr));
}
__device__ __forceinline__ void sp_lds(uint32_t (&w)[2], uint32_t addr) {
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(addr));
}
__device__ __forceinline__ void sp_prefetch_4d(const CUtensorMap* m, int c0, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global [%0, {%1, %2, %3, %2}];" ::"l"(reinterpret_cast<uint64_t>(m)),
               "r"(c0), "r"(0), "r"(c2)
               : "memory");
}
// Codes -> bf16 on as few integer instructions as possible (they run at half rate, on the busiest pipe): an unsigned
// integer u < 256 in a 16-bit lane is, read as bf16, the number u * 2^-133 (subnormal, or with the smallest exponent), so
// one fused multiply-add by a power of two takes it to (u - offset) / 64, exactly; the 64 goes into the scales.
__device__ __forceinline__ uint32_t sp_fma2(uint32_t a, uint32_t mul, uint32_t add) {
  const __nv_bfloat162 v = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&mul),
                                   *reinterpret_cast<const __nv_bfloat162*>(&add));
  return *reinterpret_cast<const uint32_t*>(&v);
}
// Byte e of two words (the inputs k and k + 1 of one feature) -> a pair of bf16 code / 64.
__device__ __forceinline__ uint32_t sp_int8_pair(uint32_t k0, uint32_t k1, int e) {
  const uint32_t t = __byte_perm(k0, k1, e | (e << 4) | ((4 + e) << 8) | ((4 + e) << 12));
  return sp_fma2((t & 0x00FF00FFu) ^ 0x00800080u, 0x7F007F00u, 0xC000C000u);            // * 2^127 - 128 / 64
}
// Nibble i & 3 of both 16-bit halves of h (its upper bytes moved down for nibbles 2 and 3) -> a pair of bf16 code / 64.
__device__ __forceinline__ uint32_t sp_int4_pair(uint32_t h, uint32_t h_upper, int i) {
  const uint32_t w = (i & 2) ? h_upper : h;
  return (i & 1) ? sp_fma2((w & 0x00F000F0u) ^ 0x00800080u, 0x7D007D00u, 0xBE00BE00u)   // * 2^123 - 8 / 64
                 : sp_fma2((w & 0x000F000Fu) ^ 0x00080008u, 0x7F007F00u, 0xBE00BE00u);  // * 2^127 - 8 / 64
}

template <int kBits, int NT, int FW>
__global__ void __launch_bounds__(kSpThreads, 2)
skinny_packed_kernel(const __grid_constant__ CUtensorMap tmW, const SkinnyPackedParams p) {
  using S = SkinnyPackedShape<kBits, NT, FW>;
  constexpr int KW = S::KW, kStages = S::kStages, kWords = kBits / 2;      // words per lane and input
  constexpr int MT = 8, N8 = NT / 8, kHalf = S::F / 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kRing);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(bars + 8 * kStages);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int fw = warp % FW, kw = warp / FW;
  const int csize = p.csize, rank = int(sk_cluster_rank()), tile = blockIdx.x / csize;
  const bool gated = FW > 1 && p.o.gate_kind >= 0;

  pdl_launch_dependents();
  // this lane's features start at local feature lf of the tile; its warp's at weight column wcol (gated: the first half of
  // the tile's warps hold gate features, the second half the up features of the same outputs)
  const int wlf = fw * kSpNF, lf = wlf + g * kSpU;
  const int wcol = !gated ? tile * S::F + wlf : (wlf < kHalf ? tile * kHalf + wlf : p.o.up_offset + tile * kHalf + wlf - kHalf);
  const int col = wcol + g * kSpU;
  const int blocks = (p.K + 31) / 32;
  const int b0 = int((long long)blocks * rank / csize) + kw, b1 = int((long long)blocks * (rank + 1) / csize);
  uint8_t* ring = smem + warp * (kStages * S::kStage);
  uint64_t* full = bars + warp * kStages;
  const int x0 = wcol * kBits / 8;
  auto issue = [&](int blk, int stage) {                   // lane 0: a block of codes into a stage
    mbar_expect_tx(&full[stage], S::kStage);
    tma_load_4d(ring + stage * S::kStage, &tmW, &full[stage], x0, 0, blk * 4, 0);
  };
  if (threadIdx.x == 0) *abort_flag = 0;
  if (lane == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      if (b0 + s * KW < b1) sp_prefetch_4d(&tmW, x0, (b0 + s * KW) * 4);
    }
    fence_barrier_init();
  }
  __syncthreads();
  pdl_wait();
  if (lane == 0)
    for (int s = 0; s < kStages; ++s)
      if (b0 + s * KW < b1) issue(b0 + s * KW, s);

  float acc[MT][N8][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < N8; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f;

  // the tokens' inputs 8 t .. 8 t + 7 of a block: pairs (0, 1), (2, 3) are the first MMA's, (4, 5), (6, 7) the second's;
  // and for int4 the group's scales of this lane's features, two fp16 a word. Both are fetched a block ahead.
  uint4 x[N8], x_next[N8];
  uint32_t sc[8], sc_next[8];
  auto fetch = [&](int blk) {
    const int k = blk * 32 + t * 8;
    const bool live = blk < b1 && k < p.K;
#pragma unroll
    for (int n = 0; n < N8; ++n) {
      const int m = n * 8 + g;
      x_next[n] = live && m < p.o.M ? *reinterpret_cast<const uint4*>(p.X + size_t(m) * p.ldx + k) : make_uint4(0, 0, 0, 0);
    }
    if (kBits == 4) {
      const uint4* s = reinterpret_cast<const uint4*>(p.scales + size_t(blk) * p.scale_ld + col);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint4 v = blk < b1 && col + 8 * (i + 1) <= p.scale_ld ? __ldg(s + i) : make_uint4(0, 0, 0, 0);
        sc_next[4 * i] = v.x; sc_next[4 * i + 1] = v.y; sc_next[4 * i + 2] = v.z; sc_next[4 * i + 3] = v.w;
      }
    }
  };
  fetch(b0);
  int stage = 0;
  uint32_t phase = 0;
  int blk = b0;
  for (; blk < b1; blk += KW) {
#pragma unroll
    for (int n = 0; n < N8; ++n) x[n] = x_next[n];
#pragma unroll
    for (int i = 0; i < 8; ++i) sc[i] = kBits == 4 ? sc_next[i] : 0u;
    fetch(blk + KW);
    if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag, p.st, kTimeoutSmemFull, (9u << 16) | stage))) break;
    // input 8 t + 2 j + b of the block lies in row r = b + 2 t + 8 j of the stage (the order of the box's dimensions), its
    // 16-byte chunks permuted by the TMA swizzle: the chunks that eight lanes read together are on different banks
    const uint32_t slot = smem_u32(ring + stage * S::kStage);
    auto codes_of = [&](int i) {
      const int r = (i & 1) + 2 * t + 8 * (i >> 1);
      return kBits == 8 ? slot + r * 128 + ((g ^ (r & 7)) << 4) : slot + r * 64 + (((g >> 1) ^ t) << 4) + ((g & 1) << 3);
    };
    if (kBits == 8) {
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        uint32_t w[4][kWords];
#pragma unroll
        for (int i = 0; i < 4; ++i) sp_lds(w[i], codes_of(4 * ks + i));
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const int j = (m >> 1) % kWords, e = (m & 1) * 2;  // features 2 m, 2 m + 1: bytes e, e + 1 of word j
          const uint32_t a0 = sp_int8_pair(w[0][j], w[1][j], e), a1 = sp_int8_pair(w[0][j], w[1][j], e + 1);
          const uint32_t a2 = sp_int8_pair(w[2][j], w[3][j], e), a3 = sp_int8_pair(w[2][j], w[3][j], e + 1);
#pragma unroll
          for (int n = 0; n < N8; ++n) sp_mma(acc[m][n], a0, a1, a2, a3, ks ? x[n].z : x[n].x, ks ? x[n].w : x[n].y);
        }
      }
    } else {
      uint32_t w[8][kWords];
#pragma unroll
      for (int i = 0; i < 8; ++i) sp_lds(w[i], codes_of(i));
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        // halves of the words of inputs (k, k + 1): [pair][low or high four features], and their upper bytes moved down
        uint32_t h[4][2], hu[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          h[q][0] = __byte_perm(w[2 * q][j], w[2 * q + 1][j], 0x5410);
          h[q][1] = __byte_perm(w[2 * q][j], w[2 * q + 1][j], 0x7632);
          hu[q][0] = h[q][0] >> 8;
          hu[q][1] = h[q][1] >> 8;
        }
#pragma unroll
        for (int mm = 0; mm < 4; ++mm) {
          const int m = j * 4 + mm, f = 2 * mm, hi = mm >> 1;
          float part[N8][4];
#pragma unroll
          for (int n = 0; n < N8; ++n) part[n][0] = part[n][1] = part[n][2] = part[n][3] = 0.f;
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            const uint32_t lo = h[2 * ks][hi], lou = hu[2 * ks][hi], up = h[2 * ks + 1][hi], upu = hu[2 * ks + 1][hi];
            const uint32_t a0 = sp_int4_pair(lo, lou, f), a1 = sp_int4_pair(lo, lou, f + 1);
            const uint32_t a2 = sp_int4_pair(up, upu, f), a3 = sp_int4_pair(up, upu, f + 1);
#pragma unroll
            for (int n = 0; n < N8; ++n) sp_mma(part[n], a0, a1, a2, a3, ks ? x[n].z : x[n].x, ks ? x[n].w : x[n].y);
          }
          float2 s = __half22float2(*reinterpret_cast<const __half2*>(&sc[m]));
          s.x *= 64.f;
          s.y *= 64.f;
#pragma unroll
          for (int n = 0; n < N8; ++n) {
            acc[m][n][0] = fmaf(part[n][0], s.x, acc[m][n][0]);
            acc[m][n][1] = fmaf(part[n][1], s.x, acc[m][n][1]);
            acc[m][n][2] = fmaf(part[n][2], s.y, acc[m][n][2]);
            acc[m][n][3] = fmaf(part[n][3], s.y, acc[m][n][3]);
          }
        }
      }
    }
    __syncwarp();                                          // every lane has read the stage
    if (lane == 0 && blk + kStages * KW < b1) issue(blk + kStages * KW, stage);
    if (++stage == kStages) { stage = 0; phase ^= 1; }
  }
  if (blk < b1 && lane == 0) {                             // gave up: let the copies in flight land (bounded) before the
    for (int s = 0; s < kStages; ++s) {                    // ring is reused
      const int ahead = s >= stage ? s - stage : s - stage + kStages;
      if (blk + ahead * KW >= b1) continue;
      for (int i = 0; i < (1 << 20); ++i)
        if (mbar_try_wait(&full[s], s >= stage ? phase : phase ^ 1)) break;
    }
  }
  __syncthreads();                                         // nobody uses the ring any more

  // ---- the warps along K, in a fixed tree
  float* buf = reinterpret_cast<float*>(smem);
#pragma unroll
  for (int off = KW / 2; off >= 1; off >>= 1) {
    if (kw >= off && kw < 2 * off) {
      float* dst = buf + size_t((kw - off) * FW + fw) * (S::kAcc * 32) + lane;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < N8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) dst[((m * N8 + n) * 4 + e) * 32] = acc[m][n][e];
    }
    __syncthreads();
    if (kw < off) {
      const float* from = buf + size_t(kw * FW + fw) * (S::kAcc * 32) + lane;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < N8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[m][n][e] += from[((m * N8 + n) * 4 + e) * 32];
    }
    __syncthreads();
  }
  // ---- the CTA's partial tile, [token][feature]
  if (kw == 0) {
#pragma unroll
    for (int m = 0; m < MT; m += 2)
#pragma unroll
      for (int n = 0; n < N8; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          *reinterpret_cast<float4*>(buf + (n * 8 + 2 * t + e) * S::kLd + lf + 2 * m) =
              make_float4(acc[m][n][e], acc[m][n][2 + e], acc[m + 1][n][e], acc[m + 1][n][2 + e]);
  }
  __syncwarp();
  sk_cluster_sync();
  sk_finish<S::F, S::kLd>(p.o, buf, csize, rank, tile, int(threadIdx.x),
                          [&](int, int n) { return kBits == 8 ? __half2float(p.scales[n]) * 64.f : 1.f; });
  __syncwarp();
  sk_cluster_sync();                                       // nobody leaves while a peer may still read its shared memory
}

template <int kBits, int NT, int FW>
static int launch_packed(const void* codes, int ld, SkinnyPackedParams& p, cudaStream_t stream) {
  using S = SkinnyPackedShape<kBits, NT, FW>;
  auto kern = skinny_packed_kernel<kBits, NT, FW>;
  // One CTA per SM as long as the tiles allow it (enforced by its shared memory: left to itself the device packs the CTAs of
  // a cluster two to an SM), split along K over as many CTAs as keep every cluster resident; with more tiles than SMs two
  // CTAs per SM and no split. Measured, 16 tokens, int8, us:
  // 4096 x 4096 (32 tiles) c = 2 / 4 / 8 (two per SM) 11.5 / 9.0 / 10.4; 14336 x 4096 c = 2 / 4 / 8 28.3 / 17.6 / 19.7;
  // 4096 x 28672 (224 tiles) c = 1 / 2 / 4 33 / 38 / 43.
  constexpr int kAlone = S::kTotal > 120 * 1024 ? S::kTotal : 120 * 1024;
  static DeviceOnce configured;
  static std::atomic<int> known[9];
  if (int e = configured.run([&] {
        return int(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kAlone));
      }))
    return e;
  const int tiles = p.o.gate_kind >= 0 ? (p.o.N + S::F / 2 - 1) / (S::F / 2) : (p.o.N + S::F - 1) / S::F;
  int c = skinny_forced_splits();
  if (!c) {
    c = (p.K + 31) / 32 / S::KW;                           // at least one block of inputs per warp
    c = c < 1 ? 1 : (c > 8 ? 8 : c);
    while (c > 1 && skinny_resident_clusters(kern, c, kSpThreads, kAlone, known) < tiles) --c;
  }
  p.csize = c;
  CUtensorMap tmW;
  // rows 8 u + 2 j + b of the weight as dimensions (b, u, j): a box of one block then lands in the order b + 2 u + 8 j
  uint64_t dims[4] = {uint64_t(ld), 2, uint64_t(p.K) / 8, 4};
  uint64_t strides[3] = {uint64_t(ld), uint64_t(ld) * 8, uint64_t(ld) * 2};
  uint32_t box[4] = {uint32_t(S::kRow), 2, 4, 4};
  if (encode_tensor_map(&tmW, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(codes), dims, strides, box,
                        kBits == 8 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B))
    return -10;
  return skinny_launch(kern, tiles * c, c, kSpThreads, tiles * c > sm_count() ? S::kTotal : kAlone, stream, tmW, p);
}

template <int kBits>
static int run_packed(const void* codes, int ld, SkinnyPackedParams& p, cudaStream_t stream) {
  const bool gated = p.o.gate_kind >= 0;
  if (p.o.M <= 8) return gated ? launch_packed<kBits, 8, 2>(codes, ld, p, stream) : launch_packed<kBits, 8, 1>(codes, ld, p, stream);
  return gated ? launch_packed<kBits, 16, 2>(codes, ld, p, stream) : launch_packed<kBits, 16, 1>(codes, ld, p, stream);
}

int skinny_packed_registers(const __nv_bfloat16* X, int ldx, const void* codes, int ld, const __half* scales, int scale_ld,
                            int bits, int K, const SkinnyOut& o, cudaStream_t stream) {
  SkinnyPackedParams p{};
  p.X = X; p.ldx = ldx; p.K = K;
  p.scales = scales; p.scale_ld = scale_ld;
  p.o = o;
  p.st = status_device_ptr();
  return bits == 8 ? run_packed<8>(codes, ld, p, stream) : run_packed<4>(codes, ld, p, stream);
}

}  // namespace idrak
