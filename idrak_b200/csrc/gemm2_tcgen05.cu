// Dense bf16/fp16 GEMM on CTA pairs: two SMs work on one 256 x 256 output tile with tcgen05.mma.cta_group::2.
//
// A cluster of two CTAs is the unit of work. Each CTA loads its own 128 rows of A and its own 128 of the 256 B rows
// (columns of C) per K block - 32 KB per stage instead of the 48 KB a lone CTA needs for a 128 x 256 tile, so every byte
// fetched from L2 feeds 1.5x the FLOPs. The even CTA of the pair (the leader) issues the MMAs; the instruction reads both
// CTAs' shared memory and writes each CTA's half of the accumulator (its 128 rows x 256 columns) into that CTA's TMEM.
//
//   warp 0       TMA producer of the operand ring
//   warp 1       MMA issuer (leader only), TMEM allocation
//   warps 2..9   epilogue arithmetic: two groups of four warps, a thread per row, group g owns 128 of the 256 columns and
//                takes them 64 at a time (a slab)
//   warps 10, 11 one thread per group moves the slabs: it has the residual or saved pre-activation of a slab loaded into
//                one of the group's two 16 KB buffers by TMA while the slab before is worked on, and stores what the
//                arithmetic leaves in the same buffer
// The epilogue is what bounded the products of a training step whose K is short (768: 12 K blocks, 6100 cycles of MMA per
// tile): with residual rows read by the thread that owns them, a load of 64 bytes ahead of its use, and the stores waited for
// by the warps that compute, a tile took 12500 cycles with bias and residual, 13700 with GELU and its derivative, 12000 with
// a factor, 5500 plain. Now 7300, 10000, 6000 and 4300.
//
// Tiles are taken whole, one after another; where the last ones would leave pairs idle they are cut along K into equal
// parts, whose fp32 sums go to the workspace, and pair_reduce_kernel adds the parts in K order and runs the epilogue, so
// the result does not depend on timing.
//
// Barriers (per stage unless noted):
//   full   - in the leader only, count 1: the leader's producer arrives with the byte count of BOTH CTAs' copies; the
//            peer's TMA loads complete their bytes on the leader's barrier (cp.async.bulk.tensor ... cta_group::2 with a
//            shared::cluster barrier address). No load here uses cluster multicast.
//   empty  - in both CTAs, count 1: tcgen05.commit.cta_group::2 with multicast to both CTAs releases the stage in each.
//   tmem_full[2]  - in both CTAs, count 1: multicast commit after the last K block of a tile.
//   tmem_empty[2] - in the leader, count 16: the 8 epilogue warps of each CTA arrive (the peer's remotely).
//   ready[group][buffer]  - count 1: the buffer may be written, or holds the slab's side input
//   filled[group][buffer] - count 4: the group's warps have written their rows of the slab
// Every wait is bounded (two seconds of %globaltimer); a CTA that gives up reports through the status word, waits
// for the copies it issued and still meets its peer at the closing cluster barrier, so neither CTA leaves while the
// other can still touch its shared memory or barriers.
//
// Covers the same reference family as the single-CTA kernel (gemm_tc_{nn,nt,tn,tt}_f32 with bias / GELU / GELU-grad /
// residual epilogues, src/Idrak.Gpu/Cuda/PtxKernels.TensorCore.cs:24-29,80-144) for the large-M products of a
// training step.
#include "gemm_epilogue.cuh"
#include <cstdlib>
#include <cstring>

IDRAK_API int idrak_gemm_pick_splits(int M, int N, int K, int bn);

namespace idrak {

constexpr int kPairBN = 256;        // columns of the pair's tile; each CTA stages half of the B rows
constexpr int kHalfBN = 128;
constexpr int kCutCost = 10, kPartsPerBlock = 7;      // see gemm_pair_plan

struct PairSmem {
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBBytes = kHalfBN * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;       // 32 KB
  static constexpr int kStages = 5;
  static constexpr int kStagingBytes = 4 * 16384;                // two buffers per epilogue group
  static constexpr int kBarrierBytes = 256;
  static constexpr int kTotal = kStages * kStageBytes + kStagingBytes + kBarrierBytes + 1024;
};
static_assert(PairSmem::kTotal <= 232448, "shared memory per CTA");

// ---------------------------------------------------------------------------------------------------------------
// cluster / cta_group::2 wrappers
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_shared_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_addr), "r"(rank));
  return out;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// A tiled load into this CTA's shared memory whose bytes complete on a barrier given by its shared::cluster address
// (the leader's). No multicast: the data lands in the issuing CTA only.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, uint32_t bar_cluster_addr, int c0,
                                                 int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Arrive on the barrier at this shared-memory offset in every CTA of `mask` once the MMAs issued so far are done.
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)),
               "h"(mask)
               : "memory");
}
__device__ __forceinline__ void tc_mma_pair_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                   uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// ---------------------------------------------------------------------------------------------------------------
// work
// ---------------------------------------------------------------------------------------------------------------
// A pair's pieces of work, walked alike by every role: tile, K blocks [kb0, kb1), and where a part goes (-1: whole tile).
// Pieces are counted off: first the tiles that are taken whole, then all the others' first parts, then their second ones, and
// so on, so that pairs at work at the same time contract over the same rows of K and find them in L2.
struct PairWork {
  int m_tiles, n_tiles, k_blocks, pairs, whole, cut, part_blocks;
  int unit, units;
  int tm, tn, kb0, kb1, slot;

  __device__ __forceinline__ PairWork(const GemmParams& p, int pair, int pairs_) {
    m_tiles = p.m_tiles; n_tiles = p.n_tiles; pairs = pairs_;
    k_blocks = (p.K + kBK - 1) / kBK;
    whole = p.whole_tiles;
    cut = m_tiles * n_tiles - whole;
    part_blocks = p.part_blocks;
    unit = pair;
    units = whole + cut * p.parts;
  }
  __device__ __forceinline__ bool next() {
    if (unit >= units) return false;
    int tile = unit, split;
    kb0 = 0;
    kb1 = k_blocks;
    slot = -1;
    if (unit >= whole) {
      slot = unit - whole;
      const int part = slot / cut;
      tile = whole + slot - part * cut;
      kb0 = part * part_blocks;
      kb1 = min(k_blocks, kb0 + part_blocks);
    }
    unit += pairs;
    unit_to_tile_n(m_tiles, n_tiles, tile, tm, tn, split);
    return true;
  }
};

// The slabs that one epilogue group stores, in order: 128 rows x 64 bf16 columns, or 32 fp32 columns of a part.
struct PairJobs {
  PairWork work;
  int group, rank, slab, sub, subs, n;
  bool staged, two, more;
  int kind;                 // 0 the result, 1 what is saved beside it (it comes first), 2 a part
  int row, col;             // first row and column in C, or in the workspace
  bool whole;               // all 64 columns are inside the matrix

  __device__ __forceinline__ PairJobs(const GemmParams& p, int pair, int pairs, int rank_, int group_)
      : work(p, pair, pairs), group(group_), rank(rank_), n(p.N), staged(p.tma_store != 0),
        two(p.act == kActGelu || p.act == kActGeluD) {
    slab = 1;               // the first call of next() takes the first piece of work
    sub = 0;
    subs = 1;
    more = true;
  }
  __device__ __forceinline__ bool next() {
    if (!more) return false;
    if (++sub >= subs) {
      sub = 0;
      ++slab;
      while (slab >= 2 || work.tn * kPairBN + (group * 2 + slab) * 64 >= n || (work.slot < 0 && !staged)) {
        if (!work.next()) { more = false; return false; }
        slab = 0;
      }
      subs = work.slot >= 0 || two ? 2 : 1;
    }
    const int c = (group * 2 + slab) * 64;
    if (work.slot >= 0) {
      kind = 2;
      row = work.slot * 2 * kBM + rank * kBM;
      col = c + sub * 32;
      whole = true;
    } else {
      kind = two && sub == 0 ? 1 : 0;
      row = work.tm * 2 * kBM + rank * kBM;
      col = work.tn * kPairBN + c;
      whole = col + 64 <= n;
    }
    return true;
  }
};

// ---------------------------------------------------------------------------------------------------------------
// the arithmetic of one slab
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float2 pk_fma(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 pk_mul(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 w, x, y;\n\t"
      "mov.b64 {%0, %1}, w;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 pk_add(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 w, x, y;\n\t"
      "mov.b64 {%0, %1}, w;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 pk_dup(float v) { return make_float2(v, v); }
// gelu_tanh and gelu_tanh_both on two values per instruction, with the constants drawn together: with t = tanh(k0 x (1 + k1 x^2)),
// gelu(x) = x (1 + t) / 2 and gelu'(x) = (1 + t) / 2 + x k0 (1 + 3 k1 x^2) (1 - t^2) / 2.
constexpr float kGelu0 = 0.7978845608028654f, kGelu1 = 0.044715f;
__device__ __forceinline__ void pk_gelu_parts(float2 x, float2& x2, float2& t, float2& half) {
  x2 = pk_mul(x, x);
  const float2 u = pk_mul(x, pk_fma(pk_dup(kGelu0 * kGelu1), x2, pk_dup(kGelu0)));
  t = make_float2(tanh_fast(u.x), tanh_fast(u.y));
  half = pk_fma(pk_dup(0.5f), t, pk_dup(0.5f));
}
__device__ __forceinline__ float2 pk_gelu(float2 x) {
  float2 x2, t, half;
  pk_gelu_parts(x, x2, t, half);
  return pk_mul(x, half);
}
__device__ __forceinline__ void pk_gelu_both(float2 x, float2& g, float2& d) {
  float2 x2, t, half;
  pk_gelu_parts(x, x2, t, half);
  g = pk_mul(x, half);
  const float2 du = pk_mul(x, pk_fma(pk_dup(-1.5f * kGelu0 * kGelu1), x2, pk_dup(-0.5f * kGelu0)));
  d = pk_fma(du, pk_fma(t, t, pk_dup(-1.0f)), half);
}

// 64 columns of a thread's row: accumulators -> bf16 in the slab's buffer, whose 16-byte pieces hold the side input where
// there is one (a thread reads and overwrites its own row only). ACT == kActGelu / kActGeluD: what is saved goes to the
// buffer and `value` keeps the packed result for the next one. The loads of four pieces go out together: one after the other
// their latencies were most of a slab's time (bias and residual: 2300 of 3700 cycles).
template <bool BIAS, int ACT, bool RES>
__device__ __forceinline__ void slab_math(const GemmParams& p, int col0, const uint32_t (&acc)[64], uint8_t* buf, int r,
                                          uint32_t (&value)[32]) {
  constexpr bool kSide = RES || ACT == kActGeluGrad || ACT == kActMulAux;
  const float2 alpha = pk_dup(p.alpha);
  uint8_t* row = buf + r * 128;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint4 sides[4], biases[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (kSide) sides[q] = *reinterpret_cast<const uint4*>(row + (((h * 4 + q) ^ (r & 7)) << 4));
      if (BIAS) biases[q] = __ldg(reinterpret_cast<const uint4*>(p.bias + col0 + (h * 4 + q) * 8));
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int g = h * 4 + q;
      const uint32_t side[4] = {sides[q].x, sides[q].y, sides[q].z, sides[q].w};
      const uint32_t b[4] = {biases[q].x, biases[q].y, biases[q].z, biases[q].w};
      uint32_t o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = make_float2(__uint_as_float(acc[g * 8 + 2 * i]), __uint_as_float(acc[g * 8 + 2 * i + 1]));
        float2 v = BIAS ? pk_fma(a, alpha, unpack_bf16x2(b[i])) : pk_mul(a, alpha);
        if (ACT == kActGeluGrad) {
          const float2 x = unpack_bf16x2(side[i]);
          v = pk_mul(v, make_float2(gelu_tanh_grad(x.x), gelu_tanh_grad(x.y)));
        } else if (ACT == kActMulAux) {
          v = pk_mul(v, unpack_bf16x2(side[i]));
        } else if (ACT == kActGelu) {
          // the activation sees the value as it is stored, so forward and backward agree
          o[i] = pack_bf16x2(v.x, v.y);
          const float2 y = pk_gelu(unpack_bf16x2(o[i]));
          value[g * 4 + i] = pack_bf16x2(y.x, y.y);
        } else if (ACT == kActGeluD) {
          float2 y, d;
          pk_gelu_both(v, y, d);
          o[i] = pack_bf16x2(d.x, d.y);
          value[g * 4 + i] = pack_bf16x2(y.x, y.y);
        }
        if (RES) v = pk_add(v, unpack_bf16x2(side[i]));
        if (ACT != kActGelu && ACT != kActGeluD) o[i] = pack_bf16x2(v.x, v.y);
      }
      *reinterpret_cast<uint4*>(row + ((g ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// The same with every test at run time (a ragged column edge, column factors, operands between 16-byte boundaries); the side
// input is read from global memory.
__device__ __forceinline__ void slab_generic(const GemmParams& p, int row, int col0, const uint32_t (&acc)[64], uint8_t* buf,
                                             int r, uint32_t (&value)[32]) {
  const bool two = p.act == kActGelu || p.act == kActGeluD;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    const int col = col0 + g * 8;
    float v[8], pre[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { v[i] = __uint_as_float(acc[g * 8 + i]) * p.alpha; pre[i] = 0.f; }
    if (row < p.M && col < p.N) epilogue_math8(p, row, col, v, min(8, p.N - col), false, pre);
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      value[g * 4 + i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
      o[i] = two ? pack_bf16x2(pre[2 * i], pre[2 * i + 1]) : value[g * 4 + i];
    }
    *reinterpret_cast<uint4*>(buf + r * 128 + ((g ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// the kernel: grid = 2 x pairs, cluster (2, 1, 1)
// ---------------------------------------------------------------------------------------------------------------
constexpr int kPairThreads = 64 + 32 * kEpiWarps + 64;

template <int A_MN, int B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmAux,
                 const __grid_constant__ CUtensorMap tmSide, const __grid_constant__ CUtensorMap tmPart, const GemmParams p) {
  using L = PairSmem;
  constexpr int kStages = L::kStages;
  constexpr int BN = kPairBN;
  extern __shared__ uint8_t smem_raw[];
  // the same offsets in both CTAs: the MMA applies one descriptor to both
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + kStages * L::kStageBytes;        // [group][buffer] of 16 KB
  uint8_t* bar_base = staging + L::kStagingBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(bar_base);
  uint64_t* empty = full + kStages;
  uint64_t* tmem_full = empty + kStages;
  uint64_t* tmem_empty = tmem_full + 2;
  uint64_t* ready = tmem_empty + 2;                          // [group * 2 + buffer]
  uint64_t* filled = ready + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(filled + 4);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();          // 0 = leader
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;
  const int pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 2 * kEpiWarps);
    }
    for (int b = 0; b < 4; ++b) {
      mbar_init(&ready[b], 1);
      mbar_init(&filled[b], 4);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 2 * BN);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  // both CTAs have their barriers and TMEM before either signals the other
  cluster_arrive();
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();                           // what follows may take an SM as soon as it is free
  pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (one per CTA)
    if (lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      PairWork w(p, pair, pairs);
      while (ok && w.next()) {
        const int row0 = w.tm * 2 * kBM + int(rank) * kBM;        // this CTA's rows of A
        const int col0 = w.tn * BN + int(rank) * kHalfBN;         // this CTA's rows of B
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.st, kTimeoutSmemEmpty, (2u << 16) | stage)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * L::kStageBytes;
          uint8_t* sb = sa + L::kABytes;
          const uint32_t bar = map_shared_to_cta(smem_u32(&full[stage]), 0);
          if (leader) mbar_expect_tx(&full[stage], 2 * L::kStageBytes);
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < kBM / 64; ++j) tma_load_2d_pair(sa + j * 8192, &tmA, bar, row0 + j * 64, kb * kBK);
          } else {
            tma_load_2d_pair(sa, &tmA, bar, kb * kBK, row0);
          }
          if (B_MN) {
#pragma unroll
            for (int j = 0; j < kHalfBN / 64; ++j) tma_load_2d_pair(sb + j * 8192, &tmB, bar, col0 + j * 64, kb * kBK);
          } else {
            tma_load_2d_pair(sb, &tmB, bar, kb * kBK, col0);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok || *abort_flag) {
        // the copies this CTA issued complete on the leader's barrier, which the peer cannot poll: give them time to
        // land (they take microseconds) before the closing barrier lets shared memory go
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) { }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && lane == 0) {
      constexpr uint32_t idesc = make_idesc_f16(2 * kBM, BN, A_MN, B_MN, 1);
      int stage = 0;
      uint32_t phase = 0;
      int local = 0;
      bool ok = true;
      unsigned long long t_acc = 0, t_ops = 0;
      const long long t_begin = p.prof ? clock64() : 0;
      PairWork w(p, pair, pairs);
      for (; ok && w.next(); ++local) {
        const int buf = local & 1;
        const uint32_t acc_phase = (local >> 1) & 1;
        const long long c0 = p.prof ? clock64() : 0;
        if (!mbar_wait(&tmem_empty[buf], acc_phase ^ 1, abort_flag, p.st, kTimeoutTmemEmpty, (2u << 16) | buf)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (p.prof) t_acc += (unsigned long long)(clock64() - c0);
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          const long long c2 = p.prof ? clock64() : 0;
          if (!mbar_wait(&full[stage], phase, abort_flag, p.st, kTimeoutSmemFull, (2u << 16) | stage)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (p.prof) t_ops += (unsigned long long)(clock64() - c2);
          const uint32_t sa = smem_u32(smem + stage * L::kStageBytes);
          const uint32_t sb = sa + L::kABytes;
#pragma unroll
          for (int kk = 0; kk < kBK / kUmmaK; ++kk) {
            const uint64_t da = A_MN ? make_smem_desc_sw128(sa + kk * 2048, 8192, 1024)
                                     : make_smem_desc_sw128(sa + kk * 32, 16, 1024);
            const uint64_t db = B_MN ? make_smem_desc_sw128(sb + kk * 2048, 8192, 1024)
                                     : make_smem_desc_sw128(sb + kk * 32, 16, 1024);
            tc_mma_pair_f16_ss(d_tmem, da, db, idesc, (kb > w.kb0 || kk > 0) ? 1u : 0u);
          }
          tc_commit_pair(&empty[stage], 0x3);     // both CTAs may refill the stage once these MMAs have read it
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if (ok) tc_commit_pair(&tmem_full[buf], 0x3);
      }
      if (p.prof) {
        p.prof[blockIdx.x * 8 + 0] = (unsigned long long)(clock64() - t_begin);
        p.prof[blockIdx.x * 8 + 1] = t_acc;
        p.prof[blockIdx.x * 8 + 2] = t_ops;
      }
    }
  } else if (warp < 2 + kEpiWarps) {
    // ------------------------------------------------------------------ epilogue arithmetic (8 warps, this CTA's 128 rows)
    const int quarter = warp & 3;                            // the TMEM lanes this warp may read
    const int group = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t empty_bar_leader[2] = {map_shared_to_cta(smem_u32(&tmem_empty[0]), 0),
                                          map_shared_to_cta(smem_u32(&tmem_empty[1]), 0)};
    int local = 0, job = 0;
    bool ok = true;
    unsigned long long t_wait = 0, t_busy = 0;
    // the group's next buffer, once it may be written
    auto take = [&]() -> uint8_t* {
      const int b = job & 1;
      if (!mbar_wait(&ready[group * 2 + b], uint32_t(job >> 1) & 1u, abort_flag, p.st, kTimeoutGeneric, (2u << 16) | (20 + b)))
        ok = false;
      return staging + (group * 2 + b) * 16384;
    };
    auto give = [&]() {
      fence_proxy_async_smem();                              // the rows were written by ordinary stores, TMA reads them
      __syncwarp();
      if (lane == 0) mbar_arrive(&filled[group * 2 + (job & 1)]);
      ++job;
    };
    PairWork w(p, pair, pairs);
    for (; ok && w.next(); ++local) {
      const int buf = local & 1;
      const uint32_t acc_phase = (local >> 1) & 1;
      const long long c0 = p.prof ? clock64() : 0;
      if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full[buf], acc_phase, abort_flag, p.st, kTimeoutTmemFull, (2u << 16) | buf))) break;
      tc_fence_after();
      const long long c1 = p.prof ? clock64() : 0;
      const uint32_t acc_addr = tmem_base + buf * BN + (uint32_t(quarter * 32) << 16);
      const int row = w.tm * 2 * kBM + int(rank) * kBM + r;
      const int n0 = w.tn * BN;
      bool released = false;
      // this CTA's half of the accumulator is free once read: tell the leader's MMA warp
      auto release = [&]() {
        tc_fence_before();
        if (lane == 0) {
          if (leader) mbar_arrive(&tmem_empty[buf]);
          else mbar_arrive_cluster(empty_bar_leader[buf]);
        }
        released = true;
      };
#pragma unroll 1
      for (int j = 0; j < 2; ++j) {
        const int cslab = group * 2 + j;
        const int col0 = n0 + cslab * 64;
        if (col0 >= p.N) break;                              // uniform over the group
        uint32_t acc[64];
        tmem_ld_32x32b_x64(acc_addr + cslab * 64, acc);
        tmem_ld_wait();
        if (j == 1 || col0 + 64 >= p.N) release();
        if (w.slot >= 0) {
          // a part: fp32, 32 columns per buffer
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint8_t* b = take();
            if (ok) {
#pragma unroll
              for (int c = 0; c < 8; ++c)
                *reinterpret_cast<uint4*>(b + r * 128 + ((c ^ (r & 7)) << 4)) =
                    make_uint4(acc[h * 32 + 4 * c], acc[h * 32 + 4 * c + 1], acc[h * 32 + 4 * c + 2], acc[h * 32 + 4 * c + 3]);
            }
            give();
          }
        } else if (p.tma_store) {
          uint32_t value[32];
          uint8_t* b = take();
          if (ok) {
            switch (col0 + 64 <= p.N ? p.epi_mode : kEpiGeneric) {     // uniform over the group
              case kEpiPlain:     slab_math<false, kActNone, false>(p, col0, acc, b, r, value); break;
              case kEpiBias:      slab_math<true, kActNone, false>(p, col0, acc, b, r, value); break;
              case kEpiBiasRes:   slab_math<true, kActNone, true>(p, col0, acc, b, r, value); break;
              case kEpiRes:       slab_math<false, kActNone, true>(p, col0, acc, b, r, value); break;
              case kEpiBiasGelu:  slab_math<true, kActGelu, false>(p, col0, acc, b, r, value); break;
              case kEpiGelu:      slab_math<false, kActGelu, false>(p, col0, acc, b, r, value); break;
              case kEpiGeluGrad:  slab_math<false, kActGeluGrad, false>(p, col0, acc, b, r, value); break;
              case kEpiBiasGeluD: slab_math<true, kActGeluD, false>(p, col0, acc, b, r, value); break;
              case kEpiGeluD:     slab_math<false, kActGeluD, false>(p, col0, acc, b, r, value); break;
              case kEpiMulAux:    slab_math<false, kActMulAux, false>(p, col0, acc, b, r, value); break;
              default:            slab_generic(p, row, col0, acc, b, r, value); break;
            }
          }
          give();
          if (p.act == kActGelu || p.act == kActGeluD) {
            b = take();
            if (ok) {
#pragma unroll
              for (int c = 0; c < 8; ++c)
                *reinterpret_cast<uint4*>(b + r * 128 + ((c ^ (r & 7)) << 4)) =
                    make_uint4(value[4 * c], value[4 * c + 1], value[4 * c + 2], value[4 * c + 3]);
            }
            give();
          }
        } else if (row < p.M) {
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const int col = col0 + g * 8;
            if (col < p.N) {
              float v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(acc[g * 8 + i]) * p.alpha;
              epilogue8(p, row, col, v, min(8, p.N - col));
            }
          }
        }
        __syncwarp();
      }
      if (!released) release();
      ok = __all_sync(0xffffffffu, ok);
      if (p.prof) {
        t_wait += (unsigned long long)(c1 - c0);
        t_busy += (unsigned long long)(clock64() - c1);
      }
    }
    if (p.prof && warp == 2 && lane == 0) {
      p.prof[blockIdx.x * 8 + 4] = t_wait;
      p.prof[blockIdx.x * 8 + 5] = t_busy;
      p.prof[blockIdx.x * 8 + 6] = (unsigned long long)local;
    }
  } else if (lane == 0) {
    // ------------------------------------------------------------------ slabs in and out (one thread per group)
    const int group = warp - 2 - kEpiWarps;
    const bool has_side = mode_has_side(p.epi_mode);
    uint8_t* bufs = staging + group * 2 * 16384;
    PairJobs stores(p, pair, pairs, int(rank), group), ahead(p, pair, pairs, int(rank), group);
    // buffer b becomes job `ahead`'s: its side input is on the way, or it may be written at once
    auto arm = [&](int b) {
      if (!ahead.next()) return;
      if (has_side && ahead.kind == 0 && ahead.whole) {
        mbar_expect_tx(&ready[group * 2 + b], 16384);
        tma_load_2d(bufs + b * 16384, &tmSide, &ready[group * 2 + b], ahead.col, ahead.row);
      } else {
        mbar_arrive(&ready[group * 2 + b]);
      }
    };
    arm(0);
    arm(1);
    bool ok = true;
    for (int job = 0; stores.next(); ++job) {
      const int b = job & 1;
      if (!mbar_wait(&filled[group * 2 + b], uint32_t(job >> 1) & 1u, abort_flag, p.st, kTimeoutGeneric, (2u << 16) | (24 + b))) {
        ok = false;
        break;
      }
      if (stores.kind == 2) tma_store_2d(&tmPart, bufs + b * 16384, stores.col, stores.row);
      else if (stores.row < p.M) tma_store_2d(stores.kind ? &tmAux : &tmC, bufs + b * 16384, stores.col, stores.row);
      tma_store_commit();
      tma_store_wait_read<0>();                              // this thread has nothing else to do meanwhile
      arm(b);
    }
    tma_store_wait<0>();
    if (!ok || *abort_flag) {
      const uint64_t t0 = global_timer_ns();                 // side inputs on their way must land before the CTA leaves
      while (global_timer_ns() - t0 < 200000ull) { }
    }
  }

  tc_fence_before();
  __syncthreads();
  // neither CTA leaves (or frees TMEM) while the other may still signal it or have MMAs reading its shared memory
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * BN);
  }
}

// Adds the parts of the tiles that were cut, in K order, and runs the epilogue. A block takes 8 rows of a tile, a thread 8
// columns of one of them; four parts are in flight at a time.
__global__ void __launch_bounds__(256) pair_reduce_kernel(const GemmParams p) {
  pdl_wait();
  const int cut = p.m_tiles * p.n_tiles - p.whole_tiles;
  const int i = blockIdx.x >> 5;
  int tm, tn, split;
  unit_to_tile_n(p.m_tiles, p.n_tiles, p.whole_tiles + i, tm, tn, split);
  const int c = (threadIdx.x & 31) * 8, col = tn * kPairBN + c;
  const int r = (blockIdx.x & 31) * 8 + (threadIdx.x >> 5), row = tm * 2 * kBM + r;
  if (row >= p.M || col >= p.N) return;
  const float* src = p.workspace + (size_t(i) * 2 * kBM + r) * kPairBN + c;
  const size_t step = size_t(cut) * 2 * kBM * kPairBN;
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = 0.f;
  for (int q = 0; q < p.parts; q += 4) {
    float4 x[4], y[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4* at = reinterpret_cast<const float4*>(src + (q + k) * step);
      x[k] = q + k < p.parts ? at[0] : make_float4(0.f, 0.f, 0.f, 0.f);
      y[k] = q + k < p.parts ? at[1] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[0] += x[k].x; v[1] += x[k].y; v[2] += x[k].z; v[3] += x[k].w;
      v[4] += y[k].x; v[5] += y[k].y; v[6] += y[k].z; v[7] += y[k].w;
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] *= p.alpha;
  epilogue8(p, row, col, v, min(8, p.N - col));
}

template <int A_MN, int B_MN>
static int launch_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const CUtensorMap& tmAux,
                       const CUtensorMap& tmSide, const CUtensorMap& tmPart, const GemmParams& p, int grid, cudaStream_t stream) {
  auto kern = gemm_pair_kernel<A_MN, B_MN>;
  static DeviceOnce configured;
  if (int e = configured.run([&] {
        return int(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem::kTotal));
      }))
    return e;
  int rc = launch_overlapped(kern, dim3(unsigned(grid)), kPairThreads, PairSmem::kTotal, stream, tmA, tmB, tmC, tmAux, tmSide, tmPart, p);
  const int cut = p.m_tiles * p.n_tiles - p.whole_tiles;
  if (rc == 0 && cut) rc = launch_overlapped(pair_reduce_kernel, dim3(unsigned(cut * 32)), 256, 0, stream, p);
  return rc;
}

static int pair_operand_map(CUtensorMap* tm, const void* ptr, int mn_extent, int k_extent, int ld, int mn_major, int fp16) {
  uint64_t dims[2], strides[1];
  uint32_t box[2];
  if (mn_major) {
    dims[0] = uint64_t(mn_extent); dims[1] = uint64_t(k_extent);
    box[0] = 64; box[1] = kBK;
  } else {
    dims[0] = uint64_t(k_extent); dims[1] = uint64_t(mn_extent);
    box[0] = kBK; box[1] = 128;
  }
  strides[0] = uint64_t(ld) * 2;
  return encode_tensor_map(tm, fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                           const_cast<void*>(ptr), dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

static int pair_env() {
  static int enabled = -1;
  if (enabled < 0) {
    const char* e = getenv("IDRAK_GEMM_PAIR");
    enabled = (e == nullptr) ? 1 : (e[0] == '0' ? 0 : (e[0] == '2' ? 2 : 1));     // 0 off, 1 where it measured faster, 2 wherever it can run
  }
  return enabled;
}

// Where a product of this size goes, and how its K is cut (`may_cut`: parts may be used). Costs are in K blocks of a wave (0.4 us);
// the figures are us, back to back, single CTAs / pairs:
//  - Of as many waves (128 x 256 on each SM, 256 x 256 on each two) pairs are 8 % faster, operands come from L2 once for 256 rows:
//    3000 x 28672 x 4096 527 / 491; a wave alone is a tie (2997 x 1024 x 1024 12.8 / 13.8, with a residual 15.4 / 14.6; the training step
//    that it is from takes 3303 with the one and 3264 with the other). But an odd number of 128 rows costs pairs a tile more, and where
//    that is a wave more single CTAs win: 300 x 28672 x 4096 88 / 104, 520 rows 118 / 131, 1030 rows 198 / 209, 1030 x 4096 x 4096 31 / 45,
//    x 14336 97 / 111; not 2100 x 28672 x 4096, 13 waves and 14, 383 / 368.
//  - The last tiles in parts along K, where they leave pairs idle: kCutCost for the second kernel and the fp32 parts through L2, of
//    which kPartsPerBlock take as long as a block. Whole and cut: 1500 x 4096 x 4096 54.0, 47.4, x 14336 163, 133; weight gradients over
//    16384 rows of 768 x 768 90, 29, of 3072 x 768 98, 64; not cut is 1030 x 6144 x 4096 (two rounds of parts, 55).
//  - Where all tiles are cut, single CTAs may have fewer to cut: 300 x 4096 x 4096 23.0 / 25.8, x 14336 50 / 56; 512 rows 27.1 / 26.5.
PairPlan gemm_pair_plan(int M, int N, int K, bool may_cut) {
  const int sms = sm_count(), pairs = sms / 2, kb = (K + kBK - 1) / kBK;
  PairPlan plan{false, 0, 1, 0, may_cut ? idrak_gemm_pick_splits(M, N, K, N <= 128 ? 128 : 256) : 1};
  const int enabled = pair_env();
  if (!enabled || M <= 128 || N < 256 || K < 128) return plan;
  const long long tiles = (long long)((M + 255) / 256) * ((N + 255) / 256);
  if (tiles > (1 << 24)) return plan;
  const long long units = (long long)((M + 127) / 128) * ((N + 255) / 256), waves = (tiles + pairs - 1) / pairs;
  plan.whole = int(tiles);
  plan.part_blocks = kb;
  plan.use = enabled == 2 || 2 * tiles >= pairs;
  const long long single_waves = (units + sms - 1) / sms;
  if (enabled == 1 && plan.use && single_waves < waves && single_waves * 1.085f * kb < waves * kb + 5.f) {
    plan.use = false;
    plan.splits = 1;
    return plan;
  }
  const int full = int(tiles / pairs) * pairs, cut = int(tiles) - full;
  if (!may_cut || cut == 0) return plan;
  // the last tiles whole, or in parts taken in `rounds` rounds
  int best = kb;
  for (int rounds = 1; rounds <= 4; ++rounds) {
    int parts = rounds * pairs / cut;
    if (parts < 2 || parts > kb) continue;
    const int blocks = (kb + parts - 1) / parts;
    parts = (kb + blocks - 1) / blocks;
    const int cost = rounds * blocks + kCutCost + cut * parts / kPartsPerBlock;
    if (cost < best) {
      best = cost;
      plan.use = true;
      plan.whole = full;
      plan.parts = parts;
      plan.part_blocks = blocks;
    }
  }
  const int s = plan.splits;
  if (enabled == 1 && plan.parts > 1 && full == 0 && s > 1 && 1.085f * ((kb + s - 1) / s) + 12.f + float(units * s / 2 / kPartsPerBlock) < best) {
    plan.use = false;
    plan.parts = 1;
  }
  return plan;
}
long long gemm_pair_workspace(const PairPlan& plan, int M, int N) {
  const long long cut = (long long)((M + 255) / 256) * ((N + 255) / 256) - plan.whole;
  return plan.use ? cut * plan.parts * 2 * kBM * kPairBN : 0;
}

// Same contract as the single-CTA launcher; `p` arrives filled except for the tile counts. tmC / tmAux are the store maps
// (box 64 x 128) made by the caller.
int gemm_pair_launch(const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, const CUtensorMap& tmC,
                     const CUtensorMap& tmAux, GemmParams p, int fp16, const PairPlan& plan, cudaStream_t stream) {
  CUtensorMap tmA, tmB, tmSide, tmPart;
  memset(&tmSide, 0, sizeof(tmSide));
  memset(&tmPart, 0, sizeof(tmPart));
  if (pair_operand_map(&tmA, A, p.M, p.K, lda, a_mn, fp16)) return -11;
  if (pair_operand_map(&tmB, B, p.N, p.K, ldb, b_mn, fp16)) return -12;
  if (p.tma_store && mode_has_side(p.epi_mode)) {
    const bool aux = mode_side_is_aux(p.epi_mode);
    const int ld = aux ? p.ld_aux : p.ldr;
    uint64_t dims[2] = {uint64_t(p.N), uint64_t(p.M)}, strides[1] = {uint64_t(ld) * 2};
    uint32_t box[2] = {64, 128};
    // rows that overlap (a broadcast residual) are read by the threads
    if (ld < p.N || encode_tensor_map(&tmSide, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, aux ? p.aux : const_cast<__nv_bfloat16*>(p.residual),
                                      dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
      p.epi_mode = kEpiGeneric;
  }
  p.m_tiles = (p.M + 2 * kBM - 1) / (2 * kBM);
  p.n_tiles = (p.N + kPairBN - 1) / kPairBN;
  p.splits = 1;
  p.whole_tiles = plan.whole;
  p.parts = plan.parts;
  p.part_blocks = plan.part_blocks;
  const int cut = p.m_tiles * p.n_tiles - p.whole_tiles;
  const int pairs = min(p.whole_tiles + cut * p.parts, sm_count() / 2);
  if (cut) {
    uint64_t dims[2] = {uint64_t(kPairBN), uint64_t(cut) * p.parts * 2 * kBM}, strides[1] = {kPairBN * 4};
    uint32_t box[2] = {32, 128};
    if (encode_tensor_map(&tmPart, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.workspace, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
      return -13;
  }
  const int grid = 2 * pairs;
  if (!a_mn && !b_mn) return launch_pair<0, 0>(tmA, tmB, tmC, tmAux, tmSide, tmPart, p, grid, stream);
  if (!a_mn && b_mn) return launch_pair<0, 1>(tmA, tmB, tmC, tmAux, tmSide, tmPart, p, grid, stream);
  if (a_mn && !b_mn) return launch_pair<1, 0>(tmA, tmB, tmC, tmAux, tmSide, tmPart, p, grid, stream);
  return launch_pair<1, 1>(tmA, tmB, tmC, tmAux, tmSide, tmPart, p, grid, stream);
}

}  // namespace idrak
