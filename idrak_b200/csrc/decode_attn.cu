// Decode-time attention over a block-table ("paged") KV cache, and the kernel that writes new keys / values
// into it.
//
// Cache layout: k_cache, v_cache = [num_blocks, block_size, kv_heads, head_dim] bf16; a sequence's blocks are
// listed in block_table[seq, :]; token t of a sequence lives in block block_table[seq, t / block_size] at
// offset t % block_size.
//
// paged_decode_kernel: grid (sequences, kv heads, splits). One CTA serves the G = heads / kv_heads query heads that share a
// KV head over one share of the sequence's keys. Its four warps each walk tiles of 16 keys through a ring of their own: the
// tile's rows arrive by TMA (a box of up to 16 consecutive slots of one cache block, one head), several tiles ahead, and a warp
// waits for nothing but its next tile. The warp takes both products transposed, so that the keys (S^T = K Q^T) and the head's
// elements (O^T = V^T P^T) fill the 16 rows of a warp-level m16n8k16 MMA and the query heads its 8 columns; P^T is turned from
// the layout of a result into that of an operand by four byte-matrix moves. With the query heads as the 16 rows - 4 of them in
// use where 32 heads share 8 - a tile of 32 keys took 1780 instructions, half of them copies a lane at a time, and the kernel was
// bound by issuing them; it is about 600 now, and the keys and values on their way bound it. Warp-level MMAs are enough: tcgen05's
// 128 rows have nothing to fill them.
//
// int8 cache: the codes enter the tensor core as exact bf16 numbers (code / 64), converted in registers on their way from
// shared memory: a lane takes 16 codes of a key at once, and since a sum over d has no order of its own the query operand is laid
// out to match; values come transposed two codes at a time and their even and odd elements form the two halves of a fragment. A
// key's scale multiplies its scores and a value's scale its probability in fp32 before the rounding to bf16.
//
// Measured, us (32 query heads on 8, head size 128): 64 sequences of 128 to 2304 tokens (386 MB) 92
// before and 77 now; 150 of 128 to 1024, int8 cache (198 MB) 91 and 54; one of 8000 20.2 and 16.1; 16 of 16 to 60 8.2 and 5.4.
//
// The host knows only a bound on the lengths, so a share is at least `min_tiles` tiles and a sequence uses as many of the
// splits as its own length fills; the other CTAs leave at once, and a sequence with one share is written out directly. Splits
// write (max, sum, partial output) and decode_merge_kernel combines them in split order.
//
// Reference counterparts: attention_decode_{f32,int8,bf16} (split over blocks, last block merges;
// src/Idrak.Gpu/Cuda/PtxKernels.Rows.cs:2047-2060), kv_write_{f32,bf16} (PtxKernels.Decoding.cs:12),
// KeyValuePages (src/Idrak.Abstraction/Generation/KeyValuePages.cs:20-34) whose pages the reference copies into a
// contiguous cache instead of attending over them in place.
#include "common.cuh"

namespace idrak {

constexpr int kDecWarps = 4;
constexpr int kDecTile = 16;       // keys per warp tile
constexpr int kDecMaxGroup = 16;   // query heads per KV head

struct DecodeParams {
  const __nv_bfloat16* q;        // [seqs, H, D], sequences q_stride elements apart
  long long q_stride;
  const __nv_bfloat16* k_cache;  // bf16 cache; with an int8 cache these point at int8 codes [blocks, block_size, Hkv, D]
  const __nv_bfloat16* v_cache;
  const float* k_scale;          // int8 cache: one scale per (slot, kv head), [blocks * block_size, Hkv]
  const float* v_scale;
  const int* block_table;        // [seqs, max_blocks]
  const int* seq_lens;           // [seqs]
  __nv_bfloat16* out;            // [seqs, H, D]
  float* partial;                // [seqs, H, splits, D + 2]
  int H, Hkv, D, block_size, max_blocks, splits;
  int min_tiles;                 // tiles per split at least
  float scale_log2;
  int window;                    // 0 = full; else attend to the last `window` positions only
  int box_log2;                  // slots that one copy brings: the largest power of two up to 16 that divides block_size
  Status* st;
};

// ---- warp-level tensor-core pieces (mma.sync m16n8k16, bf16 in, fp32 accumulate)
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t smem_row) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_row) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t smem_row) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_row) : "memory");
}
// an 8 x 8 matrix of 16-bit elements, a row per four lanes, transposed across the warp
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// 2^x, results below the smallest normal number flushed: the library's routine spends instructions on those.
__device__ __forceinline__ float dec_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two int8 codes (biased by 128, in the low bytes of the two halves) -> two bf16 values code / 64, exactly: an unsigned integer
// u < 256 in a 16-bit lane is, read as bf16, u * 2^-133, and one fused multiply-add takes it to (u - 128) / 64.
__device__ __forceinline__ uint32_t codes_pair(uint32_t t) {
  const uint32_t mul = 0x7F007F00u, add = 0xC000C000u;      // 2^127, -128 / 64
  const __nv_bfloat162 v = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&t), *reinterpret_cast<const __nv_bfloat162*>(&mul),
                                   *reinterpret_cast<const __nv_bfloat162*>(&add));
  return *reinterpret_cast<const uint32_t*>(&v);
}

// The share of a sequence's tiles that each split takes, and how many splits that leaves with work.
__device__ __forceinline__ int tiles_per_split(int span, int splits, int min_tiles) {
  return max(min_tiles, (span + splits - 1) / splits);
}
__device__ __forceinline__ void key_span(int len, int window, int& first_tile, int& span) {
  const int first_pos = (window > 0 && len > window) ? len - window : 0;
  first_tile = first_pos / kDecTile;
  span = (len + kDecTile - 1) / kDecTile - first_tile;
}

// A tile of keys or values in shared memory: 16 rows, in column blocks of up to 128 bytes as TMA writes them; with SWIZZLE the
// 16-byte pieces of a row are exchanged by the row's place in the pattern, so that the eight rows of a matrix load touch all banks.
template <int D, int KV8, bool SWIZZLE>
struct DecTile {
  static constexpr int kRowBytes = KV8 ? D : 2 * D;
  static constexpr int kBlock = kRowBytes < 128 ? kRowBytes : 128;       // bytes of a row in a column block
  static constexpr int kPitch = SWIZZLE ? kBlock : 128;                  // a copy's place starts at a multiple of 128 bytes
  static constexpr int kBlocks = kRowBytes / kBlock;
  static constexpr int kBytes = kDecTile * kPitch * kBlocks;
  static constexpr int kStage = 2 * kBytes;
  // Of a warp: three CTAs share an SM over a bf16 cache of head size 128, four otherwise. us, 64 sequences of 128 to 2304 keys /
  // 64 of 1000 / 16 of 128 to 2304: 16 KB 76.8 / 58.4 / 23.1, 24 KB and two CTAs 79.9 / 55.3 / 27.0; 150 of 128 to 1024, int8: 12 KB
  // 53.9, 16 KB and three CTAs 59.4, 24 KB 69.6; 32 of 500 to 600, 12 heads of 64: 14.8, 15.1, 19.7.
  static constexpr int kRing = !KV8 && D == 128 ? 16384 : 12288;
  static constexpr int kStages = kRing / kStage;
  static __device__ __forceinline__ uint32_t at(int row, int piece) {
    constexpr int kPieces = kBlock / 16;
    const int c = piece % kPieces;
    const int x = !SWIZZLE ? c : kBlock == 128 ? c ^ (row & 7) : c ^ ((row >> 1) & 3);
    return uint32_t((piece / kPieces) * kDecTile * kPitch + row * kPitch + x * 16);
  }
};

// NH: column tiles of 8 query heads. SWIZZLE: the boxes have 8 rows or more (a smaller block size is taken unswizzled, row groups
// of fewer rows would not start where the pattern does).
template <int D, int KV8, int NH, bool SWIZZLE>
__global__ void __launch_bounds__(kDecWarps * 32)
paged_decode_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const DecodeParams p) {
  using T = DecTile<D, KV8, SWIZZLE>;
  constexpr int S = T::kStages;
  constexpr int KS = D / 16;                             // steps of K Q^T over d, and row tiles of O^T
  extern __shared__ uint8_t dsm_raw[];
  uint8_t* dsm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dsm_raw) + 1023) & ~uintptr_t(1023));
  const int seq = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
  const int G = p.H / p.Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;                // row and column pair of this lane in an MMA fragment
  uint8_t* ring = dsm + warp * T::kRing;                 // [stage][K, V]
  uint64_t* full = reinterpret_cast<uint64_t*>(dsm + kDecWarps * T::kRing) + warp * S;
  float* scales = reinterpret_cast<float*>(dsm + kDecWarps * T::kRing + kDecWarps * S * 8) + warp * S * 32;   // int8: [stage][K, V][16]
  volatile uint32_t* abort_flag = reinterpret_cast<uint32_t*>(dsm + kDecWarps * T::kRing + kDecWarps * S * (8 + 128));
  // the warps' partial outputs are merged in the place of the tiles once every warp is done with them
  float* smerge = reinterpret_cast<float*>(dsm);

  pdl_launch_dependents();     // a dependent launched programmatically may set itself up while this kernel runs
  if (lane == 0) {
    for (int i = 0; i < S; ++i) mbar_init(&full[i], KV8 ? 33 : 1);
    if (warp == 0) *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  __syncthreads();
  pdl_wait();

  const int len = p.seq_lens[seq];
  const int first_pos = (p.window > 0 && len > p.window) ? len - p.window : 0;
  int first_tile, span;
  key_span(len, p.window, first_tile, span);
  const int per = tiles_per_split(span, p.splits, p.min_tiles);
  const bool alone = span <= per;                        // the only split of its sequence with work
  if (split > 0 && split * per >= span) return;
  const int t0 = first_tile + split * per, t1 = min(first_tile + span, t0 + per);
  const int* table = p.block_table + size_t(seq) * p.max_blocks;

  // The copies of a tile: boxes of `box` slots, each of K and V and each of their column blocks, one to a lane. The slots of the
  // boxes that the warp comes to next are looked up 32 at a time, a lane each, and the next 32 while these are in use: a lookup
  // for every tile made the warp wait for it, as long as the tile's arithmetic takes.
  const int box_log2 = p.box_log2, box_slots = 1 << box_log2, boxes_log2 = 4 - box_log2, boxes = 1 << boxes_log2;
  const int copies = boxes * 2 * T::kBlocks;
  const int mine = t1 > t0 + warp ? (t1 - t0 - warp + kDecWarps - 1) / kDecWarps : 0;       // tiles of this warp
  auto look_up = [&](int chunk) {
    const int j = chunk * 32 + lane, i = j >> boxes_log2;
    const int pos = (t0 + warp + i * kDecWarps) * kDecTile + ((j & (boxes - 1)) << box_log2);
    return i < mine && pos < len ? table[pos / p.block_size] * p.block_size + pos % p.block_size : -1;
  };
  int chunk = 0, slots = look_up(0), next_slots = look_up(1);
  auto issue = [&](int i, int stage) {
    const int j = i << boxes_log2;
    if ((j >> 5) != chunk) {
      ++chunk;
      slots = next_slots;
      next_slots = look_up(chunk + 1);
    }
    const int pos0 = (t0 + warp + i * kDecWarps) * kDecTile;
    if (lane == 0) {
      const int used = (min(len - pos0, kDecTile) + box_slots - 1) >> box_log2;       // boxes with a key in them
      mbar_expect_tx(&full[stage], uint32_t((used << box_log2) * (T::kRowBytes * 2)));
    }
    __syncwarp();
    uint8_t* to = ring + stage * T::kStage;
    if (box_log2 == 4) {                                 // a box a tile: one lane a column block of K or V
      const int slot = __shfl_sync(0xffffffffu, slots, j & 31);
      if (lane < 2 * T::kBlocks)
        tma_load_3d(to + (lane & 1) * T::kBytes + (lane >> 1) * kDecTile * T::kPitch, (lane & 1) ? &tmV : &tmK, &full[stage],
                    (lane >> 1) * (KV8 ? T::kBlock : T::kBlock / 2), kvh, slot);
    } else {
      for (int c0 = 0; c0 < copies; c0 += 32) {
        const int c = c0 + lane, box = min(c / (2 * T::kBlocks), boxes - 1), which = c & 1, column = (c % (2 * T::kBlocks)) >> 1;
        const int slot = __shfl_sync(0xffffffffu, slots, (j + box) & 31);
        if (c < copies && slot != -1)
          tma_load_3d(to + which * T::kBytes + column * kDecTile * T::kPitch + (box << box_log2) * T::kPitch, which ? &tmV : &tmK,
                      &full[stage], column * (KV8 ? T::kBlock : T::kBlock / 2), kvh, slot);
      }
    }
    if (KV8) {
      // the scales of the tile's 16 keys and 16 values, a lane each, 0 outside the sequence
      const int row = lane & 15;
      const int slot = __shfl_sync(0xffffffffu, slots, (j + (row >> box_log2)) & 31);
      const bool live = slot != -1 && pos0 + row < len;
      const float* src = (lane < 16 ? p.k_scale : p.v_scale) + (live ? (size_t(slot) + (row & (box_slots - 1))) * p.Hkv + kvh : 0);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(scales + stage * 32 + lane)), "l"(src), "r"(live ? 4 : 0)
                   : "memory");
      asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(smem_u32(&full[stage])) : "memory");
    }
  };
  for (int i = 0; i < S && i < mine; ++i) issue(i, i);

  // the queries of the heads of this KV head as B operand: column = head, and the elements of d that step ks has for this lane
  uint32_t qb[NH][KS][2];
#pragma unroll
  for (int h = 0; h < NH; ++h) {
    const int head = h * 8 + g;
    const __nv_bfloat16* src = p.q + size_t(seq) * p.q_stride + size_t(kvh * G + head) * D;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      // bf16 keys: elements 2t, 2t + 1 and 2t + 8, 2t + 9 of the step's 16; codes: a lane holds 16 codes in a row of its key's 64,
      // four of them in each of the four steps
      const int d = KV8 ? (ks >> 2) * 64 + t4 * 16 + (ks & 3) * 4 : ks * 16 + t4 * 2;
      qb[h][ks][0] = head < G ? *reinterpret_cast<const uint32_t*>(src + d) : 0u;
      qb[h][ks][1] = head < G ? *reinterpret_cast<const uint32_t*>(src + d + (KV8 ? 2 : 8)) : 0u;
    }
  }

  float o[NH][KS][4];
  float m[NH][2], l[NH][2];                              // of heads 8 h + 2 t4 and the next; sums of this lane's keys only
#pragma unroll
  for (int h = 0; h < NH; ++h) {
#pragma unroll
    for (int n = 0; n < KS; ++n) { o[h][n][0] = o[h][n][1] = o[h][n][2] = o[h][n][3] = 0.f; }
    m[h][0] = m[h][1] = -INFINITY;
    l[h][0] = l[h][1] = 0.f;
  }
  // Where this lane's pieces of a tile stand. The swizzle exchanges pieces within 128 bytes by an exclusive or, so the pieces of
  // the other steps are one exclusive or away: 32 bytes a step of two pieces.
  const uint32_t k_at = KV8 ? T::at(g, t4) : T::at(lane & 15, lane >> 4);
  const uint32_t v_at = KV8 ? T::at((lane & 7) + (((lane >> 3) & 1) << 3), lane >> 4) : T::at((lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1);
  auto step_at = [](uint32_t at, int step) {              // the piece 2 * step further on
    constexpr int kSteps = T::kBlock / 32;
    return (at ^ uint32_t((step % kSteps) * 32)) + uint32_t((step / kSteps) * kDecTile * T::kPitch);
  };

  bool ok = true;
  int stage = 0;
  uint32_t phase = 0;
  for (int i = 0; i < mine; ++i) {
    ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag, p.st, kTimeoutSmemFull, (9u << 16) | stage));
    if (!ok) break;
    // factors of this lane's two keys, rows g and g + 8
    float ks[2] = {p.scale_log2, p.scale_log2}, vs[2] = {1.f, 1.f};
    if (KV8) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        ks[e] = scales[stage * 32 + g + e * 8] * (64.f * p.scale_log2);
        vs[e] = scales[stage * 32 + 16 + g + e * 8] * 64.f;
      }
    }
    uint8_t* tile_k = ring + stage * T::kStage;
    const uint32_t sk = smem_u32(tile_k), sv = sk + T::kBytes;
    const int key0 = (t0 + warp + i * kDecWarps) * kDecTile;
    const bool whole = key0 + kDecTile <= len && key0 >= first_pos;        // every key of the tile is seen
    if (!KV8 && key0 + kDecTile > len) {
      // values past the end get probability 0, but may be anything
      for (int c = lane; c < kDecTile * T::kRowBytes / 16; c += 32) {
        const int row = c / (T::kRowBytes / 16), piece = c % (T::kRowBytes / 16);
        if (key0 + row >= len)
          *reinterpret_cast<uint4*>(tile_k + T::kBytes + T::at(row, piece)) = make_uint4(0, 0, 0, 0);
      }
      __syncwarp();
    }
    // ---- S^T [16 keys x heads] = K Q^T, two sums over alternate steps
    float s[NH][2][4];
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) { s[h][e][0] = s[h][e][1] = s[h][e][2] = s[h][e][3] = 0.f; }
    if (!KV8) {
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        uint32_t a[4];
        ldmatrix_x4(a, sk + step_at(k_at, k));
#pragma unroll
        for (int h = 0; h < NH; ++h) mma_bf16_16816(s[h][k & 1], a, qb[h][k][0], qb[h][k][1]);
      }
    } else {
#pragma unroll
      for (int kk = 0; kk < D / 64; ++kk) {
        const uint4 lo = lds128(sk + step_at(k_at, kk * 2)), hi = lds128(sk + step_at(k_at, kk * 2) + 8 * T::kPitch);
        const uint32_t w0[4] = {lo.x, lo.y, lo.z, lo.w}, w1[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const uint32_t x0 = w0[w] ^ 0x80808080u, x1 = w1[w] ^ 0x80808080u;
          const uint32_t a[4] = {codes_pair(__byte_perm(x0, 0, 0x4140)), codes_pair(__byte_perm(x1, 0, 0x4140)),
                                 codes_pair(__byte_perm(x0, 0, 0x4342)), codes_pair(__byte_perm(x1, 0, 0x4342))};
#pragma unroll
          for (int h = 0; h < NH; ++h) mma_bf16_16816(s[h][w & 1], a, qb[h][kk * 4 + w][0], qb[h][kk * 4 + w][1]);
        }
      }
    }
    // ---- online softmax (log2 domain) over the keys, per head
    uint32_t pb[NH][2];                                  // P^T as B operand
    bool moved = false;
    float mn[NH][2];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          s[h][0][e * 2 + j] = (s[h][0][e * 2 + j] + s[h][1][e * 2 + j]) * ks[e];
          if (!whole) {
            const int pos = key0 + g + e * 8;
            if (pos >= len || pos < first_pos) s[h][0][e * 2 + j] = -INFINITY;
          }
        }
        float mx = fmaxf(s[h][0][j], s[h][0][2 + j]);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        mn[h][j] = fmaxf(m[h][j], mx);
        moved = moved || mn[h][j] > m[h][j];
      }
    }
    if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        float a[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          a[j] = (m[h][j] == -INFINITY) ? 0.f : dec_exp2(m[h][j] - mn[h][j]);
          m[h][j] = mn[h][j];
          l[h][j] *= a[j];
        }
#pragma unroll
        for (int n = 0; n < KS; ++n) { o[h][n][0] *= a[0]; o[h][n][1] *= a[1]; o[h][n][2] *= a[0]; o[h][n][3] *= a[1]; }
      }
    }
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      float e[4];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float base = m[h][j] == -INFINITY ? 0.f : m[h][j];
        e[j] = dec_exp2(s[h][0][j] - base);
        e[2 + j] = dec_exp2(s[h][0][2 + j] - base);
        l[h][j] += e[j] + e[2 + j];
      }
      pb[h][0] = transpose_8x8(pack_bf16x2(e[0] * vs[0], e[1] * vs[0]));
      pb[h][1] = transpose_8x8(pack_bf16x2(e[2] * vs[1], e[3] * vs[1]));
    }
    // ---- O^T [d x heads] += V^T P^T
    if (!KV8) {
#pragma unroll
      for (int n = 0; n < KS; ++n) {
        uint32_t a[4];
        ldmatrix_x4_trans(a, sv + step_at(v_at, n));
#pragma unroll
        for (int h = 0; h < NH; ++h) mma_bf16_16816(o[h][n], a, pb[h][0], pb[h][1]);
      }
    } else {
#pragma unroll
      for (int n = 0; n < KS; n += 2) {
        uint32_t r[4];
        ldmatrix_x4_trans(r, sv + step_at(v_at, n / 2));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          // two keys' codes of elements 2u and 2u + 1: the even elements are rows 0..7 of the fragment, the odd ones rows 8..15
          const uint32_t x0 = r[e * 2] ^ 0x80808080u, x1 = r[e * 2 + 1] ^ 0x80808080u;
          const uint32_t a[4] = {codes_pair(__byte_perm(x0, 0, 0x4240)), codes_pair(__byte_perm(x0, 0, 0x4341)),
                                 codes_pair(__byte_perm(x1, 0, 0x4240)), codes_pair(__byte_perm(x1, 0, 0x4341))};
#pragma unroll
          for (int h = 0; h < NH; ++h) mma_bf16_16816(o[h][n + e], a, pb[h][0], pb[h][1]);
        }
      }
    }
    __syncwarp();                                        // every lane has read the tile
    if (i + S < mine) issue(i + S, stage);
    if (++stage == S) { stage = 0; phase ^= 1; }
  }
  if (!ok) {                                             // let the copies on their way land before the CTA leaves
    const uint64_t from = global_timer_ns();
    while (global_timer_ns() - from < 200000ull) { }
  }

  // ---- combine the 4 warps of the CTA (in warp order), then write the split's partial or the final output
  // smerge layout: [warp][head][D + 2], over the tiles: nobody may still be reading a tile
#pragma unroll
  for (int h = 0; h < NH; ++h)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      l[h][j] += __shfl_xor_sync(0xffffffffu, l[h][j], 4);
      l[h][j] += __shfl_xor_sync(0xffffffffu, l[h][j], 8);
      l[h][j] += __shfl_xor_sync(0xffffffffu, l[h][j], 16);
    }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < NH; ++h)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int head = h * 8 + t4 * 2 + j;
      if (head >= G) continue;
      float* dst = smerge + (size_t(warp) * G + head) * (D + 2);
#pragma unroll
      for (int n = 0; n < KS; ++n) {
        dst[n * 16 + (KV8 ? 2 * g : g)] = o[h][n][j];
        dst[n * 16 + (KV8 ? 2 * g + 1 : g + 8)] = o[h][n][2 + j];
      }
      if (g == 0) { dst[D] = m[h][j]; dst[D + 1] = l[h][j]; }
    }
  __syncthreads();
  for (int i = threadIdx.x; i < G * D; i += blockDim.x) {
    const int hd = i / D, d = i - hd * D;
    float mm = -INFINITY;
    for (int w = 0; w < kDecWarps; ++w) mm = fmaxf(mm, smerge[(size_t(w) * G + hd) * (D + 2) + D]);
    float ll = 0.f, oo = 0.f;
    for (int w = 0; w < kDecWarps; ++w) {
      const float* src = smerge + (size_t(w) * G + hd) * (D + 2);
      const float a = (src[D] == -INFINITY) ? 0.f : exp2f(src[D] - mm);
      ll += src[D + 1] * a;
      oo += src[d] * a;
    }
    const int head = kvh * G + hd;
    if (alone) {
      p.out[(size_t(seq) * p.H + head) * D + d] = __float2bfloat16(ll > 0.f ? oo / ll : 0.f);
    } else {
      float* pp = p.partial + ((size_t(seq) * p.H + head) * p.splits + split) * (D + 2);
      pp[d] = oo;
      if (d == 0) { pp[D] = mm; pp[D + 1] = ll; }
    }
  }
}

// out[seq, head, :] = merge of the partials of a sequence's splits, in split order. One thread per element of the head (D
// threads). The shares' weights are taken by a thread each and the loads of eight shares are in flight at a time: one after the
// other, with the weights taken by every thread, 32 shares of 32 heads of 128 took 12 to 17 us, as long as the attention of 8000 keys.
constexpr int kMergeShares = 64;
__global__ void __launch_bounds__(128) decode_merge_kernel(const DecodeParams p) {
  pdl_launch_dependents();     // a dependent launched programmatically may set itself up while this kernel runs
  pdl_wait();
  const int row = blockIdx.x, D = p.D, t = threadIdx.x;
  int first_tile, span;
  key_span(p.seq_lens[row / p.H], p.window, first_tile, span);
  const int per = tiles_per_split(span, p.splits, p.min_tiles);
  if (span <= per) return;                               // written out by its only split
  const int used = (span + per - 1) / per;
  const float* __restrict__ base = p.partial + size_t(row) * p.splits * (D + 2);
  __shared__ float weight[kMergeShares], sum[kMergeShares], red[4];
  float mm = -INFINITY, ll = 0.f, oo = 0.f;
  if (used <= 8) {                                       // few shares: all of them in flight, no barrier
    float m[8], l[8], v[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const bool there = s < used;
      m[s] = there ? base[s * (D + 2) + D] : -INFINITY;
      l[s] = there ? base[s * (D + 2) + D + 1] : 0.f;
      v[s] = there ? base[s * (D + 2) + t] : 0.f;
      mm = fmaxf(mm, m[s]);
    }
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const float a = (m[s] == -INFINITY) ? 0.f : exp2f(m[s] - mm);
      ll += l[s] * a;
      oo += v[s] * a;
    }
    p.out[size_t(row) * D + t] = __float2bfloat16(ll > 0.f ? oo / ll : 0.f);
    return;
  }
  for (int s = t; s < used; s += blockDim.x) mm = fmaxf(mm, base[s * (D + 2) + D]);
  mm = warp_max(mm);
  if ((t & 31) == 0) red[t >> 5] = mm;
  __syncthreads();
  for (int w = 0; w < int(blockDim.x >> 5); ++w) mm = fmaxf(mm, red[w]);
  for (int s0 = 0; s0 < used; s0 += kMergeShares) {
    const int n = min(kMergeShares, used - s0);
    if (t < n) {
      const float m = base[(s0 + t) * (D + 2) + D];
      weight[t] = (m == -INFINITY) ? 0.f : exp2f(m - mm);
      sum[t] = base[(s0 + t) * (D + 2) + D + 1];
    }
    __syncthreads();
    const float* src = base + size_t(s0) * (D + 2) + t;
#pragma unroll 8
    for (int s = 0; s < n; ++s) {
      ll += sum[s] * weight[s];
      oo += src[s * (D + 2)] * weight[s];
    }
    __syncthreads();                                     // the next shares' weights take the place of these
  }
  p.out[size_t(row) * D + t] = __float2bfloat16(ll > 0.f ? oo / ll : 0.f);
}

// k / v rows of new tokens -> their cache slots. src rows hold heads packed [Hkv, D]; slot = block * block_size + offset.
__global__ void kv_write_paged_kernel(const __nv_bfloat16* __restrict__ k_src, const __nv_bfloat16* __restrict__ v_src,
                                      long long src_stride, const int* __restrict__ slots,
                                      __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache,
                                      int tokens, int row_elems) {
  const int chunks = row_elems / 8;
  const long long total = (long long)tokens * chunks;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int t = int(i / chunks), c = int(i - (long long)t * chunks);
    const int slot = slots[t];
    if (slot < 0) continue;     // padding token
    const uint4 kk = *reinterpret_cast<const uint4*>(k_src + t * src_stride + c * 8);
    const uint4 vv = *reinterpret_cast<const uint4*>(v_src + t * src_stride + c * 8);
    *reinterpret_cast<uint4*>(k_cache + size_t(slot) * row_elems + c * 8) = kk;
    *reinterpret_cast<uint4*>(v_cache + size_t(slot) * row_elems + c * 8) = vv;
  }
}

template <int D, int KV8, int NH, bool SWIZZLE>
static int launch_decode(DecodeParams p, int seqs, long long slots, cudaStream_t stream) {
  using T = DecTile<D, KV8, SWIZZLE>;
  constexpr size_t kSmem = size_t(kDecWarps) * T::kRing + kDecWarps * T::kStages * (8 + 128) + 16 + 1024;
  static_assert(size_t(kDecWarps) * kDecMaxGroup * (D + 2) * 4 <= size_t(kDecWarps) * T::kRing, "the merge fits in the rings");
  auto kern = paged_decode_kernel<D, KV8, NH, SWIZZLE>;
  static DeviceOnce configured;
  if (int e = configured.run([&] { return int(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem))); }))
    return e;
  if (T::kPitch != T::kBlock) p.box_log2 = 0;
  // (elements of a head, head, slot)
  constexpr int kElem = KV8 ? 1 : 2;
  uint64_t dims[3] = {uint64_t(D), uint64_t(p.Hkv), uint64_t(slots)};
  uint64_t strides[2] = {uint64_t(D) * kElem, uint64_t(p.Hkv) * D * kElem};
  uint32_t box[3] = {uint32_t(T::kBlock / kElem), 1, 1u << p.box_log2};
  const CUtensorMapDataType type = KV8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const CUtensorMapSwizzle swizzle = !SWIZZLE ? CU_TENSOR_MAP_SWIZZLE_NONE : T::kBlock == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  CUtensorMap tk, tv;
  if (encode_tensor_map(&tk, type, 3, const_cast<__nv_bfloat16*>(p.k_cache), dims, strides, box, swizzle)) return -10;
  if (encode_tensor_map(&tv, type, 3, const_cast<__nv_bfloat16*>(p.v_cache), dims, strides, box, swizzle)) return -11;
  return launch_overlapped(kern, dim3(seqs, p.Hkv, p.splits), kDecWarps * 32, kSmem, stream, tk, tv, p);
}

}  // namespace idrak

using namespace idrak;

IDRAK_API long long idrak_decode_partial_floats(int seqs, int H, int D, int splits) {
  return splits > 1 ? (long long)seqs * H * splits * (D + 2) : 0;
}

// Over an int8 cache when k_scale / v_scale are given (one fp32 scale per (slot, kv head)). A sequence's keys are shared by
// at most `splits` CTAs per KV head, at least `min_keys` keys each (rounded up to tiles). cache_slots: blocks x block_size.
IDRAK_API int idrak_paged_decode_kv(const void* q, long long q_stride, const void* k_cache, const void* v_cache,
                                    const float* k_scale, const float* v_scale, const int* block_table,
                                    const int* seq_lens, void* out, float* partial, int seqs, int H, int Hkv, int D,
                                    int block_size, int max_blocks, long long cache_slots, int splits, int min_keys, float scale, int window,
                                    void* stream_) {
  if (D != 64 && D != 128) return -2;
  if (block_size < 1) return -7;
  const bool kv8 = k_scale != nullptr;
  if (kv8 && !v_scale) return -6;
  if (H % Hkv || H / Hkv > kDecMaxGroup) return -3;
  if (splits > 1 && !partial) return -4;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  DecodeParams p;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.q_stride = q_stride > 0 ? q_stride : (long long)H * D;
  if ((p.q_stride % 8) || (reinterpret_cast<uintptr_t>(q) & 15)) return -5;
  p.k_cache = static_cast<const __nv_bfloat16*>(k_cache);
  p.v_cache = static_cast<const __nv_bfloat16*>(v_cache);
  p.k_scale = k_scale;
  p.v_scale = v_scale;
  p.block_table = block_table;
  p.seq_lens = seq_lens;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.partial = partial;
  p.H = H; p.Hkv = Hkv; p.D = D; p.block_size = block_size; p.max_blocks = max_blocks;
  p.splits = splits < 1 ? 1 : splits;
  p.min_tiles = min_keys <= kDecTile ? 1 : (min_keys + kDecTile - 1) / kDecTile;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.window = window;
  p.box_log2 = 0;
  while (p.box_log2 < 4 && block_size % (2 << p.box_log2) == 0) ++p.box_log2;
  p.st = status_device_ptr();
  if (seqs <= 0) return 0;
  const bool swizzle = p.box_log2 >= 3;
  int rc;
#define IDRAK_DECODE(D_, Q_, N_) \
  rc = swizzle ? launch_decode<D_, Q_, N_, true>(p, seqs, cache_slots, s) : launch_decode<D_, Q_, N_, false>(p, seqs, cache_slots, s)
#define IDRAK_DECODE_HEADS(D_, Q_) \
  if (H / Hkv <= 8) IDRAK_DECODE(D_, Q_, 1); \
  else IDRAK_DECODE(D_, Q_, 2)
  if (D == 64) {
    if (kv8) { IDRAK_DECODE_HEADS(64, 1); } else { IDRAK_DECODE_HEADS(64, 0); }
  } else {
    if (kv8) { IDRAK_DECODE_HEADS(128, 1); } else { IDRAK_DECODE_HEADS(128, 0); }
  }
#undef IDRAK_DECODE_HEADS
#undef IDRAK_DECODE
  if (rc == 0 && p.splits > 1)
    rc = launch_overlapped(decode_merge_kernel, dim3(unsigned(seqs * H)), D < 128 ? 64 : 128, 0, s, p);
  return rc;
}

IDRAK_API int idrak_kv_write_paged(const void* k_src, const void* v_src, long long src_stride, const int* slots,
                                   void* k_cache, void* v_cache, int tokens, int row_elems, void* stream_) {
  if (row_elems % 8) return -2;
  const long long total = (long long)tokens * (row_elems / 8);
  long long want = (total + 255) / 256, cap = (long long)sm_count() * 8;
  kv_write_paged_kernel<<<int(want < 1 ? 1 : (want < cap ? want : cap)), 256, 0, static_cast<cudaStream_t>(stream_)>>>(
      static_cast<const __nv_bfloat16*>(k_src), static_cast<const __nv_bfloat16*>(v_src), src_stride, slots,
      static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache), tokens, row_elems);
  note_launches(1);
  return int(cudaGetLastError());
}
