// One launch between the packed QKV projection and attention: optional per-head RMS norm of queries and keys,
// rotary embedding of both, and the write of the new keys / values into the paged cache - bf16, or int8 with one
// scale per (token, kv head).
//
// The packed projection row of a token is [H query heads | Hkv key heads | Hkv value heads] x D. One warp takes one token and
// a run of heads: the angles (a power and a range-reduced sincos per pair) are taken once per run, and the loads of four heads
// are in flight at a time. 9712 tokens x 48 heads of 128: 128 us with a head per warp, 63 now. Lane l holds elements l, l + 32,
// l + 64, ... of a head (or neighbouring pairs of them, see the kernel), so both members of a rotation pair
// (i, i + rot_dim / 2) sit in the same lane.
//   query head   -> norm, rotate, written back in place (attention reads it from the projection buffer)
//   key head     -> norm, rotate, written back in place (prefill attention reads it there) and into the cache slot
//   value head   -> copied into the cache slot
// Replaces three launches of the unfused path (norm of q / k, RoPE, cache write).
//
// int8 cache: scale = max|x| / 127 per (token, kv head), code = round(x / scale); the decode attention kernel
// multiplies the scale back in (decode_attn.cu).
//
// Reference counterparts: norm_rope_heads_f32 (src/Idrak.Gpu/Cuda/PtxKernels.Decoder.cs:355-389), kv_write_bf16
// (PtxKernels.Decoding.cs:12), kv_write_int8 (PtxKernels.Quantized.cs:251).
#include "common.cuh"

namespace idrak {

struct NormRopeKvParams {
  __nv_bfloat16* qkv;            // [T, (H + 2 Hkv) D], rows row_stride elements apart
  long long row_stride;
  const int* positions;          // [T] or null (no rotation)
  const int* slots;              // [T]: block * block_size + offset, negative = do not cache; or null
  void* k_cache;                 // [slots, Hkv, D] bf16 or int8
  void* v_cache;
  float* k_scale;                // [slots, Hkv] when the cache is int8
  float* v_scale;
  const __nv_bfloat16* q_norm;   // [D] weights (already with any offset added) or null
  const __nv_bfloat16* k_norm;
  float eps;
  float theta, freq_scale;
  int rot_dim;                   // elements of a head that rotate (pairs i, i + rot_dim / 2); 0 = no rotation
  int T, H, Hkv, D, kv_int8;
  int run;                       // heads per warp
};

// One warp per token and run of heads, four heads in flight at a time (of 256 elements: one); each lane owns PER = D / 32 elements of a head.
// kPairs = 0: elements e = lane + 32 j (any rotary width that is a multiple of 64). kPairs = 1 (PER = 4, rotary width = the
// whole head or none): e = 2 lane, 2 lane + 1 and the same plus D / 2, in four-byte accesses.
template <int PER, int kPairs>
__global__ void __launch_bounds__(256) norm_rope_kv_kernel(const NormRopeKvParams p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int kBatch = PER == 8 ? 1 : 4;            // heads in flight: more than one of 256 elements only costs registers
  const int heads_total = p.H + 2 * p.Hkv;
  const int runs = (heads_total + p.run - 1) / p.run;
  const long long unit = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (unit >= (long long)p.T * runs) return;
  const int t = int(unit / runs), h0 = int(unit - (long long)t * runs) * p.run;
  const int lane = threadIdx.x & 31;
  const int D = p.D;
  const bool rotate = p.rot_dim > 0 && p.positions;
  const int hj = kPairs ? 2 : p.rot_dim >> 6;         // distance in j of a pair's members: half / 32, half = rot_dim / 2
  auto element = [&](int j) { return kPairs ? 2 * lane + (j & 1) + (j >> 1) * (PER * 16) : lane + 32 * j; };
  auto load = [&](const __nv_bfloat16* src, float (&v)[PER]) {
    if constexpr (kPairs) {
#pragma unroll
      for (int j = 0; j < PER; j += 2) {
        const float2 f = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(src + element(j)));
        v[j] = f.x;
        v[j + 1] = f.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < PER; ++j) v[j] = __bfloat162float(src[element(j)]);
    }
  };
  auto store = [&](__nv_bfloat16* dst, const float (&v)[PER]) {
    if constexpr (kPairs) {
#pragma unroll
      for (int j = 0; j < PER; j += 2) *reinterpret_cast<uint32_t*>(dst + element(j)) = pack_bf16x2(v[j], v[j + 1]);
    } else {
#pragma unroll
      for (int j = 0; j < PER; ++j) dst[element(j)] = __float2bfloat16(v[j]);
    }
  };
  float sn[PER / 2], cs[PER / 2];
  if (rotate && h0 < p.H + p.Hkv) {
    const float pos = float(p.positions[t]) * p.freq_scale;      // the arithmetic of the rope kernels, so results agree bit for bit
#pragma unroll
    for (int j = 0; j < PER / 2; ++j) {
      if (j < hj) {
        const float inv = __powf(p.theta, -2.0f * float(element(j)) / float(p.rot_dim));
        sincosf(pos * inv, &sn[j], &cs[j]);
      }
    }
  }
  const int slot = p.slots ? p.slots[t] : -1;
  __nv_bfloat16* row_base = p.qkv + size_t(t) * p.row_stride;
  const int h1 = min(heads_total, h0 + p.run);
  for (int hb = h0; hb < h1; hb += kBatch) {
    float buf[kBatch][PER];
#pragma unroll
    for (int i = 0; i < kBatch; ++i)
      if (hb + i < h1) load(row_base + size_t(hb + i) * D, buf[i]);
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int h = hb + i;
      if (h >= h1) break;
      const bool is_q = h < p.H, is_k = !is_q && h < p.H + p.Hkv;
      const int kvh = is_q ? 0 : (is_k ? h - p.H : h - p.H - p.Hkv);
      float(&v)[PER] = buf[i];
      if (is_q || is_k) {
        const __nv_bfloat16* nw = is_q ? p.q_norm : p.k_norm;
        if (nw) {
          float ss = 0.f;
#pragma unroll
          for (int j = 0; j < PER; ++j) ss += v[j] * v[j];
          ss = warp_sum(ss);
          const float r = rsqrtf(ss / float(D) + p.eps);
#pragma unroll
          for (int j = 0; j < PER; ++j)
            v[j] = __bfloat162float(__float2bfloat16(v[j] * r * __bfloat162float(nw[element(j)])));   // as a separate norm would store it
        }
        if (rotate) {
#pragma unroll
          for (int j = 0; j < PER / 2; ++j) {
            if (j < hj) {
              // v[j + hj], hj any of 1 .. PER / 2 (3 for 192 of 256): constant indices, so that v stays in registers
#pragma unroll
              for (int o = 1; o <= PER / 2; ++o) {
                if (o == hj && j + o < PER) {
                  const float a = v[j], b = v[j + o];
                  v[j] = a * cs[j] - b * sn[j];
                  v[j + o] = b * cs[j] + a * sn[j];
                }
              }
            }
          }
        }
        store(row_base + size_t(h) * D, v);
      }
      if (is_q || slot < 0) continue;
      const size_t row = (size_t(slot) * p.Hkv + kvh) * D;
      if (!p.kv_int8) {
        store(static_cast<__nv_bfloat16*>(is_k ? p.k_cache : p.v_cache) + row, v);
      } else {
        float mx = 0.f;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
          v[j] = __bfloat162float(__float2bfloat16(v[j]));       // quantise what the bf16 cache would have held
          mx = fmaxf(mx, fabsf(v[j]));
        }
        mx = warp_max(mx);
        const float scale = mx > 0.f ? mx / 127.f : 1.f;
        int8_t* dst = static_cast<int8_t*>(is_k ? p.k_cache : p.v_cache) + row;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
          const int q = __float2int_rn(v[j] / scale);
          dst[element(j)] = int8_t(max(-127, min(127, q)));
        }
        if (lane == 0) (is_k ? p.k_scale : p.v_scale)[size_t(slot) * p.Hkv + kvh] = scale;
      }
    }
  }
}

// Where each sequence's new token goes and how long the sequence is with it: the index arithmetic at the head of a decode
// step in one launch instead of nine. A position outside its table row is reported in the status word; its token is not
// cached (slot -1) and the sequence ends with the row.
__global__ void decode_slots_kernel(const int* __restrict__ positions, const int* __restrict__ table, int n, long long stride,
                                    int width, int block_size, int* __restrict__ slots, int* __restrict__ lens, Status* st) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int pos = positions[i], block = pos / block_size;
  if (pos < 0 || block >= width) {
    report(st, kBadArgument, (11u << 16) | 1u, uint32_t(i));
    slots[i] = -1;
    lens[i] = pos < 0 ? 0 : width * block_size;
    return;
  }
  slots[i] = table[i * stride + block] * block_size + pos % block_size;
  lens[i] = pos + 1;
}

}  // namespace idrak

using namespace idrak;

// slots[i] = table[i, positions[i] / block_size] * block_size + positions[i] % block_size, lens[i] = positions[i] + 1; the
// table's rows hold `width` blocks and lie `stride` apart.
IDRAK_API int idrak_decode_slots(const int* positions, const int* table, int n, long long stride, int width, int block_size,
                                 int* slots, int* lens, void* stream_) {
  if (n <= 0) return 0;
  if (block_size <= 0 || width <= 0) return -2;
  return launch_overlapped(decode_slots_kernel, dim3(unsigned((n + 127) / 128)), 128, 0, static_cast<cudaStream_t>(stream_),
                           positions, table, n, stride, width, block_size, slots, lens, status_device_ptr());
}

// qkv rows are rotated / normalised in place; keys and values also go to the cache rows named by `slots`.
// Needs D in {64, 128, 256} and rot_dim % 64 == 0 (0: no rotation). Returns 0, a CUDA error or a negative
// argument error.
IDRAK_API int idrak_norm_rope_kv(void* qkv, long long row_stride, const int* positions, const int* slots, void* k_cache,
                                 void* v_cache, float* k_scale, float* v_scale, const void* q_norm, const void* k_norm,
                                 float eps, float theta, float freq_scale, int rot_dim, int T, int H, int Hkv, int D,
                                 int kv_int8, void* stream_) {
  if (T <= 0) return 0;
  if (D != 64 && D != 128 && D != 256) return -2;
  if (rot_dim < 0 || rot_dim > D || (rot_dim & 63)) return -3;
  if (kv_int8 && slots && (!k_scale || !v_scale)) return -4;
  NormRopeKvParams p;
  p.qkv = static_cast<__nv_bfloat16*>(qkv);
  p.row_stride = row_stride;
  p.positions = positions; p.slots = slots;
  p.k_cache = k_cache; p.v_cache = v_cache; p.k_scale = k_scale; p.v_scale = v_scale;
  p.q_norm = static_cast<const __nv_bfloat16*>(q_norm);
  p.k_norm = static_cast<const __nv_bfloat16*>(k_norm);
  p.eps = eps; p.theta = theta; p.freq_scale = freq_scale; p.rot_dim = rot_dim;
  p.T = T; p.H = H; p.Hkv = Hkv; p.D = D; p.kv_int8 = kv_int8;
  const int heads = H + 2 * Hkv;
  // Heads per warp: the fewest rounds of 32 warps per SM, a round as long as a fixed part (the angles) and its heads. 9000
  // tokens of 48 heads of 128: 152 us with a head per warp, 58 with 16; 1000 of 36 over an int8 cache 14.3 / 11.5 with four, and
  // 16.4 with the 16 that merely leave four warps to every scheduler.
  long long least = 0;
  for (int run = 1; run <= 16; run *= 2) {
    const long long warps = (long long)T * ((heads + run - 1) / run), place = 32ll * sm_count();
    const long long cost = (warps + place - 1) / place * (5 + 2 * run);
    if (run == 1 || cost < least) {
      p.run = run;
      least = cost;
    }
  }
  const long long units = (long long)T * ((heads + p.run - 1) / p.run);
  const int blocks = int((units + 7) / 8);
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const bool pairs = D == 128 && (rot_dim == 0 || rot_dim == 128 || !positions) && row_stride % 2 == 0 &&
                     (reinterpret_cast<uintptr_t>(qkv) & 3) == 0 && (reinterpret_cast<uintptr_t>(k_cache) & 3) == 0 &&
                     (reinterpret_cast<uintptr_t>(v_cache) & 3) == 0;
  auto kern = D == 64 ? norm_rope_kv_kernel<2, 0>
                      : (D == 256 ? norm_rope_kv_kernel<8, 0> : (pairs ? norm_rope_kv_kernel<4, 1> : norm_rope_kv_kernel<4, 0>));
  return launch_overlapped(kern, dim3(unsigned(blocks)), 256, 0, s, p);
}
