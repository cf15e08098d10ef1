// Self-attention over a packed projection for head sizes below 64, forward and backward, in fp32 throughout.
//
// The tensor-core kernels take head sizes 64 and 128 and their probabilities as bf16 operands; smaller heads keep the probabilities
// in fp32, so their products run on the FMA units here. As separate torch operations (casts, two fp32 GEMMs, mask, softmax, casts,
// and the backward of each) a layer of 8 x 128 tokens, 4 heads of 32, took some 45 launches of 2 to 5 us, 350 us of a step with four such layers;
// here it is two, bound by latency: a block has 16 or 32 rows and walks the other side in steps of 32.
//
// A warp owns 4 or 8 rows (queries, or keys for dK and dV), a lane one of the 32 columns of a step: the lane holds its
// column's vectors in registers, the rows' come as broadcasts from shared memory, and a score needs no reduction. For the
// products over the columns the lanes stand for elements of the head, with the step's probabilities (or dS) passed through
// shared memory: a multiply-add per row and element for each broadcast.
//
// The forward pass keeps its result in fp32 too, so that delta = rowsum(dO * O) is as exact as the sum over probabilities.
//
// Reference counterparts: attention_f32 and attn_bwd_{d,kv,q}_f32 (src/Idrak.Gpu/Cuda/PtxKernels.Rows.cs:779-1750).
#include "common.cuh"

namespace idrak {

constexpr int kSaCols = 32, kSaThreads = 128;      // columns of a step: a lane each

struct SmallAttnParams {
  const __nv_bfloat16* qkv;      // [B, S, (H + 2 Hkv) D]
  const __nv_bfloat16* dout;     // [B, S, H D]
  __nv_bfloat16* out;            // [B, S, H D]
  __nv_bfloat16* dqkv;
  float* o32;                    // [B, S, H D]
  float* lse2;                   // [B, H, S], base 2
  int B, S, H, Hkv, D, causal;
  float scale;
};

// ROWS rows of D elements from row `row0` on, on their way to shared memory: fetched into registers, so that the next step's come
// while this one is worked on, then written as fp32 [ROWS][PITCH], zeros outside the sequence and the head.
template <int DP, int ROWS>
struct SaTile {
  static constexpr int kPieces = ROWS * (DP / 8), kPer = (kPieces + kSaThreads - 1) / kSaThreads;
  uint4 v[kPer];
  __device__ __forceinline__ void fetch(const __nv_bfloat16* base, size_t stride, int row0, int S, int D) {
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = threadIdx.x + j * kSaThreads, r = i / (DP / 8), c = (i % (DP / 8)) * 8;
      v[j] = i < kPieces && row0 + r < S && c < D ? *reinterpret_cast<const uint4*>(base + size_t(row0 + r) * stride + c) : make_uint4(0, 0, 0, 0);
    }
  }
  template <int PITCH>
  __device__ __forceinline__ void put(float* dst) const {
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = threadIdx.x + j * kSaThreads, r = i / (DP / 8), c = (i % (DP / 8)) * 8;
      if (i >= kPieces) continue;
      const float2 a = unpack_bf16x2(v[j].x), b = unpack_bf16x2(v[j].y), e = unpack_bf16x2(v[j].z), f = unpack_bf16x2(v[j].w);
      float4* d = reinterpret_cast<float4*>(dst + r * PITCH + c);
      d[0] = make_float4(a.x, a.y, b.x, b.y);
      d[1] = make_float4(e.x, e.y, f.x, f.y);
    }
  }
};
// a row of shared memory into registers
template <int DP>
__device__ __forceinline__ void sa_row(const float* src, float (&r)[DP]) {
#pragma unroll
  for (int c = 0; c < DP; c += 4) {
    const float4 v = *reinterpret_cast<const float4*>(src + c);
    r[c] = v.x; r[c + 1] = v.y; r[c + 2] = v.z; r[c + 3] = v.w;
  }
}
// dots of R rows of shared memory (PITCH apart, the same for every lane) with the lane's vector
template <int DP, int PITCH, int R>
__device__ __forceinline__ void sa_dots(const float* rows, const float (&v)[DP], float (&s)[R]) {
#pragma unroll
  for (int i = 0; i < R; ++i) s[i] = 0.f;
#pragma unroll
  for (int c = 0; c < DP; c += 4)
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(rows + i * PITCH + c);
      s[i] += a.x * v[c];
      s[i] += a.y * v[c + 1];
      s[i] += a.z * v[c + 2];
      s[i] += a.w * v[c + 3];
    }
}
// acc[row][element] += sum over the step's columns of w[column][row] * m[column][element]; a lane has elements lane, lane + 32
template <int DP, int PITCH, int R>
__device__ __forceinline__ void sa_accumulate(const float* w, const float* m, int lane, float (&acc)[R][(DP + 31) / 32]) {
#pragma unroll 8
  for (int j = 0; j < kSaCols; ++j) {
    float x[(DP + 31) / 32];
#pragma unroll
    for (int e = 0; e < (DP + 31) / 32; ++e) x[e] = DP < 32 && lane >= DP ? 0.f : m[j * PITCH + e * 32 + lane];
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      const float4 a = *reinterpret_cast<const float4*>(w + j * R + i);
#pragma unroll
      for (int e = 0; e < (DP + 31) / 32; ++e) {
        acc[i][e] += a.x * x[e];
        acc[i + 1][e] += a.y * x[e];
        acc[i + 2][e] += a.z * x[e];
        acc[i + 3][e] += a.w * x[e];
      }
    }
  }
}
template <int R>
__device__ __forceinline__ void sa_put(float* w, int lane, const float (&v)[R]) {
#pragma unroll
  for (int i = 0; i < R; i += 4) *reinterpret_cast<float4*>(w + lane * R + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}

// R: rows of a warp, 4 R a block
template <int DP, int R>
__global__ void __launch_bounds__(kSaThreads) small_attn_fwd_kernel(const SmallAttnParams p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int kPitch = DP + 4, kE = (DP + 31) / 32, kRows = 4 * R;
  __shared__ __align__(16) float sq[kRows * kPitch], sk[kSaCols * kPitch], sv[kSaCols * kPitch];
  __shared__ __align__(16) float sp[kSaThreads / 32][kSaCols * R];
  const int q0 = (gridDim.x - 1 - blockIdx.x) * kRows, h = blockIdx.y, b = blockIdx.z;      // the longest rows first
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kvh = h / (p.H / p.Hkv);
  const size_t stride = size_t(p.H + 2 * p.Hkv) * p.D;
  const __nv_bfloat16* base = p.qkv + size_t(b) * p.S * stride;
  const __nv_bfloat16 *kbase = base + size_t(p.H + kvh) * p.D, *vbase = base + size_t(p.H + p.Hkv + kvh) * p.D;
  const float sl2 = p.scale * 1.4426950408889634f;
  SaTile<DP, kSaCols> tk, tv;
  tk.fetch(kbase, stride, 0, p.S, p.D);
  tv.fetch(vbase, stride, 0, p.S, p.D);
  {
    SaTile<DP, kRows> tq;
    tq.fetch(base + size_t(h) * p.D, stride, q0, p.S, p.D);
    tq.template put<kPitch>(sq);
  }
  float o[R][kE] = {}, m[R], l[R];
#pragma unroll
  for (int i = 0; i < R; ++i) { m[i] = -INFINITY; l[i] = 0.f; }
  const int end = p.causal ? min(p.S, q0 + kRows) : p.S;
  for (int k0 = 0; k0 < end; k0 += kSaCols) {
    __syncthreads();
    tk.template put<kPitch>(sk);
    tv.template put<kPitch>(sv);
    __syncthreads();
    tk.fetch(kbase, stride, k0 + kSaCols, p.S, p.D);
    tv.fetch(vbase, stride, k0 + kSaCols, p.S, p.D);
    float s[R];
    {
      float kr[DP];
      sa_row<DP>(sk + lane * kPitch, kr);
      sa_dots<DP, kPitch, R>(sq + warp * R * kPitch, kr, s);
    }
    const int key = k0 + lane;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = q0 + warp * R + i;
      s[i] = key >= p.S || (p.causal && key > row) ? -INFINITY : s[i] * sl2;
      const float mn = fmaxf(m[i], warp_max(s[i]));
      const float base2 = mn == -INFINITY ? 0.f : mn, a = exp2f(m[i] - base2);
      m[i] = mn;
      s[i] = exp2f(s[i] - base2);
      l[i] = l[i] * a + s[i];
#pragma unroll
      for (int e = 0; e < kE; ++e) o[i][e] *= a;
    }
    sa_put<R>(sp[warp], lane, s);
    __syncwarp();
    sa_accumulate<DP, kPitch, R>(sp[warp], sv, lane, o);
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = q0 + warp * R + i;
    const float sum = warp_sum(l[i]);
    if (row >= p.S) continue;
    const size_t at = (size_t(b) * p.S + row) * p.H * p.D + size_t(h) * p.D;
#pragma unroll
    for (int e = 0; e < kE; ++e) {
      const int d = e * 32 + lane;
      if (d < p.D) {
        const float v = o[i][e] / sum;
        p.o32[at + d] = v;
        p.out[at + d] = __float2bfloat16(v);
      }
    }
    if (lane == 0) p.lse2[(size_t(b) * p.H + h) * p.S + row] = m[i] + log2f(sum);
  }
}

// The first `q_tiles` blocks of a (head, batch) take dQ of 4 R queries each. The others take dK and dV of 4 R keys of a KV head
// over every query that sees them, of all the heads that share it, summed in order; they are launched for the first head of each
// group. Both find delta for themselves, so that they are one launch.
template <int DP, int R>
__global__ void __launch_bounds__(kSaThreads) small_attn_bwd_kernel(const SmallAttnParams p, int tiles) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int kPitch = DP + 4, kE = (DP + 31) / 32, kRows = 4 * R;
  extern __shared__ __align__(16) float sa_smem[];
  float *ra = sa_smem, *rb = ra + kRows * kPitch, *ca = rb + kRows * kPitch, *cb = ca + kSaCols * kPitch, *sw = cb + kSaCols * kPitch;
  const int h0 = blockIdx.y, b = blockIdx.z, group = p.H / p.Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kvh = h0 / group;
  const size_t stride = size_t(p.H + 2 * p.Hkv) * p.D, orow = size_t(p.H) * p.D;
  const __nv_bfloat16 *base = p.qkv + size_t(b) * p.S * stride, *dbase = p.dout + size_t(b) * p.S * orow;
  const __nv_bfloat16 *kbase = base + size_t(p.H + kvh) * p.D, *vbase = base + size_t(p.H + p.Hkv + kvh) * p.D;
  const float* obase = p.o32 + size_t(b) * p.S * orow;
  const float* lbase = p.lse2 + size_t(b) * p.H * p.S;
  const float sl2 = p.scale * 1.4426950408889634f;
  float* w = sw + warp * 2 * kSaCols * R;
  SaTile<DP, kSaCols> ta, tb;
  if (int(blockIdx.x) < tiles) {
    const int q0 = (tiles - 1 - int(blockIdx.x)) * kRows;                 // the longest rows first
    ta.fetch(kbase, stride, 0, p.S, p.D);
    tb.fetch(vbase, stride, 0, p.S, p.D);
    {
      SaTile<DP, kRows> tq, td;
      tq.fetch(base + size_t(h0) * p.D, stride, q0, p.S, p.D);
      td.fetch(dbase + size_t(h0) * p.D, orow, q0, p.S, p.D);
      tq.template put<kPitch>(ra);
      td.template put<kPitch>(rb);
    }
    __syncthreads();
    float dq[R][kE] = {}, lse[R], dl[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = q0 + warp * R + i;
      float acc = 0.f;
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        const int d = e * 32 + lane;
        if (row < p.S && d < p.D) acc += rb[(warp * R + i) * kPitch + d] * obase[size_t(row) * orow + size_t(h0) * p.D + d];
      }
      dl[i] = warp_sum(acc);
      lse[i] = row < p.S ? lbase[size_t(h0) * p.S + row] : INFINITY;
    }
    const int end = p.causal ? min(p.S, q0 + kRows) : p.S;
    for (int k0 = 0; k0 < end; k0 += kSaCols) {
      __syncthreads();
      ta.template put<kPitch>(ca);
      tb.template put<kPitch>(cb);
      __syncthreads();
      ta.fetch(kbase, stride, k0 + kSaCols, p.S, p.D);
      tb.fetch(vbase, stride, k0 + kSaCols, p.S, p.D);
      float s[R], dp[R];
      {
        float r[DP];
        sa_row<DP>(ca + lane * kPitch, r);
        sa_dots<DP, kPitch, R>(ra + warp * R * kPitch, r, s);
        sa_row<DP>(cb + lane * kPitch, r);
        sa_dots<DP, kPitch, R>(rb + warp * R * kPitch, r, dp);
      }
      const int key = k0 + lane;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const bool out = key >= p.S || (p.causal && key > q0 + warp * R + i);
        s[i] = out ? 0.f : exp2f(s[i] * sl2 - lse[i]) * (dp[i] - dl[i]) * p.scale;
      }
      sa_put<R>(w, lane, s);
      __syncwarp();
      sa_accumulate<DP, kPitch, R>(w, ca, lane, dq);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = q0 + warp * R + i;
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        const int d = e * 32 + lane;
        if (row < p.S && d < p.D) p.dqkv[(size_t(b) * p.S + row) * stride + size_t(h0) * p.D + d] = __float2bfloat16(dq[i][e]);
      }
    }
    return;
  }
  if (h0 % group) return;
  const int k0 = (int(blockIdx.x) - tiles) * kRows;
  {
    SaTile<DP, kRows> tk, tv;
    tk.fetch(kbase, stride, k0, p.S, p.D);
    tv.fetch(vbase, stride, k0, p.S, p.D);
    tk.template put<kPitch>(ra);
    tv.template put<kPitch>(rb);
  }
  const int from = p.causal ? k0 / kSaCols * kSaCols : 0;
  float dk[R][kE] = {}, dv[R][kE] = {};
  ta.fetch(base + size_t(h0) * p.D, stride, from, p.S, p.D);
  tb.fetch(dbase + size_t(h0) * p.D, orow, from, p.S, p.D);
  for (int h = h0; h < h0 + group; ++h) {
    for (int q0 = from; q0 < p.S; q0 += kSaCols) {
      __syncthreads();
      ta.template put<kPitch>(ca);
      tb.template put<kPitch>(cb);
      const int row = q0 + lane;
      const float ls = row < p.S ? lbase[size_t(h) * p.S + row] : INFINITY;
      float dl = 0.f;
      __syncthreads();
      const bool more = q0 + kSaCols < p.S;
      if (more || h + 1 < h0 + group) {
        const int nh = more ? h : h + 1, nq = more ? q0 + kSaCols : from;
        ta.fetch(base + size_t(nh) * p.D, stride, nq, p.S, p.D);
        tb.fetch(dbase + size_t(nh) * p.D, orow, nq, p.S, p.D);
      }
      float s[R], dp[R];
      {
        float r[DP];
        sa_row<DP>(ca + lane * kPitch, r);
        sa_dots<DP, kPitch, R>(ra + warp * R * kPitch, r, s);
        sa_row<DP>(cb + lane * kPitch, r);
        if (row < p.S) {
          const float* o = obase + size_t(row) * orow + size_t(h) * p.D;
#pragma unroll
          for (int c = 0; c < DP; c += 4)
            if (c < p.D) {
              const float4 v = *reinterpret_cast<const float4*>(o + c);
              dl += r[c] * v.x + r[c + 1] * v.y + r[c + 2] * v.z + r[c + 3] * v.w;
            }
        }
        sa_dots<DP, kPitch, R>(rb + warp * R * kPitch, r, dp);
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int key = k0 + warp * R + i;
        const bool out = row >= p.S || key >= p.S || (p.causal && key > row);
        s[i] = out ? 0.f : exp2f(s[i] * sl2 - ls);
        dp[i] = out ? 0.f : s[i] * (dp[i] - dl) * p.scale;
      }
      sa_put<R>(w, lane, s);
      sa_put<R>(w + kSaCols * R, lane, dp);
      __syncwarp();
      sa_accumulate<DP, kPitch, R>(w, cb, lane, dv);
      sa_accumulate<DP, kPitch, R>(w + kSaCols * R, ca, lane, dk);
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = k0 + warp * R + i;
#pragma unroll
    for (int e = 0; e < kE; ++e) {
      const int d = e * 32 + lane;
      if (row < p.S && d < p.D) {
        __nv_bfloat16* at = p.dqkv + (size_t(b) * p.S + row) * stride + size_t(p.H + kvh) * p.D + d;
        at[0] = __float2bfloat16(dk[i][e]);
        at[size_t(p.Hkv) * p.D] = __float2bfloat16(dv[i][e]);
      }
    }
  }
}

template <int DP, int R>
static int launch_small(const SmallAttnParams& p, bool backward, cudaStream_t stream) {
  const int tiles = (p.S + 4 * R - 1) / (4 * R);
  if (!backward) return launch_overlapped(small_attn_fwd_kernel<DP, R>, dim3(tiles, p.H, p.B), kSaThreads, 0, stream, p);
  constexpr size_t kSmem = (2 * 4 * R + 2 * kSaCols) * (DP + 4) * 4 + kSaThreads / 32 * 2 * kSaCols * R * 4;
  static DeviceOnce configured;
  if (int e = configured.run([&] {
        return int(cudaFuncSetAttribute(small_attn_bwd_kernel<DP, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem)));
      }))
    return e;
  return launch_overlapped(small_attn_bwd_kernel<DP, R>, dim3(2 * tiles, p.H, p.B), kSaThreads, kSmem, stream, p, tiles);
}

// Four rows a warp while blocks of 16 rows are few to an SM: the chain of a step is half as long; eight share the broadcasts of a
// step among twice as many multiply-adds. us, forward and backward, heads of 32, 4 / 8 rows (torch operations before): 8 x 128, 4 heads
// 29, 31 (112); 2 x 300, 4 heads 45, 59 (129); 16 x 256, 12 heads 285, 239 (462); 2 x 2048, 16 heads 2548, 2072 (4159).
template <int DP>
static int small_attn(const SmallAttnParams& p, bool backward, cudaStream_t stream) {
  const long long blocks = (long long)((p.S + 15) / 16) * p.H * p.B;
  return blocks <= 8ll * sm_count() ? launch_small<DP, 4>(p, backward, stream) : launch_small<DP, 8>(p, backward, stream);
}

}  // namespace idrak

using namespace idrak;

// Attention over qkv [B, S, (H + 2 Hkv) D], D a multiple of 8 up to 64. Forward (dout null): out and o32 [B, S, H D], lse2
// [B, H, S]. Backward: dqkv like qkv, from dout, o32 and lse2 of the forward pass.
IDRAK_API int idrak_small_attention(const void* qkv, const void* dout, void* out, void* dqkv, float* o32, float* lse2, int B,
                                    int S, int H, int Hkv, int D, int causal, float scale, void* stream_) {
  if (D <= 0 || D > 64 || D % 8) return -2;
  if (Hkv <= 0 || H % Hkv) return -3;
  if (H > 65535 || B > 65535) return -4;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(dout)) & 15) return -5;
  if (B <= 0 || S <= 0) return 0;
  SmallAttnParams p{static_cast<const __nv_bfloat16*>(qkv), static_cast<const __nv_bfloat16*>(dout), static_cast<__nv_bfloat16*>(out),
                    static_cast<__nv_bfloat16*>(dqkv), o32, lse2, B, S, H, Hkv, D, causal, scale};
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (D <= 16) return small_attn<16>(p, dout != nullptr, stream);
  if (D <= 32) return small_attn<32>(p, dout != nullptr, stream);
  return small_attn<64>(p, dout != nullptr, stream);
}
