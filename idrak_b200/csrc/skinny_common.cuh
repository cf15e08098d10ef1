// Pieces shared by the few-row products (skinny_gemm.cu, skinny_packed.cu): cluster addressing, the epilogue, the choice of
// the K split.
#pragma once
#include "common.cuh"
#include <cstdlib>

namespace idrak {

__device__ __forceinline__ uint32_t sk_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t sk_map_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_addr), "r"(rank));
  return out;
}
__device__ __forceinline__ float sk_ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 sk_ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sk_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Brings a box into L2 and reads nothing: allowed before the kernels ahead have finished writing it.
__device__ __forceinline__ void sk_prefetch_2d(const CUtensorMap* m, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(m)), "r"(c0),
               "r"(c1)
               : "memory");
}

__device__ __forceinline__ float sk_gate(float g, int kind) {
  if (kind == 0) return g / (1.f + __expf(-g));
  if (kind == 1) return gelu_tanh(g);
  return fmaxf(g, 0.f);
}

// Where a few-row product goes, and what its epilogue adds.
struct SkinnyOut {
  __nv_bfloat16* C;              // [M, ldc]
  int ldc;
  const __nv_bfloat16* bias;     // [N] or null (gated: [2 N])
  const __nv_bfloat16* residual; // [M, ldr] or null
  int ldr;
  int M, N;                      // N = output features (gated: ff)
  int gate_kind;                 // -1: plain; else 0 silu, 1 gelu (tanh), 2 relu
  int up_offset;                 // gated: the weight's first up feature
  int up_index;                  // gated: its bias and int8 scale
};

// The end of a few-row product: each of the `csize` CTAs of a cluster holds the partial tile part[token][F] (rows kLd
// floats apart) of its K range; this CTA finishes the tokens rank, rank + csize, ...: it sums the partials in rank order
// through distributed shared memory, four features per 16-byte load, multiplies by factor(token, output) and runs the
// epilogue. Gated: features [0, F / 2) are gate, [F / 2, F) their up features. t = 0 .. 255. The cluster has met before.
template <int F, int kLd, class Factor>
__device__ __forceinline__ void sk_finish(const SkinnyOut& o, const float* part, int csize, int rank, int tile, int t,
                                          Factor factor) {
  constexpr int kHalf = F / 2;
  const bool gated = o.gate_kind >= 0;
  const int mine = (o.M - rank + csize - 1) / csize;
  const uint32_t part_addr = smem_u32(part);
  uint32_t peer[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) peer[r] = r < csize ? sk_map_rank(part_addr, r) : 0u;
  auto sum4 = [&](int m, int f, float (&v)[4]) {
    const uint32_t off = uint32_t((m * kLd + f) * 4);
    v[0] = v[1] = v[2] = v[3] = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < csize) {
        const float4 a = sk_ld_cluster4(peer[r] + off);
        v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
      }
    }
  };
  const int fours = (gated ? kHalf : F) / 4;
  const bool wide = (o.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(o.C) & 7) == 0;
  for (int idx = t; idx < mine * fours; idx += 256) {
    const int i = idx / fours, j = (idx - i * fours) * 4;
    const int m = rank + i * csize;
    const int n0 = (gated ? tile * kHalf : tile * F) + j;
    if (n0 >= o.N) continue;
    float v[4], u[4] = {0.f, 0.f, 0.f, 0.f};
    sum4(m, j, v);
    if (gated) sum4(m, kHalf + j, u);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int n = min(n0 + e, o.N - 1);
      v[e] *= factor(m, n);
      if (o.bias) v[e] += __bfloat162float(o.bias[n]);
      if (gated) {
        u[e] *= factor(m, o.up_index + n);
        if (o.bias) u[e] += __bfloat162float(o.bias[o.up_index + n]);
        v[e] = sk_gate(v[e], o.gate_kind) * u[e];
      }
      if (o.residual) v[e] += __bfloat162float(o.residual[size_t(m) * o.ldr + n]);
    }
    __nv_bfloat16* out = o.C + size_t(m) * o.ldc + n0;
    if (wide && n0 + 4 <= o.N) {
      *reinterpret_cast<uint2*>(out) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n0 + e < o.N) out[e] = __float2bfloat16(v[e]);
    }
  }
}

// skinny_packed.cu: few-row products over packed weights with the operands in registers, up to this many tokens.
constexpr int kSkinnyRegisterRows = 16;
int skinny_packed_registers(const __nv_bfloat16* X, int ldx, const void* codes, int ld, const __half* scales, int scale_ld,
                            int bits, int K, const SkinnyOut& o, cudaStream_t stream);

// IDRAK_SKINNY_SPLITS = 1 .. 8 overrides the K split of the few-row products (for measurements).
inline int skinny_forced_splits() {
  const char* e = getenv("IDRAK_SKINNY_SPLITS");
  const int f = e ? atoi(e) : 0;
  return f >= 1 && f <= 8 ? f : 0;
}

// Clusters of c CTAs of this kernel that the device holds at once (its SMs come in groups, and a cluster lives in one), by
// query; kept per kernel and size in `known` (one per kernel, zero at first).
template <class K>
int skinny_resident_clusters(K kern, int c, int threads, size_t smem, std::atomic<int> (&known)[9]) {
  int n = known[c].load(std::memory_order_relaxed);
  if (n > 0) return n;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(c));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(c);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = 1;
  }
  known[c].store(n, std::memory_order_relaxed);
  return n;
}

// The launch all of them use: clusters of c CTAs and programmatic serialization - the CTAs may start while the kernel
// before them in the stream drains; they stop at pdl_wait() before their first read of global memory. IDRAK_PDL=0 launches
// the ordinary way.
template <class K, class... A>
int skinny_launch(K kern, int grid, int c, int threads, size_t smem, cudaStream_t stream, const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(c);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  static const bool pdl = [] { const char* e = getenv("IDRAK_PDL"); return !(e && e[0] == '0'); }();
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  const int rc = int(cudaLaunchKernelEx(&cfg, kern, args...));
  note_launches(1);
  return rc;
}

}  // namespace idrak
