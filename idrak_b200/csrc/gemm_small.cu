// Small bf16 products, C[M, N] = epilogue(alpha * op(A) op(B)): the layers and gradients of a narrow model.
//
// Such a product is a chain of fixed costs. On the tcgen05 kernel (gemm_tcgen05.cu) the chain is tensor maps, barrier and
// tensor-memory set-up, TMA, MMA, tensor memory to registers to shared memory to TMA, and where K is cut to fill the machine the
// parts go through global memory to a second launch. Here a CTA has a tile of 64 x 64, copies its operands 16 bytes a lane
// into a ring of four blocks of 64 along K, takes them as they lie (ldmatrix, transposing where the operand is MN-major) into
// warp-level MMAs, and needs no set-up; K is cut over a cluster of up to 8, which sums the parts through distributed shared memory
// in rank order. The warp-level tensor path is the slower one (a K block takes 0.45 us alone on an SM, 0.3 in turn), so only
// products of few blocks come here. Eight warps of 32 x 16 and not four of 32 x 32: a block is a chain of waits for copies, fragments
// and MMAs, and the second warp of a scheduler fills them (K = 512: 7.2 -> 6.1 us). us, back to back, before and now:
//   1024 x 384 x 128          6.3, 4.1     its input gradient (K 384)    7.3, 5.1     its weight gradient (K 1024)   11.7, 6.0
//   200 x 1024 x 256          7.0, 4.6                       (K 1024)  11.9, 6.3                      (K 200)      6.8, 4.6
// The training step of a 4-layer model of width 128 on 1024 tokens: 837, 612. Launched the ordinary way: with programmatic
// serialization a chain of these back to back is faster, but in that step, among other kernels of 2 to 8 us, each took 1 us longer
// to start (612 -> 644, 714 where the others are launched so as well).
//
// Reference counterparts: gemm_tc_{nn,nt,tn,tt}_f32 (src/Idrak.Gpu/Cuda/PtxKernels.TensorCore.cs:24-29) at small sizes.
#include "gemm_epilogue.cuh"
#include "skinny_common.cuh"

namespace idrak {

constexpr int kSmT = 64, kSmK = 64, kSmStages = 4, kSmThreads = 256;
constexpr int kSmTile = kSmT * kSmK * 2;                       // 64 rows of 128 bytes, pieces exchanged by the row
constexpr int kSmLd = kSmT + 4;
constexpr int kSmBytes = kSmStages * 2 * kSmTile;
static_assert((kSmT * kSmLd + 9 * kSmT) * 4 <= kSmBytes, "the result passes through the ring");

// Column sums of the stored A (its rows summed over K: the bias gradient beside a weight gradient).
struct SmallSums {
  void* out;               // [M] bf16 or fp32
  int fp32, accumulate;
};

struct SmallOperand {
  const __nv_bfloat16* p;
  int ld, mn, extent;      // mn: stored [K, extent]; else [extent, K]
};

__device__ __forceinline__ void sm_ldmatrix(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void sm_ldmatrix_trans(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ uint32_t sm_at(int row, int piece) { return uint32_t(row * 128 + ((piece ^ (row & 7)) << 4)); }

// a block of an operand: 64 rows (of the matrix, or of K) of 64 elements; what lies outside is zero
template <int MN>
__device__ __forceinline__ void sm_load(const SmallOperand& o, int first, int k0, int K, uint32_t dst) {
#pragma unroll
  for (int i = 0; i < kSmT * 8 / kSmThreads; ++i) {
    const int c = int(threadIdx.x) + i * kSmThreads, r = c >> 3, piece = c & 7;
    const int row = MN ? k0 + r : first + r, col = (MN ? first : k0) + piece * 8;      // of the stored matrix
    const int rows = MN ? K : o.extent, cols = MN ? o.extent : K;
    const int bytes = row < rows ? max(0, min(16, (cols - col) * 2)) : 0;
    const __nv_bfloat16* src = bytes ? o.p + size_t(row) * o.ld + col : o.p;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + sm_at(r, piece)), "l"(src), "r"(bytes) : "memory");
  }
}

template <int A_MN, int B_MN, int SUMS>
__global__ void __launch_bounds__(kSmThreads)
small_gemm_kernel(const SmallOperand a, const SmallOperand b, const GemmParams p, const SmallSums sums) {
  extern __shared__ __align__(128) uint8_t sm_smem[];
  const uint32_t base = smem_u32(sm_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * kSmT, n0 = blockIdx.z * kSmT;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * 16;       // this warp's 32 x 16 of the tile
  const int csize = int(gridDim.x), rank = int(blockIdx.x);    // the cluster: the parts of K of one tile
  const int all = (p.K + kSmK - 1) / kSmK, first = all * rank / csize, blocks = all * (rank + 1) / csize;
  pdl_launch_dependents();                                     // what follows may be set up meanwhile
  auto issue = [&](int kb) {
    if (kb < blocks) {
      const uint32_t at = base + (kb % kSmStages) * 2 * kSmTile;
      sm_load<A_MN>(a, m0, kb * kSmK, p.K, at);
      sm_load<B_MN>(b, n0, kb * kSmK, p.K, at + kSmTile);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < kSmStages - 1; ++i) issue(first + i);
  float acc[2][2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
  const bool summing = SUMS && blockIdx.z == 0;                // one CTA of a row of tiles has every row of A pass through it
  float cs[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int kb = first; kb < blocks; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kSmStages - 2) : "memory");
    __syncthreads();                                           // block kb has landed; block kb - 1 has been read
    issue(kb + kSmStages - 1);
    const uint32_t sa = base + (kb % kSmStages) * 2 * kSmTile, sb = sa + kSmTile;
    if (summing) {                                             // 8 columns of the rows t / 8 and t / 8 + 32
      uint32_t w[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[i][0]), "=r"(w[i][1]), "=r"(w[i][2]), "=r"(w[i][3])
                     : "r"(sa + sm_at(int(threadIdx.x >> 3) + i * 32, int(threadIdx.x & 7))) : "memory");
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = unpack_bf16x2(w[0][e]), g = unpack_bf16x2(w[1][e]);
        cs[2 * e] += f.x + g.x;
        cs[2 * e + 1] += f.y + g.y;
      }
    }
#pragma unroll
    for (int ks = 0; ks < kSmK / 16; ++ks) {
      uint32_t fa[2][4], fb[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = wm + i * 16;
        if (A_MN) sm_ldmatrix_trans(fa[i], sa + sm_at(ks * 16 + (lane & 7) + ((lane >> 4) << 3), m / 8 + ((lane >> 3) & 1)));
        else sm_ldmatrix(fa[i], sa + sm_at(m + (lane & 15), ks * 2 + (lane >> 4)));
      }
      if (B_MN) sm_ldmatrix_trans(fb, sb + sm_at(ks * 16 + (lane & 7) + (((lane >> 3) & 1) << 3), wn / 8 + (lane >> 4)));
      else sm_ldmatrix(fb, sb + sm_at(wn + (lane & 7) + ((lane >> 4) << 3), ks * 2 + ((lane >> 3) & 1)));
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
              : "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3])
              : "r"(fa[i][0]), "r"(fa[i][1]), "r"(fa[i][2]), "r"(fa[i][3]), "r"(fb[j * 2]), "r"(fb[j * 2 + 1]));
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                             // nobody reads the ring any more
  float* out = reinterpret_cast<float*>(sm_smem);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = wm + i * 16 + (lane >> 2), c = wn + j * 8 + (lane & 3) * 2;
      *reinterpret_cast<float2*>(out + r * kSmLd + c) = make_float2(acc[i][j][0], acc[i][j][1]);
      *reinterpret_cast<float2*>(out + (r + 8) * kSmLd + c) = make_float2(acc[i][j][2], acc[i][j][3]);
    }
  float* csum = out + kSmT * kSmLd;                            // [8 warps][64], then the CTA's 64 sums
  if (summing) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      cs[e] += __shfl_xor_sync(0xffffffffu, cs[e], 8);
      cs[e] += __shfl_xor_sync(0xffffffffu, cs[e], 16);
      if (lane < 8) csum[warp * kSmT + lane * 8 + e] = cs[e];
    }
    __syncthreads();
    if (threadIdx.x < kSmT) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += csum[w * kSmT + threadIdx.x];
      csum[8 * kSmT + threadIdx.x] = s;
    }
    __syncwarp();
  }
  if (csize > 1) sk_cluster_sync();
  else __syncthreads();
  const int rows = kSmT / csize;                               // this CTA finishes these rows of the tile
  uint32_t peer[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) peer[r] = r < csize ? sk_map_rank(base, r) : 0u;
  for (int c = int(threadIdx.x); c < rows * 8; c += kSmThreads) {
    const int at = rank * rows + (c >> 3), row = m0 + at, col = n0 + (c & 7) * 8;
    if (row >= p.M || col >= p.N) continue;
    const uint32_t off = uint32_t(at * kSmLd + (c & 7) * 8) * 4;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < csize) {
        const float4 x = sk_ld_cluster4(peer[r] + off), y = sk_ld_cluster4(peer[r] + off + 16);
        v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w; v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] *= p.alpha;
    epilogue8(p, row, col, v, min(8, p.N - col));
  }
  if (summing && rank == 0 && threadIdx.x < kSmT && m0 + int(threadIdx.x) < p.M) {
    const int m = m0 + int(threadIdx.x);
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < csize) s += sk_ld_cluster(peer[r] + uint32_t((kSmT * kSmLd + 8 * kSmT + int(threadIdx.x)) * 4));
    if (sums.fp32) {
      float* o = static_cast<float*>(sums.out) + m;
      *o = sums.accumulate ? *o + s : s;
    } else {
      __nv_bfloat16* o = static_cast<__nv_bfloat16*>(sums.out) + m;
      *o = __float2bfloat16(sums.accumulate ? __bfloat162float(*o) + s : s);
    }
  }
  __syncwarp();
  if (csize > 1) sk_cluster_sync();                            // a peer may still read this CTA's part
}

template <int A_MN, int B_MN, int SUMS = 0>
static int launch_small(const SmallOperand& a, const SmallOperand& b, const GemmParams& p, int cuts, cudaStream_t stream,
                        const SmallSums& sums = SmallSums{}) {
  auto kern = small_gemm_kernel<A_MN, B_MN, SUMS>;
  static DeviceOnce configured;
  if (int e = configured.run([&] { return int(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmBytes)); })) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(cuts), unsigned((p.M + kSmT - 1) / kSmT), unsigned((p.N + kSmT - 1) / kSmT));
  cfg.blockDim = dim3(kSmThreads);
  cfg.dynamicSmemBytes = kSmBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(cuts);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cuts > 1 ? 1 : 0;
  const int rc = int(cudaLaunchKernelEx(&cfg, kern, a, b, p, sums));
  if (rc) cudaGetLastError();
  note_launches(1);
  return rc;
}

// How many CTAs share K of a tile here, or 0: the tcgen05 kernels. Measured over widths of 128 to 768 and 64 to 3072 rows, in us
// there / here (tiles x K blocks):
//  - the whole product is limited, tiles * blocks: one that K is not cut for there 96 x 4 6.9 / 5.4, 144 x 4 7.0 / 6.1, 48 x 12 9.4 / 8.0,
//    but 192 x 4 7.1 / 7.0, 96 x 8 8.2 / 8.3, 128 x 8 8.3 / 9.9; one that K is cut for 64 x 16 12.0 / 10.4, 48 x 24 24.4 / 11.1,
//    4 x 48 12.9 / 7.4, but 96 x 16 12.4 / 14.2, 64 x 48 20.0 / 17.6 (12.9 there once N is 256);
//  - the tiles are resident at once: 432 x 1 6.0 / 5.1, 576 x 1 6.1 / 7.5;
//  - K is cut as long as a part has two blocks and the parts leave SMs free: 32 x 8 in 1, 2, 4 parts 6.3, 5.5, 6.7; 16 x 16 in 1 to 8
//    10.2, 7.3, 6.1, 6.8. `ordered`: in one pass, in K order, as there, so that a row has the same bits whatever the number of rows.
int gemm_small_cuts(int M, int N, int K, bool ordered, bool cut_there) {
  const long long tiles = (long long)((M + kSmT - 1) / kSmT) * ((N + kSmT - 1) / kSmT);
  const int blocks = (K + kSmK - 1) / kSmK, sms = sm_count();
  if (tiles > 3 * sms || tiles * blocks > (cut_there ? 8 * sms : 4 * sms + sms / 3)) return 0;
  int cuts = 1;
  if (!ordered)
    while (cuts < 8 && tiles * cuts * 2 <= sms * 2 / 3 && blocks >= 4 * cuts) cuts *= 2;
  return (blocks + cuts - 1) / cuts <= 16 ? cuts : 0;
}

int gemm_small_launch(const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, GemmParams p, int cuts, cudaStream_t stream) {
  p.splits = 1;
  const SmallOperand a{static_cast<const __nv_bfloat16*>(A), lda, a_mn, p.M}, b{static_cast<const __nv_bfloat16*>(B), ldb, b_mn, p.N};
  if (!a_mn && !b_mn) return launch_small<0, 0>(a, b, p, cuts, stream);
  if (!a_mn && b_mn) return launch_small<0, 1>(a, b, p, cuts, stream);
  if (a_mn && !b_mn) return launch_small<1, 0>(a, b, p, cuts, stream);
  return launch_small<1, 1>(a, b, p, cuts, stream);
}

}  // namespace idrak

using namespace idrak;

// Whether idrak_weight_bias_grad takes a layer of these sizes: 1 or 0.
IDRAK_API int idrak_weight_bias_grad_fits(int tokens, int out_features, int in_features) {
  if (tokens <= 0 || out_features <= 0 || in_features <= 0) return 0;
  return gemm_small_cuts(out_features, in_features, tokens, false, gemm_cuts_k(out_features, in_features, tokens)) > 0 ? 1 : 0;
}

// dW (+)= dy^T x and db (+)= the column sums of dy, in one launch: dy [tokens, out], x [tokens, in], bf16, leading dimensions in
// elements and multiples of 8; dw [out, in] and db [out] in bf16 or fp32. For the sizes that idrak_weight_bias_grad_fits names. The
// sums are taken in fp32 from the blocks of dy that pass through shared memory anyway, by the CTAs of the first column of tiles; a
// pass of their own was two launches, 5 us beside a gradient of 6 (the training step named above: 603 us, now 547).
IDRAK_API int idrak_weight_bias_grad(const void* dy, int ld_dy, const void* x, int ld_x, void* dw, int ldw, int dw_fp32, int dw_accumulate,
                                     void* db, int db_fp32, int db_accumulate, int tokens, int out_features, int in_features, void* stream_) {
  if ((ld_dy & 7) || (ld_x & 7)) return -2;
  if ((reinterpret_cast<uintptr_t>(dy) & 15) || (reinterpret_cast<uintptr_t>(x) & 15)) return -3;
  if (!idrak_weight_bias_grad_fits(tokens, out_features, in_features)) return -4;
  const int cuts = gemm_small_cuts(out_features, in_features, tokens, false, gemm_cuts_k(out_features, in_features, tokens));
  GemmParams p{};
  p.M = out_features; p.N = in_features; p.K = tokens;
  p.C = dw; p.ldc = ldw; p.c_fp32 = dw_fp32;
  p.beta = dw_accumulate;
  p.alpha = 1.f;
  p.splits = 1;
  const SmallOperand a{static_cast<const __nv_bfloat16*>(dy), ld_dy, 1, p.M}, b{static_cast<const __nv_bfloat16*>(x), ld_x, 1, p.N};
  return launch_small<1, 1, 1>(a, b, p, cuts, static_cast<cudaStream_t>(stream_), SmallSums{db, db_fp32, db_accumulate});
}
