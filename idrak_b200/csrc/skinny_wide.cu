// Products of 65 to 256 rows (a large decode batch, a prompt of a page): C[M, N] = X[M, K] W[N, K]^T, bound by streaming W once.
//
// As in skinny_gemm.cu the product is computed transposed, weights on the 128-row side of the tensor-core tile, and the CTAs of a
// cluster split K and sum their parts through distributed shared memory in rank order. Here a CTA has 256 output features - two
// accumulators of 128 x NT, NT the rows rounded up to 16 - so that a block of X, which every CTA reads again from L2, is paid by
// twice the weights: at 160 rows 0.6 bytes of X for each of W, where 128 features would take 1.25 and the dense kernel's
// 256 x 256 tiles compute and store 256 rows whatever there are. One CTA has an SM to itself and the partial sums pass through
// the operand ring's memory 128 rows at a time.
//
//   warp 0      TMA producer: two W tiles and the X tile of a K block (64) per stage
//   warp 1      MMA issuer
//   warps 2..9  move the accumulators to shared memory and finish the rows (skinny_common.cuh)
//
// Launched with programmatic serialization, the first weight blocks on their way into L2 while the kernels ahead finish.
// Measured, us, dense kernel and this, with residual, at 65 / 128 / 160 rows: 6144 x 4096 24.9, 18.1 / 29.3, 21.5 / 25.6, 24.6; 4096 x
// 14336 39.6, 34.1 / 43.0, 37.5 / 43.0, 41.6; 768 x 3072 14.0, 9.9 / 16.7, 12.3 / 25.6, 15.4. What bounds it is what an SM draws from
// L2, some 43 bytes a cycle, and the rows' passes at the end.
//
// Every mbarrier wait is bounded; every thread reaches every cluster barrier whatever happened before.
//
// Reference counterparts: gemm_tc_nt_f32 (src/Idrak.Gpu/Cuda/PtxKernels.TensorCore.cs:24-29) at these sizes.
#include "skinny_common.cuh"

namespace idrak {

constexpr int kWdFeat = 256, kWdBK = 64, kWdThreads = 320;
constexpr int kWdLd = kWdFeat + 4;            // floats of a row of the partial sums
constexpr int kWdRows = 128;                  // rows of a pass
constexpr int kWdMaxStages = 8;
constexpr int kWdW = kWdFeat * kWdBK * 2;     // weights of a stage

struct SkinnyWideParams {
  SkinnyOut o;
  int K, nt, stages, csize;
  Status* st;
};

__global__ void __launch_bounds__(kWdThreads, 1)
skinny_wide_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SkinnyWideParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int NT = p.nt, kStages = p.stages, kStage = kWdW + NT * kWdBK * 2;
  float* part = reinterpret_cast<float*>(smem);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStage);
  uint64_t* empty = full + kWdMaxStages;
  uint64_t* acc_full = empty + kWdMaxStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int csize = p.csize, rank = int(sk_cluster_rank()), tile = blockIdx.x / csize;
  const int kblocks = (p.K + kWdBK - 1) / kWdBK;
  const int kb0 = int((long long)kblocks * rank / csize), kb1 = int((long long)kblocks * (rank + 1) / csize);

  pdl_launch_dependents();
  auto issue = [&](int kb, int stage) {
    uint8_t* at = smem + stage * kStage;
    mbar_expect_tx(&full[stage], kStage);
    tma_load_2d(at, &tmW, &full[stage], kb * kWdBK, tile * kWdFeat);
    tma_load_2d(at + kWdW / 2, &tmW, &full[stage], kb * kWdBK, tile * kWdFeat + 128);
    tma_load_2d(at + kWdW, &tmX, &full[stage], kb * kWdBK, 0);
  };
  const int first = min(kStages, kb1 - kb0);            // stages filled before the CTA-wide sync (all are free then)
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    for (int i = 0; i < first; ++i) {
      sk_prefetch_2d(&tmW, (kb0 + i) * kWdBK, tile * kWdFeat);
      sk_prefetch_2d(&tmW, (kb0 + i) * kWdBK, tile * kWdFeat + 128);
    }
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    fence_barrier_init();
    pdl_wait();                                          // the kernels before this one have written the rows
    for (int i = 0; i < first; ++i) issue(kb0 + i, i);   // in flight while tensor memory is allocated below
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();                                            // every thread that reads global memory (bias, residual)
  const uint32_t tmem_acc = *tmem_slot;                  // the features' halves at columns 0 and 256
  bool ok = true;

  if (warp == 0) {
    if (lane == 0) {
      int stage = first % kStages;
      uint32_t phase = first == kStages ? 1u : 0u;
      for (int kb = kb0 + first; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.st, kTimeoutSmemEmpty, (11u << 16) | stage)) {
          ok = false;
          break;
        }
        issue(kb, stage);
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
      if (!ok || *abort_flag) {                          // let the copies on their way land before the ring is reused
        const uint64_t from = global_timer_ns();
        while (global_timer_ns() - from < 200000ull) { }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_f16(128, NT, 0, 0, 1);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full[stage], phase, abort_flag, p.st, kTimeoutSmemFull, (11u << 16) | (16 + stage))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sw = smem_u32(smem + stage * kStage), sx = sw + kWdW;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int kk = 0; kk < kWdBK / 16; ++kk)
            tc_mma_f16_ss(tmem_acc + h * 256, make_smem_desc_sw128(sw + h * (kWdW / 2) + kk * 32, 16, 1024),
                          make_smem_desc_sw128(sx + kk * 32, 16, 1024), idesc, (kb > kb0 || kk > 0) ? 1u : 0u);
        tc_commit(&empty[stage]);
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
      if (ok) tc_commit(acc_full);
    }
  }

  const bool have = kb1 > kb0;
  if (warp >= 2) {
    if (have) ok = mbar_wait(acc_full, 0, abort_flag, p.st, kTimeoutTmemFull, (11u << 16) | 60);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
  }
  const int q = warp & 3;                                // the TMEM lane quarter this warp may read
  const int set = (warp - 2) >> 2;                       // which half of the features it moves
  for (int r0 = 0; r0 < p.o.M; r0 += kWdRows) {
    if (warp >= 2) {
      const int rows = min(kWdRows, NT - r0), f = set * 128 + q * 32 + lane;
      for (int c = 0; c < rows; c += 16) {
        uint32_t v[16];
        if (have && ok) {
          tmem_ld_32x32b_x16(tmem_acc + (uint32_t(q * 32) << 16) + set * 256 + r0 + c, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0u;        // no K blocks here, or gave up
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) part[(c + i) * kWdLd + f] = __uint_as_float(v[i]);
      }
      tc_fence_before();
    }
    // every thread of every CTA of the cluster: the pass's partial sums are complete and visible
    __syncwarp();
    sk_cluster_sync();
    if (warp >= 2) {
      SkinnyOut o = p.o;
      o.M = min(kWdRows, p.o.M - r0);
      o.C += size_t(r0) * o.ldc;
      if (o.residual) o.residual += size_t(r0) * o.ldr;
      sk_finish<kWdFeat, kWdLd>(o, part, csize, rank, tile, int(threadIdx.x) - 64, [](int, int) { return 1.f; });
    }
    // nobody overwrites them or leaves while a peer may still read its shared memory
    __syncwarp();
    sk_cluster_sync();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_acc, 512);
  }
}

}  // namespace idrak

using namespace idrak;

// C[M, N] (bf16) = X[M, K] W[N, K]^T (+ bias) (+ residual), 1 <= M <= 256; K % 8 == 0, rows of X and W on 16-byte boundaries.
// one_pass: K is not cut. Returns 0, a CUDA error, or a negative argument error.
IDRAK_API int idrak_skinny_wide(const void* X, int ldx, const void* W, int ldw, void* C, int ldc, int M, int N, int K, const void* bias,
                                const void* residual, int ldr, int one_pass, void* stream_) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > 256) return -2;
  if ((K & 7) || (ldx & 7) || (ldw & 7)) return -3;
  if ((reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(W) & 15)) return -4;
  SkinnyWideParams p{};
  p.o = {static_cast<__nv_bfloat16*>(C), ldc, static_cast<const __nv_bfloat16*>(bias), static_cast<const __nv_bfloat16*>(residual), ldr, M, N,
         -1, 0, 0};
  p.K = K;
  p.nt = (M + 15) / 16 * 16;
  const int stage = kWdW + p.nt * kWdBK * 2;
  constexpr int kBars = 512;
  p.stages = min(kWdMaxStages, (232448 - 1024 - kBars) / stage);
  static_assert(kWdRows * kWdLd * 4 <= 3 * (kWdW + 16 * kWdBK * 2) || kWdRows * kWdLd * 4 <= 184 * 1024, "a pass fits in the ring");
  p.st = status_device_ptr();
  CUtensorMap tmW, tmX;
  uint64_t dims[2] = {uint64_t(K), uint64_t(N)}, strides[1] = {uint64_t(ldw) * 2};
  uint32_t box[2] = {uint32_t(kWdBK), 128};
  if (encode_tensor_map(&tmW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(W), dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
    return -10;
  uint64_t xdims[2] = {uint64_t(K), uint64_t(M)}, xstrides[1] = {uint64_t(ldx) * 2};
  uint32_t xbox[2] = {uint32_t(kWdBK), uint32_t(p.nt)};
  if (encode_tensor_map(&tmX, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(X), xdims, xstrides, xbox, CU_TENSOR_MAP_SWIZZLE_128B))
    return -11;
  const size_t smem = size_t(p.stages) * stage + kBars + 1024;
  static DeviceOnce configured;
  static std::atomic<int> known[9];
  if (int e = configured.run([&] { return int(cudaFuncSetAttribute(skinny_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448)); }))
    return e;
  const int tiles = (N + kWdFeat - 1) / kWdFeat, kblocks = (K + kWdBK - 1) / kWdBK;
  int c = one_pass ? 1 : min(8, kblocks);
  while (c > 1 && skinny_resident_clusters(skinny_wide_kernel, c, kWdThreads, 232448, known) < tiles) --c;
  p.csize = c;
  return skinny_launch(skinny_wide_kernel, tiles * c, c, kWdThreads, smem, static_cast<cudaStream_t>(stream_), tmW, tmX, p);
}
