// The blocks of a decoder over the packed tokens of a prefill, as one call: (norm | qkv | norms of q and k, RoPE, cache write |
// attention of every prompt over its own keys | output projection + residual | norm | gate and up, activation | down + residual)
// per layer, the launches of the library's own entry points in the order in which the modules' forwards make them.
//
// A short prompt was bound by the host: 13 calls a layer from the interpreter at 20 to 30 us each. Four layers of 4096 x 14336 over
// 45 tokens took 1390 us for 650 us of kernels; a launch from here is 2 to 4 us.
//
// Reference counterpart: the prefill step of TextGenerator (src/Idrak/Generation/TextGenerator.cs:569-623), whose layers run
// as a recorded list of kernels as well.
#include "common.cuh"

extern "C" {
int idrak_norm_fwd(const void* x, const void* residual, const void* w, const void* b, void* out, void* sum_out, float* mean,
                   float* rstd, int rows, int C, float eps, int rms, void* stream_);
int idrak_gemm_few_rows(int M, int N, int K);
long long idrak_gemm_workspace_elems(int M, int N, int K);
int idrak_gemm_bf16(const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, void* C, int ldc, int c_fp32, int M, int N,
                    int K, const void* bias, const void* residual, int ldr, int act, void* aux, int ld_aux, int beta, float alpha,
                    int splits, float* workspace, int fp16, void* stream_);
int idrak_skinny_gemm(const void* X, int ldx, const void* W, int ldw, void* C, int ldc, int M, int N, int K, const void* bias,
                      const void* residual, int ldr, int gate_kind, float norm_eps, int one_pass, void* stream_);
int idrak_skinny_wide(const void* X, int ldx, const void* W, int ldw, void* C, int ldc, int M, int N, int K, const void* bias,
                      const void* residual, int ldr, int one_pass, void* stream_);
int idrak_norm_rope_kv(void* qkv, long long row_stride, const int* positions, const int* slots, void* k_cache, void* v_cache,
                       float* k_scale, float* v_scale, const void* q_norm, const void* k_norm, float eps, float theta,
                       float freq_scale, int rot_dim, int T, int H, int Hkv, int D, int kv_int8, void* stream_);
int idrak_flash_fwd_ex(const void* q, const void* k, const void* v, void* o, float* lse, int B, int H, int Hkv, int Sq, int Skv, int D,
                       long long q_row_stride, long long k_row_stride, long long v_row_stride, long long o_row_stride,
                       long long q_batch_stride, long long k_batch_stride, long long v_batch_stride, float scale, int causal, int window,
                       const int* row_start, float softcap, void* stream_);
int idrak_gated_fwd(const void* gu, void* out, int rows, int H, int kind, void* stream_);
}

namespace idrak {

// Pointers and settings of a layer; mirrored field by field in serve/native_prefill.py.
struct PrefillLayer {
  const void *attn_norm_w, *attn_norm_b, *qkv_w, *qkv_b, *q_norm, *k_norm, *o_w, *o_b;
  const void *mlp_norm_w, *mlp_norm_b, *up_w, *up_b, *down_w, *down_b;
  void *k_cache, *v_cache;
  float *k_scale, *v_scale;
  double attn_norm_eps, mlp_norm_eps, scale, theta;
  long long rot_dim;
};

struct PrefillArgs {
  const int *positions, *slots;
  const long long* prompts;      // [count][3]: first row, prompts of this length side by side, length
  void *x;                       // [tokens, dim]: the embedded tokens, then the result
  void *y, *normed;              // [tokens, dim]
  void *qkv, *attn;              // [tokens, (H + 2 Hkv) D], [tokens, H D]
  void *up, *act;                // [tokens, 2 ff], [tokens, ff]: may lie over qkv and attn
  float *mean, *rstd, *lse;      // [tokens], [tokens], [tokens, H]
  float* workspace;              // idrak_prefill_workspace floats
  long long tokens, dim, heads, kv_heads, head_dim, ff, count, attn_rms, mlp_rms, gate_kind, kv_int8;
  double qk_eps;
};

// x W^T (+ bias) (+ residual) on the kernel that ops.gemm takes for a product of this size.
static int product(const void* x, const void* w, void* out, int M, int N, int K, const void* bias, const void* residual, float* workspace,
                   void* stream) {
  const int few = idrak_gemm_few_rows(M, N, K);
  if (few == 3) return idrak_skinny_wide(x, K, w, K, out, N, M, N, K, bias, residual, residual ? N : 0, 0, stream);
  if (few)
    return idrak_skinny_gemm(x, K, w, K, out, N, M, N, K, bias, residual, residual ? N : 0, -1, -1.f, few == 2, stream);
  return idrak_gemm_bf16(x, K, 0, w, K, 0, out, N, 0, M, N, K, bias, residual, residual ? N : 0, 0, nullptr, 0, 0, 1.f, 0, workspace, 0,
                         stream);
}

}  // namespace idrak

using namespace idrak;

// fp32 workspace elements that the products of these sizes need.
IDRAK_API long long idrak_prefill_workspace(int tokens, int dim, int qkv, int out, int ff) {
  long long most = 0;
  const int sizes[4][2] = {{qkv, dim}, {dim, out}, {2 * ff, dim}, {dim, ff}};
  for (auto& s : sizes) {
    const long long n = idrak_gemm_workspace_elems(tokens, s[0], s[1]);
    most = n > most ? n : most;
  }
  return most;
}

// Returns 0 or the first error of a launch, with the layer in `failed_layer`.
IDRAK_API int idrak_prefill_blocks(const PrefillLayer* layers, int count, const PrefillArgs* args, int* failed_layer, void* stream) {
  const PrefillArgs& a = *args;
  const int T = int(a.tokens), dim = int(a.dim), H = int(a.heads), Hkv = int(a.kv_heads), D = int(a.head_dim), ff = int(a.ff);
  const int qkv_cols = (H + 2 * Hkv) * D;
  char* qkv = static_cast<char*>(a.qkv);
  char* attn = static_cast<char*>(a.attn);
  for (int i = 0; i < count; ++i) {
    const PrefillLayer& l = layers[i];
    *failed_layer = i;
    int rc = idrak_norm_fwd(a.x, nullptr, l.attn_norm_w, l.attn_norm_b, a.normed, nullptr, a.mean, a.rstd, T, dim, float(l.attn_norm_eps),
                            int(a.attn_rms), stream);
    if (!rc) rc = product(a.normed, l.qkv_w, a.qkv, T, qkv_cols, dim, l.qkv_b, nullptr, a.workspace, stream);
    if (!rc)
      rc = idrak_norm_rope_kv(a.qkv, qkv_cols, a.positions, a.slots, l.k_cache, l.v_cache, l.k_scale, l.v_scale, l.q_norm, l.k_norm,
                              float(a.qk_eps), float(l.theta), 1.f, int(l.rot_dim), T, H, Hkv, D, int(a.kv_int8), stream);
    for (long long p = 0; p < a.count && !rc; ++p) {
      const long long first = a.prompts[3 * p], many = a.prompts[3 * p + 1], len = a.prompts[3 * p + 2];
      char* q = qkv + first * qkv_cols * 2;
      rc = idrak_flash_fwd_ex(q, q + (long long)H * D * 2, q + (long long)(H + Hkv) * D * 2, attn + first * H * D * 2, a.lse, int(many), H, Hkv,
                              int(len), int(len), D, qkv_cols, qkv_cols, qkv_cols, (long long)H * D, len * qkv_cols, len * qkv_cols,
                              len * qkv_cols, float(l.scale), 1, 0, nullptr, 0.f, stream);
    }
    if (!rc) rc = product(a.attn, l.o_w, a.y, T, dim, H * D, l.o_b, a.x, a.workspace, stream);
    if (!rc)
      rc = idrak_norm_fwd(a.y, nullptr, l.mlp_norm_w, l.mlp_norm_b, a.normed, nullptr, a.mean, a.rstd, T, dim, float(l.mlp_norm_eps),
                          int(a.mlp_rms), stream);
    if (!rc) rc = product(a.normed, l.up_w, a.up, T, 2 * ff, dim, l.up_b, nullptr, a.workspace, stream);
    if (!rc) rc = idrak_gated_fwd(a.up, a.act, T, ff, int(a.gate_kind), stream);
    if (!rc) rc = product(a.act, l.down_w, a.x, T, dim, ff, l.down_b, a.y, a.workspace, stream);
    if (rc) return rc;
  }
  return 0;
}
