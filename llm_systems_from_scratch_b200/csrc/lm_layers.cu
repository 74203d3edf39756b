// All layers of one serving step of the TransformerLM from one call: the same launches, in the same order and with the same arguments, that
// the ops make one by one.  A launch through Python takes the host about 13 us, which is what bounds short prompts (200 tokens, 24 layers of
// 2048: 2845 us op by op, 2300 from here, when the device needed that).
// Which kernel a product takes is decided by the caller (`LmProduct`), once per step.
#include "gemm_common.cuh"

using namespace b200;

extern "C" {
int b200_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int rows, int d, float eps, cudaStream_t st);
int b200_gemm_bf16(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda, long long ldb, long long ldc,
                   long long ldr, int a_mn, int b_mn, int epi, int bn_hint, int max_ctas, uint32_t* status, cudaStream_t stream);
int b200_gemm_bf16_pair(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda, long long ldb, long long ldc,
                        long long ldr, int a_mn, int b_mn, int epi, uint32_t* status, cudaStream_t stream);
int b200_gemm_bf16_splitk(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda, long long ldb,
                          long long ldc, long long ldr, int epi, float* ws, long long ws_floats, uint32_t* tile_counters, int n_counters,
                          uint32_t* status, cudaStream_t stream);
int b200_gemm_few_rows(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda, long long ldb, long long ldc,
                       long long ldr, int epi, int splits, const GemmFinish* finish, uint32_t* status, cudaStream_t stream);
int b200_gemm_bf16_append(const void* A, const void* B, void* C, int M, int K, long long lda, long long ldb, long long ldc, int epi,
                          const QkvAppend* append, uint32_t* status, cudaStream_t stream);
int b200_rope_kv_append(void* qkv, const float* cos_sin, const int* positions, void* k_cache, void* v_cache, const long long* slots,
                        long long rows, int d, int dh, int ctx, long long num_slots, uint32_t* status, cudaStream_t st);
int b200_flash_varlen_fwd(const void* qkv, void* o, const int* cu_seqlens, int batch, int max_seq, int total_rows, int heads, int dh,
                          float scale, uint32_t* status, cudaStream_t stream);
int b200_paged_decode(const void* q, const void* k_cache, const void* v_cache, const int* block_tables, const int* context_lens, void* out,
                      float* part_o, float* part_ml, int rows, int q_ld, int heads, int dh, int page_size, int max_pages, int splits,
                      float scale, int num_pages, uint32_t* status, cudaStream_t st);
int b200_silu_mul_fwd(const void* gu, void* h, long long rows, int F, cudaStream_t st);
int b200_gemm_bf16_pair_swiglu(const void* A, const void* B, void* C, void* H, int M, int F, int K, long long lda, long long ldb, long long ldc,
                               long long ldh, const unsigned long long* src_ptrs, void* gather_dst, unsigned long long shard_bytes, int world,
                               int rank, uint32_t* status, cudaStream_t stream);
int b200_gemm_bf16_grouped(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda, long long ldb,
                           long long ldc, long long ldr, const int* tile_group, int n_groups, int group_rows, int batch, int a_step, int c_step,
                           int swiglu, int epi, int head_gate, int most, const GemmFinish* finish, uint32_t* status,
                           cudaStream_t stream);
}

// Passed by pointer through the C interface: the field order is part of it.
struct LmProduct {
  int kind;                    // 0 single CTAs, 1 CTA pairs, 2 sliced through the workspace, 3 few rows (`slices` of K)
  int slices;
};
struct LmLayer {
  const void *wqkv, *wo, *wgu, *wdown, *n1, *n2;
  void *k, *v;                 // cache
};
enum LmGlu : int { LM_GLU_PAIR = 0, LM_GLU_GROUPED = 1, LM_GLU_ROUNDED = 2 };      // ROUNDED: product to `gu`, then silu_mul
struct LmStep {
  const LmLayer* layers;
  void *x, *y;                 // residual stream (rows, d): in, and scratch; the result is in x
  void *h, *qkv, *o, *gu, *act;        // (rows, d), (rows, 3 d), (rows, d), (rows, 2 ff) or null, (rows, ff)
  float* rstd;
  const float* cos_sin;
  const int* positions;
  const long long* slots;
  const int *cu, *tables, *ctx_lens;   // attention among the step's rows (cu), or through the cache (cu null)
  float *part_o, *part_ml, *ws;
  uint32_t *counters, *status;
  long long num_slots, ws_floats;
  int n_layers, rows, d, heads, ff, rope_ctx, batch, max_seq, page_size, max_pages, splits, num_pages, n_counters, append, glu;
  float eps, scale;
  LmProduct pqkv, po, pgu, pdown;
};

static int lm_product(const LmStep& s, const LmProduct& p, const void* a, const void* w, void* c, const void* res, int n, int k, cudaStream_t st) {
  const int epi = res != nullptr ? EPI_BF16_RES : EPI_BF16;
  const long long ldr = res != nullptr ? n : 0;
  switch (p.kind) {
    case 0: return b200_gemm_bf16(a, w, c, res, s.rows, n, k, k, k, n, ldr, 0, 0, epi | EPI_B_STABLE, 0, 0, s.status, st);
    case 1: return b200_gemm_bf16_pair(a, w, c, res, s.rows, n, k, k, k, n, ldr, 0, 0, epi, s.status, st);
    case 2: return b200_gemm_bf16_splitk(a, w, c, res, s.rows, n, k, k, k, n, ldr, epi | EPI_B_STABLE, s.ws, s.ws_floats, s.counters, s.n_counters, s.status, st);
    case 3: return b200_gemm_few_rows(a, w, c, res, s.rows, n, k, k, k, n, ldr, epi | EPI_B_STABLE, p.slices, nullptr, s.status, st);
  }
  return -11;
}

// All matrices row-major without gaps.  Returns the number of launches, or a launch's error.
extern "C" int b200_lm_layers(const LmStep* step, cudaStream_t st) {
  const LmStep& s = *step;
  if (s.rows <= 0 || s.heads <= 0 || s.d % s.heads) return -10;
  const int dh = s.d / s.heads;
  int launches = 0;
#define LM(call)                 \
  do {                           \
    const int rc_ = (call);      \
    if (rc_) return rc_;         \
    ++launches;                  \
  } while (0)
  for (int i = 0; i < s.n_layers; ++i) {
    const LmLayer& w = s.layers[i];
    LM(b200_rmsnorm_fwd(s.x, w.n1, s.h, s.rstd, s.rows, s.d, s.eps, st));
    if (s.append) {
      const QkvAppend a = {s.cos_sin, s.positions, s.slots, (__nv_bfloat16*)w.k, (__nv_bfloat16*)w.v, s.num_slots, s.d, dh, s.rope_ctx};
      LM(b200_gemm_bf16_append(s.h, w.wqkv, s.qkv, s.rows, s.d, s.d, s.d, 3ll * s.d, EPI_B_STABLE, &a, s.status, st));
    } else {
      LM(lm_product(s, s.pqkv, s.h, w.wqkv, s.qkv, nullptr, 3 * s.d, s.d, st));
      LM(b200_rope_kv_append(s.qkv, s.cos_sin, s.positions, w.k, w.v, s.slots, s.rows, s.d, dh, s.rope_ctx, s.num_slots, s.status, st));
    }
    if (s.cu != nullptr) {
      LM(b200_flash_varlen_fwd(s.qkv, s.o, s.cu, s.batch, s.max_seq, s.rows, s.heads, dh, s.scale, s.status, st));
    } else {
      LM(b200_paged_decode(s.qkv, w.k, w.v, s.tables, s.ctx_lens, s.o, s.part_o, s.part_ml, s.rows, 3 * s.d, s.heads, dh, s.page_size, s.max_pages,
                           s.splits, s.scale, s.num_pages, s.status, st));
    }
    LM(lm_product(s, s.po, s.o, w.wo, s.y, s.x, s.d, s.d, st));
    LM(b200_rmsnorm_fwd(s.y, w.n2, s.h, s.rstd, s.rows, s.d, s.eps, st));
    // -13: the TMA-store epilogue is switched off; the other kernel then
    const int paired = s.glu != LM_GLU_PAIR ? -13 : b200_gemm_bf16_pair_swiglu(s.h, w.wgu, nullptr, s.act, s.rows, s.ff, s.d, s.d, s.d, 0, s.ff, nullptr,
                                                                               nullptr, 0, 0, 0, s.status, st);
    if (paired != -13) {
      LM(paired);
    } else if (s.glu != LM_GLU_ROUNDED) {
      LM(b200_gemm_bf16_grouped(s.h, w.wgu, s.act, nullptr, s.rows, s.ff, s.d, s.d, s.d, s.ff, 0, nullptr, 0, 2 * s.ff, 1, 0, 0, 1, EPI_B_STABLE, 0,
                                0, nullptr, s.status, st));
    } else {
      LM(lm_product(s, s.pgu, s.h, w.wgu, s.gu, nullptr, 2 * s.ff, s.d, st));
      LM(b200_silu_mul_fwd(s.gu, s.act, s.rows, s.ff, st));
    }
    LM(lm_product(s, s.pdown, s.act, w.wdown, s.x, s.y, s.d, s.ff, st));
  }
#undef LM
  return launches;
}
