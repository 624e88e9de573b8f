// C entry points of the library that are also called from inside it (model.cu strings them into
// whole passes over a stack of transformer blocks). The definitions document the arguments.
#pragma once
#include <stddef.h>

extern "C" {
int gfs_gemm_bf16_rope(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda, int ldb,
                       int ldc, int ldr, int a_mn_major, int b_mn_major, int add, void* ws, size_t ws_bytes,
                       int force_split, const void* rope_cos, const void* rope_sin, int rope_cols, int rope_d,
                       int rope_b, void* stream);
int gfs_gemm2_bf16(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda, int ldb, int ldc,
                   int ldr, int a_mn_major, int b_mn_major, const void* rope_cos, const void* rope_sin, int rope_cols,
                   int rope_d, int rope_b, void* stream);
int gfs_gemm_bf16_swiglu(int mode, const void* a, const void* b, void* c, void* extra, int M, int I, int K, int lda,
                         int ldb, int ldc, int ld_extra, void* stream);
int gfs_gemm2_bf16_swiglu(int mode, const void* a, const void* b, void* c, void* extra, int M, int I, int K, int lda,
                          int ldb, int ldc, int ld_extra, void* stream);
int gfs_gemm2_wgrad_grouped(int n, const unsigned long long* A, const unsigned long long* B,
                            const unsigned long long* C, const int* M, const int* N, const int* K, const int* lda,
                            const int* ldb, const int* ldc, const int* accumulate, void* stream);
int gfs_gemm_tile(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda, int ldb, int ldc,
                  int ldr, int a_mn_major, int b_mn_major, const void* rope_cos, const void* rope_sin, int rope_cols,
                  int rope_d, int rope_b, int swi_mode, void* swi_extra, int swi_ld, int bn, int split, void* stream);
int gfs_gemm_tile_wgrad_grouped(int n, const unsigned long long* A, const unsigned long long* B,
                                const unsigned long long* C, const int* M, const int* N, const int* K, const int* lda,
                                const int* ldb, const int* ldc, const int* accumulate, int bn, int split, void* stream);
int gfs_linear(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda, int ldb, int ldc,
               int ldr, int a_mn_major, int b_mn_major, const void* rope_cos, const void* rope_sin, int rope_cols,
               int rope_d, int rope_b, int pair_min_tiles, void* stream);
int gfs_linear_swiglu(int mode, const void* a, const void* b, void* c, void* extra, int M, int I, int K, int lda,
                      int ldb, int ldc, int ld_extra, int pair_min_tiles, void* stream);
int gfs_wgrad_grouped(int n, const unsigned long long* A, const unsigned long long* B, const unsigned long long* C,
                      const int* M, const int* N, const int* K, const int* lda, const int* ldb, const int* ldc,
                      const int* accumulate, void* stream);
int gfs_rmsnorm_fwd(const void* x, const void* w, void* y, void* rstd, int rows, int H, float eps, void* stream);
int gfs_dropout_residual_norm(const void* z, const void* residual, void* x, const void* w, void* y, void* rstd, int rows,
                              int H, float eps, float p, unsigned long long seed, void* stream);
int gfs_rmsnorm_bwd_dropout(const void* dy, const void* x, const void* w, const void* rstd, const void* dres, void* dx,
                            void* dmask, void* partial, int rows, int H, float p, unsigned long long seed, void* stream);
int gfs_rmsnorm_bwd_parts(int rows);
int gfs_rmsnorm_bwd(const void* dy, const void* x, const void* w, const void* rstd, const void* dres, void* dx,
                    void* dw, void* partial, int rows, int H, int accumulate_dw, void* stream);
int gfs_rmsnorm_dw_reduce_multi(int n, const unsigned long long* partial, const unsigned long long* dw,
                                const int* parts, const int* accumulate, int H, void* stream);
int gfs_dropout_residual(const void* x, const void* residual, void* out, long long n, float p, unsigned long long seed,
                         int backward, void* stream);
int gfs_embedding_fwd(const void* ids, const void* W, void* out, int B, int S, int H, int v0, int v1, int s0,
                      int s_count, void* stream);
int gfs_embedding_sort_shift(long long n, int v);
int gfs_embedding_sort_keys(const void* ids_bs, void* keys, int B, int S, int v0, int v1, void* stream);
int gfs_embedding_bwd_keys(const void* keys, const void* dout, void* dW, int n, int H, int shift, void* stream);
int gfs_gemm2_ce_parts(int N);
int gfs_gemm2_bf16_ce(const void* A, const void* B, void* C, void* partials, int M, int N, int K, int lda, int ldb,
                      int ldc, void* stream);
int gfs_ce_fwd(const void* logits, const void* target, void* stats, void* lse, void* loss, int M, int Vp, long ld,
               int v0, int single_rank, int target_batch, void* rows_target, void* stream);
int gfs_ce_from_partials(const void* partials, const void* logits, const void* target, void* stats, void* lse,
                         void* loss, int parts, int M, int Vp, long ld, int v0, int single_rank, int target_batch,
                         void* rows_target, void* stream);
int gfs_ce_bwd(void* logits, const void* lse, const void* target, const void* grad_rows, float grad_all, int M, int Vp,
               long ld, int v0, void* stream);
int gfs_mean_f32(const void* x, void* out, int n, void* stream);
int gfs_flash_fwd(const void* q, const void* k, const void* v, void* o, void* o_copy, void* lse, int S, int B, int nh,
                  int D, const long long* strides, float scale, int causal, int o_f16, void* stream);
int gfs_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* dO, const void* lse,
                  void* dvec, void* dq, void* dk, void* dv, int S, int B, int nh, int D, const long long* strides,
                  float scale, int causal, const void* rope_cos, const void* rope_sin, void* do_bf16, void* stream);
}
