// The C entry points of libtb200_cuda.so that the operators call: the .cu files define them, csrc/ops.cpp calls them through
// pointers of these types, tandem_b200/ops through ctypes.  What each one does is said where it is defined.
// They return 0, a negative code of this library or a positive cudaError_t, unless said otherwise.
#pragma once
#include <cuda_runtime_api.h>

#ifdef __cplusplus
extern "C" {
#endif

// symm.cu
const char* tb_last_error();
const char* tb_error_string(int code);

// gemm.cu
int tb_gemm_error();
const char* tb_gemm_last_error();
void tb_gemm_force_tile(int which);
void tb_gemm_tma_store(int on);
void tb_gemm_force_splits(int n);
void tb_gemm_plan(int M, int N, int K, int* out4);
long long tb_gemm_workspace_bytes(int M, int N, int K);
int tb_gemm_bf16(const void* A, const void* B, void* out, int M, int N, int K, int lda, int ldb, int ldc, int a_mn, int b_mn, int flags,
                 const void* bias, const void* aux_in, void* aux_out, int max_ctas, void* workspace, long long workspace_bytes,
                 cudaStream_t stream);
int tb_gemm_gathered(const void* A, void* out, int M, int N, int K, int lda, int ldc, int flags, const void* bias, const void* aux_in,
                     void* aux_out, void* const* shards, const long long* shard_lo, const long long* shard_hi, int n_ranks, void* full,
                     long long w_off, long long tail_bytes, void* ready, unsigned epoch, int chunk_bytes, int n_start,
                     cudaStream_t stream);
int tb_gemm_reciprocals(const float* d, float* out, long long n, cudaStream_t stream);

// attention.cu
int tb_attn_error();
int tb_attn_fwd(const void* qkv, void* out, float* lse, int B, int T, int H, int HD, cudaStream_t stream);
int tb_attn_bwd(const void* qkv, const void* out, const void* d_out, const float* lse, void* dqkv, float* delta, int B, int T, int H, int HD,
                cudaStream_t stream);

// layers.cu
int tb_stream_wait(cudaStream_t waiter, cudaStream_t signaller);
int tb_stream_wait_events();
int tb_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, int M, int D, float eps,
                     cudaStream_t stream);
int tb_layernorm_bwd_blocks(int M);
int tb_layernorm_bwd(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, void* dx, void* dw,
                     void* db, float* scratch, int M, int D, cudaStream_t stream);
int tb_layernorm_bwd_add(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, const void* add, void* dx,
                         void* dw, void* db, float* scratch, int M, int D, cudaStream_t stream);
int tb_col_sum(const void* x, int M, int N, int ld, void* out_bf16, float* scratch, cudaStream_t stream);
int tb_xent_fwd(const void* logits, const long long* targets, float* lse, float* row_loss, float* loss, int rows, int V, int ld,
                cudaStream_t stream);
int tb_xent_bwd(void* logits, const long long* targets, const float* lse, const float* grad_scale, int rows, int V, int ld,
                int width, cudaStream_t stream);
int tb_embed_fwd(const long long* idx, const void* tok, const void* pos, void* out, int rows, int T, int D, cudaStream_t stream);
int tb_embed_bwd(const long long* idx, const void* dy, float* dtok32, void* dtok, void* dpos, int B, int T, int D, int V,
                 cudaStream_t stream);

#ifdef __cplusplus
}
#endif
