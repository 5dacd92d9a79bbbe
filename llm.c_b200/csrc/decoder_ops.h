// Entry points that csrc/decoder.cu calls from the other files.  Their definitions include this header too: an argument list that changes on one side
// alone does not compile (C linkage has no argument types to tell the two apart).
#pragma once
#include "common.cuh"

extern "C" {
int llmc_encoder_fwd(bf16* out, const int* tokens, const bf16* wte, const bf16* wpe, int B, int T, int C, int V, cudaStream_t stream);
int llmc_rmsnorm_fwd(bf16* out, float* rstd, const bf16* inp, const bf16* weight, int N, int C, float eps, cudaStream_t stream);
int llmc_rmsnorm_fused_residual_fwd(bf16* residual, bf16* normed, float* rstd, const bf16* inp1, const bf16* inp2, const bf16* weight, int N, int C,
                                    float eps, cudaStream_t stream);
int llmc_rope_fwd_cache(bf16* packed, const bf16* raw, const float* freqs, bf16* kcache, bf16* vcache, int cache_len, long long N, int T, int NH, int NKV,
                        int HS, cudaStream_t stream);
int llmc_rope_cache(bf16* q, bf16* kcache, bf16* vcache, const bf16* raw, const float* freqs, int freqs_len, int B, int Tq, int Tmax, int start_pos,
                    int NH, int NKV, int HS, const int* pos_ptr, cudaStream_t stream);
int llmc_attention_fwd(bf16* out, float* lse, const bf16* qkv, int B, int T, int NH, int hs, cudaStream_t stream);
int llmc_cached_attention(bf16* out, const bf16* q, const bf16* kcache, const bf16* vcache, int B, int Tq, int Tmax, int start_pos, int NH, int NKV,
                          int HS, const int* pos_ptr, float* ws, cudaStream_t stream);
int llmc_cached_attention_rope(bf16* out, const bf16* raw, const float* freqs, int freqs_len, bf16* kcache, bf16* vcache, int B, int Tq, int Tmax,
                               int start_pos, int NH, int NKV, int HS, const int* pos_ptr, float* ws, int early, cudaStream_t stream);
int llmc_swiglu_fwd(bf16* h, const bf16* x12, long long N, int H, cudaStream_t stream);
int llmc_stream_gemm_chained(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, int form, cudaStream_t stream);
int llmc_stream_gemm_logits(float* out, int cols, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int* advance, cudaStream_t stream);
int llmc_stream_gemm_swiglu_chained(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream);
int llmc_gemm2t_chained(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream);
int llmc_gemm2t_swiglu_chained(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream);
int llmc_gemm2(const bf16* A, const bf16* B, bf16* D, const bf16* bias, bf16* aux, int M, int N, int K, int lda, int ldb, int ldd, int a_mn_major,
               int b_mn_major, int mode, int accumulate, int splits, float* workspace, unsigned int* counters, cudaStream_t stream);
int llmc_gemm(const bf16* A, const bf16* B, bf16* D, const bf16* bias, bf16* aux, int M, int N, int K, int lda, int ldb, int ldd, int a_mn_major,
              int b_mn_major, int mode, int accumulate, int splits, float* workspace, unsigned int* counters, int max_ctas, cudaStream_t stream);
}
