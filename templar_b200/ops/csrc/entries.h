// Entry points of the kernel library that the autograd nodes in C++ call (csrc_host/autograd.cpp), declared once: the CUDA
// sources define them against these declarations and the nodes take the types of their function pointers from them, so that a
// changed argument list does not compile on either side alone.  The builder hands both a number made from this file
// (TPLR_ABI), and the nodes refuse a library with another one.
#pragma once

extern "C" {
int tplr_abi();
int tplr_add_rmsnorm_fwd(const void* res, const void* delta, const void* w, void* h_out, void* y, float* rstd, long long T, int D,
                         float eps, void* stream);
int tplr_add_rmsnorm_bwd_v2(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx, float* dw,
                            long long T, int D, unsigned int* status, void* stream);
int tplr_gemm2_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int a_mn,
                    int b_mn, int epi, unsigned int* status, int max_pairs, void* stream);
int tplr_gemm2_acc_splits(int M, int N, int K);
int tplr_gemm2_acc_split(const void* A, const void* B, float* C, float* ws, int M, int N, int K, long long lda, long long ldb,
                         long long ldc, int a_mn, int b_mn, unsigned int* status, void* stream);
int tplr_gemm2_out_splits(int M, int N, int K);
int tplr_gemm2_bf16_split(const void* A, const void* B, void* C, float* ws, int M, int N, int K, long long lda, long long ldb,
                          long long ldc, int a_mn, int b_mn, unsigned int* status, void* stream);
int tplr_gemm2_swiglu(const void* X, const void* W, void* GU, void* H, int M, int F, int K, long long ldx, long long ldw, long long ldgu,
                      long long ldh, unsigned int* status, void* stream);
int tplr_gemm2_swiglu_bwd(const void* dY, const void* W2, const void* GU, void* dGU, int M, int F, int K, long long lddy,
                          long long ldw2, long long ldgu, long long lddgu, unsigned int* status, void* stream);
int tplr_gemm2_rope(const void* X, const void* W, void* QKV, int M, int N, int K, long long ldx, long long ldw, long long ldc,
                    const float* cosb, const float* sinb, int S, int rope_cols, int head_dim, unsigned int* status, void* stream);
int tplr_attention_fwd(const void* qkv, void* out, float* lse, int B, int S, int H, int KV, int head_dim, long long ld_qkv,
                       long long ld_o, float scale, unsigned int* status, void* stream);
int tplr_gemm2_attn_dout(const void* dY, const void* Wo, const void* O, void* dO, float* delta, int M, int N, int K, int S, int head_dim,
                         long long lddy, long long ldwo, long long ldo, long long lddo, unsigned int* status, void* stream);
int tplr_attention_bwd_scratch_cols(int B, int S, int H, int KV, int head_dim);
int tplr_attention_bwd_unrope_delta(const void* qkv, const void* out, const void* dout, const float* lse, float* delta, float* dq32,
                                    void* dqkv, int B, int S, int H, int KV, int head_dim, long long ld_qkv, long long ld_o,
                                    float scale, const float* cosb, const float* sinb, unsigned int* status, void* stream);
}
