// The C launchers that more than one source names: the native host module calls them, and the pair GEMMs hand their small
// outputs to the single-CTA ones. Included where each is defined, so that the compiler compares the parameter lists.
// 0: enqueued (or nothing to do); -2: an argument that the kernels do not take; any other code is the driver's.
#pragma once

extern "C" {
// gemm_tcgen05.cu
int ss_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                 int a_mn, int b_mn, int c_f32, int accumulate, float alpha, int bn, int num_sms, int* status, void* stream);
int ss_gemm_swiglu_bf16(const void* A, const void* B, void* gu, void* h, int M, int F, int K, long long lda, long long ldb,
                        long long ldgu, long long ldh, int bn, int* status, void* stream);
int ss_gemm_swiglu_bwd_bf16(const void* A, const void* B, const void* gu, void* dgu, int M, int F, int K, long long lda,
                            long long ldb, long long ldgu, long long lddgu, int bn, int* status, void* stream);
// gemm_tcgen05_2cta.cu
int ss_gemm2_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                  int a_mn, int b_mn, int c_f32, int accumulate, float alpha, int num_sms, int* status, void* stream);
int ss_gemm2_residual_bf16(const void* A, const void* B, const void* src, void* C, int M, int N, int K, long long lda,
                           long long ldb, long long ldsrc, long long ldc, int* status, void* stream);
int ss_gemm2_swiglu_bf16(const void* A, const void* B, void* gu, void* h, int M, int F, int K, long long lda, long long ldb,
                         long long ldgu, long long ldh, int* status, void* stream);
int ss_gemm2_swiglu_bwd_bf16(const void* A, const void* B, const void* gu, void* dgu, int M, int F, int K, long long lda,
                             long long ldb, long long ldgu, long long lddgu, int* status, void* stream);
// norm.cu
int ss_rmsnorm_fwd(void* x, const void* delta, const void* w, void* y, float* rstd, int T, int D, float eps,
                   int zero_centered, int* status, void* stream);
int ss_rmsnorm_bwd(const void* x, const void* w, const void* gy, const float* rstd, void* dx, float* dw, int T, int D,
                   int zero_centered, int accumulate, int* status, void* stream);
// elementwise.cu
int ss_rope(void* buf, const int* positions, int T, long long row_stride, int col0, int heads, int dh, int rot, float theta,
            int inverse, void* stream);
// attention_fwd.cu, attention_bwd.cu
int ss_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* cu_seqlens, int nseq, int T,
                int Hq, int Hkv, int dh, long long ldq, long long ldk, long long ldv, long long ldo, float scale,
                int* status, void* stream);
int ss_attn_bwd_g(const void* q, const void* k, const void* v, const void* out, const float* lse, const void* dout, void* dq,
                  void* dk, void* dv, const int* cu_seqlens, float* delta_scratch, int nseq, int T, int Hq, int Hkv, int dh,
                  long long ldq, long long ldk, long long ldv, long long ldo, long long lddq, long long lddk, long long lddv,
                  float scale, int* status, void* stream);
}
