// Entry points of libb200ops.so that the native layers (torch_ops.cpp) call. The sources that define them
// include this header too, so that a changed signature does not compile on one side only.
#pragma once

extern "C" {

int b200_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                   int a_mn, int b_mn, int out_fp32, int accumulate, int bn, int max_ctas, void* stream);

// Both gradients of a linear layer; see gemm_grads.cu. *launches: kernels launched, 1 or 2.
int b200_linear_grads(const void* dy, const void* x, const void* w, void* dx, void* dw, int M, int N, int K, long long lddy,
                      long long ldx, long long ldw, long long lddx, long long lddw, int accumulate, int* launches, void* stream);

int b200_rmsnorm_fwd(const void* x, const void* res, void* h_out, const void* w, void* y, float* rstd, int T, int H, float eps,
                     void* stream);
int b200_embedding_fwd(const long long* ids, const void* table, void* out, long long T, int H, void* stream);
int b200_embedding_bwd(const long long* ids, const void* dout, void* dtable, long long T, int H, void* stream);
int b200_cross_entropy(void* logits, const long long* targets, float* loss, int T, int V, long long ld, float grad_scale, void* stream);
int b200_rmsnorm_bwd_partial_rows();
int b200_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                     float* dw_partial, void* dw, int accumulate_dw, int T, int H, void* stream);

int b200_swiglu_fwd(const void* gu, void* out, long long T, int F, void* stream);
int b200_swiglu_bwd(const void* dout, const void* gu, void* dgu, long long T, int F, void* stream);

// gate|up = x w^T with act = silu(gate) * up, and the gradient at gate|up from dy and the down projection w; see
// gemm_swiglu.cu. The bwd call wants `scratch` [M][F] bf16 where b200_gemm_swiglu_bwd_launches says 2.
int b200_gemm_swiglu(const void* x, const void* w, void* gu, void* act, int M, int F, int K, long long ldx, void* stream);
int b200_gemm_swiglu_bwd(const void* dy, const void* w, const void* gu, void* dgu, void* scratch, int M, int F, int K, long long lddy,
                         void* stream);
int b200_gemm_swiglu_launches(const void* x, const void* w, int M, int F, int K, long long ldx);
int b200_gemm_swiglu_bwd_launches(const void* dy, const void* w, int M, int F, int K, long long lddy);

int b200_rope_qkv(void* qkv, long long pitch, void* q, void* k, void* v, const long long* strides, const float* cs,
                  const float* sn, long long T, int nq, int nkv, int hd, int seq, int backward, void* stream);

}  // extern "C"
