// C entry points that are called from another file than their own. Both sides include this, so that the compiler compares the
// arguments: with C linkage the linker would not.
#pragma once
#include <stdint.h>

extern "C" {
int otb_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, long rows, int D, float inv_d, float eps, int dtype, void* stream);
int otb_gemm_bf16(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long lda, long ldb, long ldc, long ldr, int a_mn,
                  int b_mn, int epi, uint32_t* status, int max_ctas, void* stream);
int otb_gemm_f32(const float* A, const float* B, float* C, const float* R, int M, int N, int K, long lda, long ldb, long ldc, long ldr,
                 int a_mn, int b_mn, int epi, void* stream);
int otb_qknorm_rope_fwd(const void* in, long ld_in, void* out, long ld_out, float* rstd, const float* cosb, const float* sinb, long rows,
                        int heads, int D, int seq_len, int do_norm, float inv_d, float eps, int dtype, void* stream);
int otb_attn_fwd(const void* qk, long ldqk, const void* qkv, long ldqkv, void* O, long ldo, float* lse, int B, int T, int H, int Hkv, int D,
                 int window, float scale, uint32_t* status, void* stream);
int otb_attn_f32_fwd(const float* qk, long ldqk, const float* qkv, long ldqkv, float* O, long ldo, float* lse, int B, int T, int H, int Hkv,
                     int D, int window, float scale, void* stream);
int otb_swiglu_fwd(const void* gu, void* h, long rows, int F, int dtype, void* stream);
}
