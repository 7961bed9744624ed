// Entry points of the library that its own host code calls (block_exec.cu). The files that define them include this too, so a definition whose
// arguments have changed does not compile.
#pragma once
#include <cuda_runtime.h>

extern "C" {
// The kernels of a product, as plans number them (ops/gemm_plan.py): single CTAs, CTA pairs, pairs with wide tiles, single CTAs with narrow ones.
#define GEMM_FORMS(F) \
  F(FORM_ONE, mtb200_gemm_bf16) F(FORM_PAIR, mtb200_gemm2_bf16) F(FORM_WIDE, mtb200_gemm2_wide_bf16) F(FORM_N64, mtb200_gemm_n64_bf16) F(FORM_N128, mtb200_gemm_n128_bf16)
typedef int GemmEntry(const void*, long long, int, const void*, long long, int, void*, long long, int, const void*, long long, const void*, int, int, int,
                      float, int, unsigned long long*, unsigned long long, float*, long long, float2*, int*, cudaStream_t);
#define F(form, entry) form,
enum { GEMM_FORMS(F) };
#undef F
#define F(form, entry) GemmEntry entry;
GEMM_FORMS(F)
#undef F
inline GemmEntry* gemm_entry(int form) {
#define F(form, entry) case form: return entry;
  switch (form) { GEMM_FORMS(F) default: return nullptr; }
#undef F
}
int mtb200_gemm_act(const void*, long long, const void*, void*, void*, const void*, int, int, int, int, int, int, int*, cudaStream_t);
int mtb200_swiglu_fwd(const void*, void*, long long, int, cudaStream_t);
int mtb200_geglu_fwd(const void*, void*, long long, int, cudaStream_t);
int mtb200_gelu_fwd(const void*, void*, long long, cudaStream_t);
int mtb200_swiglu_bwd(const void*, const void*, void*, long long, int, cudaStream_t);
int mtb200_swiglu_bwd_act(void*, const void*, void*, long long, int, cudaStream_t);
int mtb200_geglu_bwd(const void*, const void*, void*, long long, int, cudaStream_t);
int mtb200_geglu_bwd_act(void*, const void*, void*, long long, int, cudaStream_t);
int mtb200_gelu_bwd(const void*, const void*, void*, long long, cudaStream_t);
int mtb200_gelu_bwd_act(void*, const void*, void*, long long, cudaStream_t);
int mtb200_rmsnorm_fwd(const void*, const void*, void*, float*, float, int, int, int*, cudaStream_t);
int mtb200_layernorm_fwd(const void*, const void*, const void*, void*, float*, float*, float, int, int, int*, cudaStream_t);
int mtb200_norm_bwd_blocks(int, int);
int mtb200_rmsnorm_bwd(const void*, const void*, const float*, const void*, const void*, void*, float*, void*, int, int, int*, cudaStream_t);
int mtb200_layernorm_bwd(const void*, const void*, const float*, const float*, const void*, const void*, void*, float*, void*, void*, int, int, int*,
                         cudaStream_t);
int mtb200_rope(void*, const int*, const float*, int, long long, int, int, int, cudaStream_t);
int mtb200_head_rmsnorm_fwd(void*, const void*, const void*, void*, float*, const int*, const float*, float, int, long long, int, int, int, cudaStream_t);
int mtb200_head_rmsnorm_bwd_blocks(int, int);
int mtb200_head_rmsnorm_bwd(void*, const void*, const float*, const void*, const void*, float*, void*, void*, const int*, const float*, int, long long,
                            long long, int, int, int, cudaStream_t);
int mtb200_attn_fwd(const void*, long long, void*, long long, float*, const int*, int, int, int, int, int, int, float, int*, cudaStream_t);
int mtb200_attn_fwd_one(const void*, long long, void*, long long, float*, const int*, int, int, int, int, int, float, int*, cudaStream_t);
int mtb200_attn_bwd(const void*, long long, const void*, long long, const void*, long long, void*, long long, const float*, float*, float*, const int*, int,
                    int, int, int, int, int, unsigned long long*, unsigned long long, float*, long long, float, int, int*, cudaStream_t);
int mtb200_colsum(const void*, long long, void*, float*, int, int, cudaStream_t);
int mtb200_embedding_fwd(const void*, const long long*, void*, int, int, int, int*, cudaStream_t);
int mtb200_embedding_bwd_scan(void*, const long long*, const void*, int, int, int, int*, cudaStream_t);
int mtb200_scatter_rows(const long long*, const void*, void*, const float*, float*, int, int, int, int*, cudaStream_t);
int mtb200_ce_fwd_bwd(const void*, long long, int, const float2*, const long long*, float*, void*, long long, int, int, float, long long, cudaStream_t);
int mtb200_accumulate(float*, const void*, long long, int, int, cudaStream_t);
}
