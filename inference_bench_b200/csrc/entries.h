// Entry points that this library also calls from one source file in another (csrc/dense_layer.cu launches a layer through them). C linkage carries no types, so
// the files that define them include this header too: a changed argument list does not compile until it is changed here and at every call.
#pragma once
#include "kv_view.cuh"

extern "C" {
int ib_add_rmsnorm(float* x, const float* delta, int P, long long delta_stride, const float* w, void* out, int out_dtype, const int* rows, int n_rows, int H, float eps, int write_x,
                   cudaStream_t stream);
int ib_silu_mul(const float* gu, int P, long long stride, void* act, int act_dtype, int T, int I, const float* limit, float slope, cudaStream_t stream);
int ib_qk_norm_rope_kv(const float* qkv, int P, long long stride_p, const float* q_norm_w, const float* k_norm_w, float eps, const float* cos_t, const float* sin_t, int rot_half,
                       const int* positions, const int* seg_of_token, void* q_out, int act_dtype, const IbKvView* kv, int write_kv, int T, int heads, unsigned* status,
                       const float* bias, int qk_dim, int v_dim, int row, int q_col, int k_col, int v_col, int unit_norm_after, cudaStream_t stream);
int ib_attention_prefill_ws(const void* q, const IbKvView* kv, const int* tile_seg, const int* tile_row0, int n_tiles, const int* seg_start, const int* seg_pos0, int window, float scale,
                            void* out, int heads, const void* kv_map, long long view_row0, int max_keys, unsigned* status, cudaStream_t stream);
int ib_attention_decode_stream(const void* q, const IbKvView* kv, const int* dec_tokens, int n_dec, const int* positions, const int* seg_of_token, int window, float scale, float* part_o,
                               float* part_ml, void* out, int heads, int max_slices, int tiles_per_slice, const void* kv_map, long long view_row0, unsigned* status, cudaStream_t stream);
int ib_gemm_tcgen05(const void* x, const void* w, float* out, int T, int N, int K, int bn, int splits, int wide, unsigned* status, cudaStream_t stream);
int ib_gemm_swiglu_tcgen05(const void* x, const void* w, void* act, int T, int I, int K, int bn, int half, const float* limit, float slope, unsigned* status, cudaStream_t stream);
int ib_gemm_tcgen05_2cta(const void* x, const void* w, float* out, int T, int N, int K, unsigned* status, cudaStream_t stream);
int ib_gemm_tcgen05_2cta_add(const void* x, const void* w, float* out, int T, int N, int K, unsigned* status, cudaStream_t stream);
int ib_gemm_swiglu_tcgen05_2cta(const void* x, const void* w, void* act, int T, int I, int K, const float* limit, float slope, unsigned* status, cudaStream_t stream);
int ib_gemm_qkv_tcgen05_2cta(const void* x, const void* w, int T, int K, const float* q_norm_w, const float* k_norm_w, float eps, const float* cos_t, const float* sin_t,
                             const int* positions, const int* seg_of_token, void* q_out, const IbKvView* kv, int write_kv, int heads, unsigned* status, cudaStream_t stream);
}
