// Launch functions that other sources of the library call.  The sources that define them include this file too, so that a
// definition with other arguments does not compile.
#pragma once
#include "common.cuh"

IFX_API int ifx_add_rmsnorm(float* residual, const void* delta, int delta_dtype, int n_partials, long long partial_stride,
                            const float* weight, float eps, void* out, int out_dtype, const int* rows, int n_rows, int hidden,
                            int write_residual, cudaStream_t stream);
IFX_API int ifx_qkv_rope_kv_write(void* qkv, int dtype, const float* bias, const float* cos_t, const float* sin_t, int rot_dim,
                                  const int* slot_map, void* k_layer, void* v_layer, long long page_stride, int page_size,
                                  int n_tokens, int n_heads, int n_kv, int head_dim, const float* partials, int n_partials,
                                  cudaStream_t stream);
IFX_API int ifx_gemm_umma_skinny(const void* X, long long ldx, const void* W, float* out, int tokens, int n_out, int K, int k_parts,
                                 int w_fixed, int* error_flag, cudaStream_t stream);
IFX_API int ifx_gemm_umma_skinny_glu(const void* X, long long ldx, const void* W, void* out, long long ldo, int tokens, int inter,
                                     int K, int w_fixed, int* error_flag, cudaStream_t stream);
IFX_API int ifx_gemv_bf16(const void* X, const void* W, const float* bias, void* out, int out_dtype, int M, int n_out, int K,
                          long long ldx, long long ldo, int act, int k_splits, float limit, float alpha, float shift,
                          cudaStream_t stream);
IFX_API int ifx_attn_prefill_umma(const void* q, long long q_stride, void* out, long long out_stride, void* k_layer, void* v_layer,
                                  long long page_stride, int page_size, const int* block_tables, int bt_stride,
                                  const int* tile_entry, const int* tile_q0, int n_tiles, const int* entry_q_start,
                                  const int* entry_q_len, const int* entry_ctx_start, int n_heads, int n_kv, int head_dim,
                                  float scale, int window, int* error_flag, float* part_o, float* part_ml, int n_splits,
                                  int num_pages, int tile_rows, const float* gate, int gate_parts, long long gate_part_stride,
                                  int gate_stride, cudaStream_t stream);
IFX_API int ifx_attn_decode_bf16(const void* q, long long q_stride, void* out, long long out_stride, void* k_layer, void* v_layer,
                                 long long page_stride, int page_size, const int* block_tables, int bt_stride,
                                 const int* dec_entries, int n_dec, const int* entry_q_start, const int* entry_q_len,
                                 const int* entry_ctx_start, float* part_o, float* part_ml, int n_heads, int n_kv, int head_dim,
                                 float scale, int window, int n_splits, cudaStream_t stream);
IFX_API int ifx_attn_decode_even_bf16(const void* q, long long q_stride, void* out, long long out_stride, void* k_layer,
                                      void* v_layer, long long page_stride, int page_size, const int* block_tables, int bt_stride,
                                      const int* dec_entries, int n_dec, const int* entry_q_start, const int* entry_q_len,
                                      const int* entry_ctx_start, float* part_o, float* part_ml, int* piece_count, int n_heads,
                                      int n_kv, int head_dim, float scale, int window, int max_pieces, int* error_flag,
                                      cudaStream_t stream);
