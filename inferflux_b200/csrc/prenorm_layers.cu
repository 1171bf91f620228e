// The kernels of several pre-norm layers launched by one call: norm, q/k/v, rotation and cache write, attention, output
// projection, norm, gate/up with SwiGLU, down, layer after layer.
//
// A step with a prompt portion of a few rows takes the GPU less time than a host needs that checks, allocates and launches
// kernel by kernel from Python: 12 to 16 us a launch, eight or nine launches a layer, against 60 to 90 us of kernels a layer
// for 77 rows of the 3B sizes.  The kernels and their arguments are the ones that the parts launch one by one
// (parts/block.py, attention.py, feed_forward.py, linear.py), and so are the results; only who calls them differs.
// Host code only.
#include "launchers.h"

// What the layers of a call share.  Pointers are device memory.  The fields' order and types are those of ops.PrenormStep.
struct PrenormStep {
  float* residual;                                  // [rows, hidden], updated
  void *x, *qkv, *attn, *act;                       // bfloat16 scratch: [rows, hidden], [rows, width], [rows, heads * 128], [rows, inter]
  float *qkv_sums, *delta;                          // float32 partial sums: [qkv_parts][rows, width]; of o and down, the larger of the two
  const float *cos_t, *sin_t;                       // [rows, 64]
  const int *slot_map, *block_tables, *entry_q_start, *entry_q_len, *entry_ctx_start;
  const int *tile_entry, *tile_q0, *dec_entries;
  float *part_o, *part_ml, *dec_o, *dec_ml;
  int *piece_count, *error_flag;
  cudaStream_t stream;
  long long page_stride;
  int rows, hidden, inter, n_heads, n_kv, page_size, bt_stride, num_pages;
  int qkv_parts, o_parts, down_parts;
  int gate_up_streams;                              // gate and up by the weight-streaming kernel, not the few-row one
  int n_tiles, tile_rows, n_splits;                 // of the prompt portions
  int n_dec, dec_splits, dec_pieces;                // single tokens: dec_pieces > 0: shared out by tiles, else dec_splits parts of the keys
  float scale;
};
// One layer, eleven 64-bit words.
struct PrenormLayer {
  const float* norm1; const void* qkv_w; const float* qkv_bias; void *k_layer, *v_layer; const void* o_w;
  const float* norm2; const void *gate_up_w, *down_w; double eps1, eps2;
};

// The layers in order; the last one's result stays in step->delta as down_parts partial sums.  launched: receives how many kernels
// were launched.  Rows: 9 to 128.
IFX_API int ifx_prenorm_layers(const PrenormStep* step, const PrenormLayer* layers, int n_layers, int* launched) {
  const PrenormStep& s = *step;
  *launched = 0;
  if (s.rows < 9 || s.rows > 128 || !s.error_flag) return IFX_ERR_UNSUPPORTED;
  const int hd = 128, width = (s.n_heads + 2 * s.n_kv) * hd, nq = s.n_heads * hd;
  const long long sum_stride = (long long)s.rows * s.hidden;
  int n = 0, rc = 0;
  for (int i = 0; i < n_layers && !rc; ++i) {
    const PrenormLayer& l = layers[i];
    rc = ifx_add_rmsnorm(s.residual, i ? s.delta : nullptr, IFX_F32, i ? s.down_parts : 1, i && s.down_parts > 1 ? sum_stride : 0, l.norm1,
                         (float)l.eps1, s.x, IFX_BF16, nullptr, s.rows, s.hidden, 1, s.stream);
    if (!rc) rc = ifx_gemm_umma_skinny(s.x, s.hidden, l.qkv_w, s.qkv_sums, s.rows, width, s.hidden, s.qkv_parts, 1, s.error_flag, s.stream);
    if (!rc) rc = ifx_qkv_rope_kv_write(s.qkv, IFX_BF16, l.qkv_bias, s.cos_t, s.sin_t, hd, s.slot_map, l.k_layer, l.v_layer, s.page_stride,
                                        s.page_size, s.rows, s.n_heads, s.n_kv, hd, s.qkv_sums, s.qkv_parts, s.stream);
    n += 3;
    if (!rc && s.n_tiles) {
      rc = ifx_attn_prefill_umma(s.qkv, width, s.attn, nq, l.k_layer, l.v_layer, s.page_stride, s.page_size, s.block_tables, s.bt_stride,
                                 s.tile_entry, s.tile_q0, s.n_tiles, s.entry_q_start, s.entry_q_len, s.entry_ctx_start, s.n_heads, s.n_kv, hd,
                                 s.scale, 0, s.error_flag, s.part_o, s.part_ml, s.n_splits, s.num_pages, s.tile_rows, nullptr, 0, 0, 0, s.stream);
      n += 1 + (s.n_splits > 1);
    }
    if (!rc && s.n_dec) {
      if (s.dec_pieces > 0) {
        rc = ifx_attn_decode_even_bf16(s.qkv, width, s.attn, nq, l.k_layer, l.v_layer, s.page_stride, s.page_size, s.block_tables, s.bt_stride,
                                       s.dec_entries, s.n_dec, s.entry_q_start, s.entry_q_len, s.entry_ctx_start, s.dec_o, s.dec_ml,
                                       s.piece_count, s.n_heads, s.n_kv, hd, s.scale, 0, s.dec_pieces, s.error_flag, s.stream);
        n += 2;
      } else {
        rc = ifx_attn_decode_bf16(s.qkv, width, s.attn, nq, l.k_layer, l.v_layer, s.page_stride, s.page_size, s.block_tables, s.bt_stride,
                                  s.dec_entries, s.n_dec, s.entry_q_start, s.entry_q_len, s.entry_ctx_start, s.dec_o, s.dec_ml, s.n_heads,
                                  s.n_kv, hd, s.scale, 0, s.dec_splits, s.stream);
        n += 1 + (s.dec_splits > 1);
      }
    }
    if (!rc) rc = ifx_gemm_umma_skinny(s.attn, nq, l.o_w, s.delta, s.rows, s.hidden, nq, s.o_parts, 1, s.error_flag, s.stream);
    if (!rc) rc = ifx_add_rmsnorm(s.residual, s.delta, IFX_F32, s.o_parts, s.o_parts > 1 ? sum_stride : 0, l.norm2, (float)l.eps2, s.x, IFX_BF16,
                                  nullptr, s.rows, s.hidden, 1, s.stream);
    if (!rc) rc = s.gate_up_streams ? ifx_gemv_bf16(s.x, l.gate_up_w, nullptr, s.act, IFX_BF16, s.rows, s.inter, s.hidden, s.hidden, s.inter, 1, 1, 0.0f,
                                               0.0f, 0.0f, s.stream)
                               : ifx_gemm_umma_skinny_glu(s.x, s.hidden, l.gate_up_w, s.act, s.inter, s.rows, s.inter, s.hidden, 1, s.error_flag, s.stream);
    if (!rc) rc = ifx_gemm_umma_skinny(s.act, s.inter, l.down_w, s.delta, s.rows, s.hidden, s.inter, s.down_parts, 1, s.error_flag, s.stream);
    n += 4;
  }
  *launched = n;
  return rc;
}
