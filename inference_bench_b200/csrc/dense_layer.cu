// The kernels of one dense layer (norm, q/k/v, attention, output, norm, gate/up, down) of a bfloat16 step outside a graph, launched by one call.
//
// Nothing here runs on the device: the call is the list of launches that the parts make one by one from Python, in the same order with the same
// arguments. What bounds a step of a short prompt portion is the host: a part's wrapper checks its tensors, asks for an output and works out a tile in
// about 15 us, a launch takes 3, and the kernel itself 3 to 10. The forms of the products and the buffers are worked out once a step
// (kernels/dense.py); a layer then costs its launches. 100 tokens in two layers of the 0.6B sizes: 514 to 277 us of host a step (with the step's arrays
// in one transfer), 61 tokens behind 900 in eight layers 883 to 445, as long as its kernels.
#include "entries.h"

// How a product runs. kind 0: the single-CTA kernel, `splits` partial sums of tiles of bn tokens; 1: CTA pairs, one sum; 2: CTA pairs, added to the
// residual stream; 3: with the epilogue that finishes it (q/k/v: norm, rotation and cache write on CTA pairs; gate/up: the activation, on CTA pairs where
// bn is 0, else tiles of bn tokens, `wide` telling whether gate and up share an accumulator).
struct IbDenseProduct {
  int kind, bn, splits, wide;
};

struct IbDenseStep {   // what the layers of a step have in common
  float* x;            // the residual stream [T, hidden]
  void* h;             // [T, hidden]
  float* partial;      // partial sums of any one product
  void* q;             // [T, heads * head_dim]
  void* o;             // the same
  void* act;           // [T, inter]
  float* part_o;       // decoded tokens: [n_dec, heads, max_slices, head_dim] and two numbers each
  float* part_ml;
  const float* cos_t;
  const float* sin_t;
  const int* positions;
  const int* seg_of_token;
  const int* seg_start;
  const int* seg_pos0;
  const int* dec_tokens;
  const int* tile_seg;
  const int* tile_row0;
  const void* kv_map;
  unsigned* status;
  cudaStream_t stream;
  IbDenseProduct qkv, out, gate_up, down;
  int T, hidden, inter, heads, kv_heads, head_dim, rot_half, window, n_dec, n_tiles, max_slices, tiles_per_slice, tile_keys;
  float norm_eps, ff_norm_eps, qk_eps, scale;
};

struct IbDenseLayer {
  const float* norm;
  const void* w_qkv;
  const void* w_out;
  const float* ff_norm;
  const void* w_gate_up;
  const void* w_down;
  const float* q_norm;
  const float* k_norm;
  const IbKvView* kv;
  long long kv_row0;    // the view's first row in the pool's tensor map
  const float* delta;   // what the layer before left to add: delta_parts sums of [T, hidden], or null
  int delta_parts;
};

// A launch, unless one before it was refused: the layer then ends, with the text of that one's error.
#define IB_LAYER_RUN(launch, kernels) \
  do {                                \
    if ((launch) != 0) return -1;     \
    n += (kernels);                   \
  } while (0)

// Returns the number of kernels launched, or -1 with the error's text set: nothing is launched behind a kernel that was refused.
extern "C" int ib_dense_layer(const IbDenseStep* s, const IbDenseLayer* l) {
  const int T = s->T, H = s->hidden, Q = s->heads * s->head_dim, R = Q + 2 * s->kv_heads * s->head_dim;
  if (T <= 0 || (s->n_dec > 0 && !s->part_o) || s->n_dec + s->n_tiles <= 0) {
    ib_set_error("dense_layer: bad sizes T=%d n_dec=%d n_tiles=%d", T, s->n_dec, s->n_tiles);
    return -1;
  }
  int n = 0;
  auto product = [&](const IbDenseProduct& p, const void* in, const void* w, int N, int K) {
    if (p.kind == 2) return ib_gemm_tcgen05_2cta_add(in, w, s->x, T, N, K, s->status, s->stream);
    if (p.kind == 1) return ib_gemm_tcgen05_2cta(in, w, s->partial, T, N, K, s->status, s->stream);
    return ib_gemm_tcgen05(in, w, s->partial, T, N, K, p.bn, p.splits, p.wide, s->status, s->stream);
  };
  auto norm = [&](const float* delta, int parts, const float* w, float eps) {
    return ib_add_rmsnorm(s->x, delta, delta ? parts : 0, delta ? (long long)T * H : 0, w, s->h, IB_BF16, nullptr, T, H, eps, 1, s->stream);
  };
  IB_LAYER_RUN(norm(l->delta, l->delta_parts, l->norm, s->norm_eps), 1);
  if (s->qkv.kind == 3) {
    IB_LAYER_RUN(ib_gemm_qkv_tcgen05_2cta(s->h, l->w_qkv, T, H, l->q_norm, l->k_norm, s->qk_eps, s->cos_t, s->sin_t, s->positions, s->seg_of_token, s->q, l->kv, 1, s->heads,
                                          s->status, s->stream), 1);
  } else {
    IB_LAYER_RUN(product(s->qkv, s->h, l->w_qkv, R, H), 1);
    IB_LAYER_RUN(ib_qk_norm_rope_kv(s->partial, s->qkv.kind == 1 ? 1 : s->qkv.splits, (long long)T * R, l->q_norm, l->k_norm, s->qk_eps, s->cos_t, s->sin_t, s->rot_half,
                                    s->positions, s->seg_of_token, s->q, IB_BF16, l->kv, 1, T, s->heads, s->status, nullptr, s->head_dim, s->head_dim, 0, 0, 0, 0, 0, s->stream), 1);
  }
  if (s->n_dec)
    IB_LAYER_RUN(ib_attention_decode_stream(s->q, l->kv, s->dec_tokens, s->n_dec, s->positions, s->seg_of_token, s->window, s->scale, s->part_o, s->part_ml, s->o, s->heads,
                                            s->max_slices, s->tiles_per_slice, s->kv_map, l->kv_row0, s->status, s->stream), 2);
  if (s->n_tiles)
    IB_LAYER_RUN(ib_attention_prefill_ws(s->q, l->kv, s->tile_seg, s->tile_row0, s->n_tiles, s->seg_start, s->seg_pos0, s->window, s->scale, s->o, s->heads, s->kv_map, l->kv_row0,
                                         s->tile_keys, s->status, s->stream), 1);
  IB_LAYER_RUN(product(s->out, s->o, l->w_out, H, Q), 1);
  IB_LAYER_RUN(norm(s->out.kind == 2 ? nullptr : s->partial, s->out.kind == 1 ? 1 : s->out.splits, l->ff_norm, s->ff_norm_eps), 1);
  const IbDenseProduct& g = s->gate_up;
  if (g.kind == 3 && g.bn == 0) {
    IB_LAYER_RUN(ib_gemm_swiglu_tcgen05_2cta(s->h, l->w_gate_up, s->act, T, s->inter, H, nullptr, 0.f, s->status, s->stream), 1);
  } else if (g.kind == 3) {
    IB_LAYER_RUN(ib_gemm_swiglu_tcgen05(s->h, l->w_gate_up, s->act, T, s->inter, H, g.bn, g.wide, nullptr, 0.f, s->status, s->stream), 1);
  } else {
    IB_LAYER_RUN(product(g, s->h, l->w_gate_up, 2 * s->inter, H), 1);
    IB_LAYER_RUN(ib_silu_mul(s->partial, g.kind == 1 ? 1 : g.splits, (long long)T * 2 * s->inter, s->act, IB_BF16, T, s->inter, nullptr, 0.f, s->stream), 1);
  }
  IB_LAYER_RUN(product(s->down, s->act, l->w_down, H, s->inter), 1);
  return n;
}

// The sizes of IbDenseStep and IbDenseLayer, for a caller that mirrors them in another language.
extern "C" int ib_dense_sizes(int* step, int* layer) {
  *step = (int)sizeof(IbDenseStep), *layer = (int)sizeof(IbDenseLayer);
  return 0;
}
