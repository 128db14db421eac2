// The launches of all layers of a Llama-style model for few tokens (up to 64) in bfloat16, from one call.
//
// A step of few tokens that is not a recorded one launches five or six kernels a layer, each some 10 to 40 us of the GPU's time or less; from
// Python a launch takes 20 us and more (arguments checked one by one, results allocated, the call converted), so the GPU waited for the
// host: 16 layers of width 2048 took 1.9 ms of which it worked 0.75.  Here the host's part is a loop over the layers; every buffer
// between the kernels is the caller's.  The kernels, their arguments and their order are those of parts/attention.py, parts/mlp.py and
// parts/block.py, so the results have the same bits.
//
// Each kernel family is a library of its own: the caller hands over their entry points.
#include "common.cuh"

typedef int (*BnLinearTc)(const void* x, const void* w, void* out, int out_dtype, int M, int N, int K, int ldo, int mode, int cluster,
                          const float* row_ss, int ss_parts, int ss_stride, float inv_width, float eps, const void* gain, int gain_dtype, void* xg,
                          float* ss_out, int ss_out_stride, int* status, cudaStream_t stream);
typedef int (*BnLinearResident)(const void* x, const void* w, void* out, int out_dtype, int M, int N, int K, int ldo, int mode, const float* row_ss,
                                int ss_parts, int ss_stride, float inv_width, float eps, const void* gain, int gain_dtype, void* xg, float* ss_out,
                                int ss_out_stride, cudaStream_t stream);
typedef int (*BnRopeAppend)(void* x, int dtype, int n_tokens, int row_stride, int n_rot_heads, int head_dim, int rotary_dims, float theta_scale,
                            const int* tok_pos, int k_off, int v_off, int n_kv_heads, const int* tok_seq, const int* slots, const int* page_table,
                            int pt_stride, void* k_cache, void* v_cache, cudaStream_t stream);
typedef int (*BnDecode)(const void* qkv, int q_stride, int k_off, int v_off, void* out, int out_stride, int n_seqs, int n_heads, int n_kv_heads,
                        int head_dim, float scale, int window, int rotary_dims, float theta_scale, const int* tok_pos, const int* slots,
                        const int* page_table, int pt_stride, void* k_cache, void* v_cache, int n_cache_pages, int* status, float* part_o,
                        float* part_ml, int n_splits, int pages_per_block, int* tickets, int n_tickets, cudaStream_t stream);
typedef int (*BnDecodeItems)(const void* qkv, int q_stride, int k_off, int v_off, void* out, int out_stride, int n_seqs, int n_heads, int n_kv_heads,
                             int head_dim, float scale, int window, int rotary_dims, float theta_scale, const int* tok_pos, const int* slots,
                             const int* page_table, int pt_stride, void* k_cache, void* v_cache, int n_cache_pages, int* status, float* part_o,
                             float* part_ml, int* tickets, int n_tickets, const int* items, int n_items, int item_group, cudaStream_t stream);
typedef int (*BnPrefill)(const void* q, int q_stride, int n_tokens, void* out, int out_stride, int n_tiles, int n_heads, int n_kv_heads, int head_dim,
                         float scale, int window, const int* tile_seq, const int* tile_row0, const int* seq_start, const int* seq_pos0,
                         const int* slots, const int* page_table, int pt_stride, const void* k_cache, const void* v_cache, int n_cache_pages,
                         int* status, cudaStream_t stream);

// (engine/few_layers.py holds the same two structures)
struct FewLayer {
  const void *w_qkv, *w_o, *w_gate_up, *w_down;
  const void *gain_ffn, *gain_next;  // the norms behind the two residual additions; gain_next null: the last product goes to `delta`
  void *k_cache, *v_cache;
  const int* page_table;
  int gain_ffn_dtype, gain_next_dtype, pt_stride, n_cache_pages;
  float eps_ffn, eps_next;
};
struct FewStep {
  const FewLayer* layers;
  BnLinearTc linear_tc;
  BnLinearResident resident;
  BnRopeAppend rope;
  BnDecode decode;
  BnDecodeItems decode_items;
  BnPrefill prefill;
  float* x;        // [M, width] the residual
  const void* h;   // [M, width] the first layer's normed rows
  void *qkv, *attn, *act, *mid, *next, *delta;  // mid, next: rows for the products behind the two additions
  float *mid_ss, *next_ss;                      // and their sums of squares, [parts][M]
  const int *tok_pos, *tok_seq, *slots, *tile_seq, *tile_row0, *seq_start, *seq_pos0, *items;
  float *part_o, *part_ml;
  int *tickets, *status;
  int n_layers, M, n_seqs, width, inter, n_heads, n_kv_heads, head_dim, act_code, rotary_dims, window;
  int decoding, n_splits, pages_per_block, n_tickets, n_items, item_group, n_tiles;
  int res_qkv, res_o, res_gate_up, res_down;  // whether each product is of the kernel for small matrices
  int cluster_o, cluster_down;                // blocks per tile of the other, where it adds to the residual
  float scale, theta_scale;
};

extern "C" int bn_few_layers(const FewStep* s, cudaStream_t stream) {
  const int q_dim = s->n_heads * s->head_dim, kv_dim = s->n_kv_heads * s->head_dim, n_qkv = q_dim + 2 * kv_dim;
  const float inv_width = 1.0f / s->width;
  // one product; ss (or null): the sums of squares of rows that still lack their norm's scale
  auto product = [&](int resident, const void* x, const void* w, void* out, int out_dtype, int N, int K, int ldo, int mode, int cluster, const float* ss,
                     int parts, float eps, const void* gain, int gain_dtype, void* xg, float* ss_out) {
    const float inv = ss ? inv_width : 0.f, e = ss ? eps : 0.f;
    const int stride = ss ? s->M : 0;
    if (resident)
      return s->resident(x, w, out, out_dtype, s->M, N, K, ldo, mode, ss, parts, stride, inv, e, gain, gain_dtype, xg, ss_out, ss_out ? s->M : 0, stream);
    return s->linear_tc(x, w, out, out_dtype, s->M, N, K, ldo, mode, cluster, ss, parts, stride, inv, e, gain, gain_dtype, xg, ss_out,
                        ss_out ? s->M : 0, s->status, stream);
  };
  const int tiles = (s->width + 127) / 128, small = (s->width + 15) / 16;
  const int mid_parts = s->res_o ? small : tiles * s->cluster_o, next_parts = s->res_down ? small : tiles * s->cluster_down;
  const void* h = s->h;
  const float* ss = nullptr;
  float eps = 0.f;
  for (int i = 0; i < s->n_layers; ++i) {
    const FewLayer& l = s->layers[i];
    int rc = product(s->res_qkv, h, l.w_qkv, s->qkv, BN_BF16, n_qkv, s->width, n_qkv, 0, 0, ss, ss ? next_parts : 0, eps, nullptr, 0, nullptr, nullptr);
    if (rc != BN_OK) return rc;
    if (s->decoding && s->items != nullptr) {
      rc = s->decode_items(s->qkv, n_qkv, q_dim, q_dim + kv_dim, s->attn, q_dim, s->n_seqs, s->n_heads, s->n_kv_heads, s->head_dim, s->scale, s->window,
                           s->rotary_dims, s->theta_scale, s->tok_pos, s->slots, l.page_table, l.pt_stride, l.k_cache, l.v_cache, l.n_cache_pages,
                           s->status, s->part_o, s->part_ml, s->tickets, s->n_tickets, s->items, s->n_items, s->item_group, stream);
    } else if (s->decoding) {
      rc = s->decode(s->qkv, n_qkv, q_dim, q_dim + kv_dim, s->attn, q_dim, s->n_seqs, s->n_heads, s->n_kv_heads, s->head_dim, s->scale, s->window,
                     s->rotary_dims, s->theta_scale, s->tok_pos, s->slots, l.page_table, l.pt_stride, l.k_cache, l.v_cache, l.n_cache_pages, s->status,
                     s->part_o, s->part_ml, s->n_splits, s->pages_per_block, s->tickets, s->n_tickets, stream);
    } else {
      rc = s->rope(s->qkv, BN_BF16, s->M, n_qkv, s->n_heads + s->n_kv_heads, s->head_dim, s->rotary_dims, s->theta_scale, s->tok_pos, q_dim,
                   q_dim + kv_dim, s->n_kv_heads, s->tok_seq, s->slots, l.page_table, l.pt_stride, l.k_cache, l.v_cache, stream);
      if (rc != BN_OK) return rc;
      rc = s->prefill(s->qkv, n_qkv, s->M, s->attn, q_dim, s->n_tiles, s->n_heads, s->n_kv_heads, s->head_dim, s->scale, s->window, s->tile_seq,
                      s->tile_row0, s->seq_start, s->seq_pos0, s->slots, l.page_table, l.pt_stride, l.k_cache, l.v_cache, l.n_cache_pages, s->status,
                      stream);
    }
    if (rc != BN_OK) return rc;
    rc = product(s->res_o, s->attn, l.w_o, s->x, BN_F32, s->width, q_dim, s->width, 3, s->cluster_o, nullptr, 0, 0.f, l.gain_ffn, l.gain_ffn_dtype, s->mid,
                 s->mid_ss);
    if (rc != BN_OK) return rc;
    rc = product(s->res_gate_up, s->mid, l.w_gate_up, s->act, BN_BF16, 2 * s->inter, s->width, s->inter, 2 | s->act_code << 8, 0, s->mid_ss, mid_parts,
                 l.eps_ffn, nullptr, 0, nullptr, nullptr);
    if (rc != BN_OK) return rc;
    if (l.gain_next != nullptr)
      rc = product(s->res_down, s->act, l.w_down, s->x, BN_F32, s->width, s->inter, s->width, 3, s->cluster_down, nullptr, 0, 0.f, l.gain_next,
                   l.gain_next_dtype, s->next, s->next_ss);
    else
      rc = product(s->res_down, s->act, l.w_down, s->delta, BN_BF16, s->width, s->inter, s->width, 0, 0, nullptr, 0, 0.f, nullptr, 0, nullptr, nullptr);
    if (rc != BN_OK) return rc;
    h = s->next;
    ss = s->next_ss;
    eps = l.eps_next;
  }
  return BN_OK;
}
