// One backbone pass over packed tokens (prefill), enqueued by one call: the launches of every layer in the order of
// tah_b200/engine/engine.py's _packed_pass, which remains for tensor parallelism and the opt-in forms.  A pass of a short prompt is
// 28 layers x 9 to 13 launches of 3 to 30 us each; bound to Python (argument conversion, output allocation, plan and checks: 12 us a
// launch) the GPU waited for the host: two passes over 700 tokens took 11.8 ms, 10.0 ms from here.
#include <cuda_runtime.h>
#include <stddef.h>

extern "C" {
int tahb_gemm(const void*, const void*, void*, const void*, const void*, const void*, int, int, int, int, long long, long long, long long,
              long long, long long, long long, int, int, int, int, int*, cudaStream_t);
int tahb_gemm_few(const void*, const void*, void*, const void*, const void*, const void*, int, int, int, int, long long, long long, long long,
                  long long, long long, long long, int, float, float, int, cudaStream_t);
int tahb_gemm_persist(const void*, const void*, void*, const void*, const void*, const void*, int, int, int, int, long long, long long,
                      long long, long long, long long, long long, int, float, float, int, int, int, int*, cudaStream_t, const void*, const void*,
                      int);
int tahb_rmsnorm(const void*, const void*, void*, int, int, long long, long long, float, cudaStream_t);
int tahb_qk_norm_rope_kv(const void*, const void*, const void*, void*, void*, void*, void* const*, int, const int*, const int*, const int*,
                         int, int, int, int, int, long long, float, float, cudaStream_t);
int tahb_prefill_attn(const void*, void*, void* const*, void* const*, const long long*, const int* const*, const int* const*,
                      const int* const*, int, const int*, const int*, int, long long, int, int, int, float, float*, int, int*, cudaStream_t);
}

// Kernel-ready weights of a layer (tah_b200/engine/weights.py); a_* / b_* are null without an adapter.
struct TahbPassWeights {
  const void *ln1, *ln2, *q_norm, *k_norm, *w_qkv, *w_o, *w_gu, *w_down;
  const void *a_qkv, *b_qkv, *a_o, *b_o, *a_gu, *b_gu, *a_down, *b_down;
};
// How a product runs: kind 1 the few-token kernel, 2 the persistent one with its tile width, 0 one tile per CTA with form, tile width and split.
struct TahbProductPlan {
  int kind, dual, splits, bn;
};
struct TahbPass {
  const TahbPassWeights* layers;
  const void* final_norm;
  void *h, *xn, *qkv, *q, *o, *act;                 // [n, .] activations; h: the residual stream, its input at entry
  void *t_qkv, *t_o, *t_gu, *t_down;                // [n, r] adapter inputs, or null
  void* const* taps;                                // [layers + 1] where the input of a layer is copied to, or null
  void* const* k_own;                               // [layers] keys and values of this pass, packed
  void* const* v_own;
  void* const* pool;                                // [layers] paged cache of this depth
  void* const* k_seg[3];                            // [layers] keys and values of the shallower passes
  void* const* v_seg[3];
  long long n_kv[3];                                // rows of every segment, this pass's last
  const int* base[3];
  const int* count[3];
  const int *pos, *slots, *tile_q0, *tile_qn;
  int* status;
  int n_layers, n, hidden, inter, nq, nkv, hd, page_size, n_seg, n_tiles, attn_heads;
  int r_qkv, r_o, r_gu, r_down;                     // 0 without the adapter
  float eps, theta, scale;
  TahbProductPlan p_qkv, p_o, p_gu, p_down, p_a_qkv, p_a_o, p_a_gu, p_a_down;
};

extern "C" int tahb_packed_pass(const TahbPass* a, int* launches, cudaStream_t stream) {
  const int n = a->n, H = a->hidden, I = a->inter, D = a->nq * a->hd, F = (a->nq + 2 * a->nkv) * a->hd;
  int rc = 0, count = 0;
  if (a->n_seg < 1 || a->n_seg > 3) return -1;
  // out = x W^T (+ t B^T) (+ residual); rows: rows of W, ldo: row pitch of out
  auto product = [&](const TahbProductPlan& p, const void* w, const void* x, void* out, const void* res, const void* b, const void* t,
                     int rows, int K, int R, int ldo) {
    if (rc) return;
    ++count;
    const bool stacked = p.dual == 1;
    if (p.kind == 2)
      rc = tahb_gemm_persist(w, x, out, res, b, t, n, rows, K, R, K, K, ldo, res ? ldo : 0, R, R, p.dual ? 2 : 0, 0.f, 0.f, 0, 0, p.bn, a->status,
                             stream, nullptr, nullptr, 0);
    else if (p.kind == 1)
      rc = tahb_gemm_few(w, x, out, res, b, t, n, rows, K, R, K, K, ldo, ldo, R, R, p.dual, 0.f, 0.f, 1, stream);
    else
      rc = tahb_gemm(w, x, out, res, b, t, n, stacked ? rows / 2 : rows, K, R, K, K, ldo, res ? ldo : 0, R, R, p.dual, stacked ? rows / 2 : 0,
                     p.splits, p.bn, a->status, stream);
  };
  auto adapter = [&](const TahbProductPlan& p, const void* A, const void* x, void* t, int K, int R) {
    if (R) product(p, A, x, t, nullptr, nullptr, nullptr, R, K, 0, R);
  };
  auto norm = [&](const void* w) {
    if (rc) return;
    ++count;
    rc = tahb_rmsnorm(a->h, w, a->xn, n, H, H, H, a->eps, stream);
  };
  norm(a->layers[0].ln1);
  for (int li = 0; li < a->n_layers && !rc; ++li) {
    const TahbPassWeights& L = a->layers[li];
    if (a->taps[li] != nullptr &&
        cudaMemcpyAsync(a->taps[li], a->h, (size_t)n * H * 2, cudaMemcpyDeviceToDevice, stream) != cudaSuccess)
      return -40;
    adapter(a->p_a_qkv, L.a_qkv, a->xn, a->t_qkv, H, a->r_qkv);
    product(a->p_qkv, L.w_qkv, a->xn, a->qkv, nullptr, L.b_qkv, a->t_qkv, F, H, a->r_qkv, F);
    if (rc) break;
    void* cache[1] = {a->pool[li]};
    rc = tahb_qk_norm_rope_kv(a->qkv, L.q_norm, L.k_norm, a->q, a->k_own[li], a->v_own[li], cache, 1, nullptr, a->slots, a->pos, n, a->nq,
                              a->nkv, a->hd, a->page_size, F, a->eps, a->theta, stream);
    if (rc) break;
    void *ks[3], *vs[3];
    for (int s = 0; s + 1 < a->n_seg; ++s) {
      ks[s] = a->k_seg[s][li];
      vs[s] = a->v_seg[s][li];
    }
    ks[a->n_seg - 1] = a->k_own[li];
    vs[a->n_seg - 1] = a->v_own[li];
    rc = tahb_prefill_attn(a->q, a->o, ks, vs, a->n_kv, a->base, a->count, a->count, a->n_seg, a->tile_q0, a->tile_qn, a->n_tiles, n, a->nq,
                           a->nkv, a->hd, a->scale, nullptr, a->attn_heads, a->status, stream);
    count += 2;
    adapter(a->p_a_o, L.a_o, a->o, a->t_o, D, a->r_o);
    product(a->p_o, L.w_o, a->o, a->h, a->h, L.b_o, a->t_o, H, D, a->r_o, H);
    norm(L.ln2);
    adapter(a->p_a_gu, L.a_gu, a->xn, a->t_gu, H, a->r_gu);
    product(a->p_gu, L.w_gu, a->xn, a->act, nullptr, L.b_gu, a->t_gu, 2 * I, H, a->r_gu, I);
    adapter(a->p_a_down, L.a_down, a->act, a->t_down, I, a->r_down);
    product(a->p_down, L.w_down, a->act, a->h, a->h, L.b_down, a->t_down, H, I, a->r_down, H);
    norm(li + 1 < a->n_layers ? a->layers[li + 1].ln1 : a->final_norm);
  }
  *launches = count;
  return rc;
}
