// The layers of a dense decoder over a batch of prompt rows, launched by one call: per layer QKV product with rotation and cache write, attention, O
// product, residual and norm, gate/up product with SwiGLU, down product, residual and norm -- the launchers that the operators of the
// Python side call one by one, in the same order and with the same arguments. Nothing is computed here. What it is for: a launch through the
// operators takes 20 us of host time, so that prompts of up to a hundred rows were bound by the host (37 rows, 8 layers of an 8B-sized stack: 64
// launches, 1495 -> 1249 us a call).
#include "launchers.h"
#include <stddef.h>

using namespace ff;

struct FfDenseLayer { const void *wqkv, *wo, *post_ln, *wgu, *wdown, *next_ln; void *kcache, *vcache; };

// x: residual rows [rows, hidden], n: normed rows, in and out; qkv, att, mid, o: rows of (hq + 2 hkv) * 128, hq * 128, ffn and hidden elements.
// cos_sin: rotation table of the rows (ff_rope_table).
struct FfDenseStack {
  void *x, *n, *qkv, *att, *mid, *o;
  const float* cos_sin;
  const int *slots, *block_table, *q_start, *q_lens, *ctx_lens;
  float* scratch;
  int* counters;
  int* status;
  long long scratch_bytes, counter_bytes;
  int layers, rows, hidden, ffn, hq, hkv, batch, max_q_len, max_blocks, num_blocks, window;
  float scale, eps;
};

// scratch of the decode products of a stack's shapes, in bytes. Rows beyond what the decode product takes (FF_SKINNY_MAX_ROWS) are refused: there the
// operators called one by one are as quick.
FF_EXPORT int ff_dense_stack_workspace(int rows, int hidden, int ffn, int hq, int hkv, long long* scratch_bytes, long long* counter_bytes) {
  *scratch_bytes = *counter_bytes = 0;
  if (rows <= 0) return FF_HOST_BAD_SHAPE;
  if (rows > FF_SKINNY_MAX_ROWS) return FF_HOST_TOO_LARGE;
  auto take = [&](int grid, long long sb, long long cb) {
    if (sb > *scratch_bytes) *scratch_bytes = sb;
    if (cb > *counter_bytes) *counter_bytes = cb;
    return grid < 0 ? grid : FF_HOST_OK;
  };
  long long sb = 0, cb = 0;
  int g = ff_gemm_skinny_plan_epi(rows, (hq + 2 * hkv) * 128, hidden, 2, &sb, &cb);
  if (int r = take(g, sb, cb)) return r;
  g = ff_gemm_skinny_plan(rows, hidden, hq * 128, &sb, &cb);
  if (int r = take(g, sb, cb)) return r;
  g = ff_gemm_skinny_plan_epi(rows, 2 * ffn, hidden, 1, &sb, &cb);
  if (int r = take(g, sb, cb)) return r;
  g = ff_gemm_skinny_plan(rows, hidden, ffn, &sb, &cb);
  return take(g, sb, cb);
}

FF_EXPORT int ff_dense_stack(const FfDenseLayer* layers, const FfDenseStack* a, cudaStream_t s) {
  if (layers == nullptr || a == nullptr || a->layers <= 0 || a->rows <= 0 || a->hidden % 8 || a->ffn % 128 || a->hq <= 0 || a->hkv <= 0 || a->cos_sin == nullptr) return FF_HOST_BAD_SHAPE;
  const int rows = a->rows, hidden = a->hidden, ffn = a->ffn, qkv_dim = (a->hq + 2 * a->hkv) * 128, att_dim = a->hq * 128;
  long long sb = 0, cb = 0;
  if (int r = ff_dense_stack_workspace(rows, hidden, ffn, a->hq, a->hkv, &sb, &cb)) return r;
  if (sb > a->scratch_bytes || cb > a->counter_bytes) return FF_HOST_TOO_LARGE;
  auto product = [&](const void* x, const void* w, void* y, int n, int k) -> int {
    const int grid = ff_gemm_skinny_plan(rows, n, k, nullptr, nullptr);
    return grid < 0 ? grid : ff_gemm_skinny(x, w, y, rows, n, k, k, k, n, grid, a->scratch, a->counters, a->status, s);
  };
  for (int i = 0; i < a->layers; ++i) {
    const FfDenseLayer& l = layers[i];
    const int gq = ff_gemm_skinny_plan_epi(rows, qkv_dim, hidden, 2, nullptr, nullptr), gu = ff_gemm_skinny_plan_epi(rows, 2 * ffn, hidden, 1, nullptr, nullptr);
    if (gq < 0 || gu < 0) return gq < 0 ? gq : gu;
    if (int r = ff_gemm_skinny_rope_kv(a->n, l.wqkv, a->qkv, rows, qkv_dim, hidden, hidden, hidden, qkv_dim, gq, a->scratch, a->counters, a->cos_sin, a->slots,
                                       l.kcache, l.vcache, a->hq, a->hkv, 128, 64, a->num_blocks, a->status, s)) return r;
    if (int r = ff_attn_prefill_tc(a->qkv, l.kcache, l.vcache, a->block_table, a->q_start, a->q_lens, a->ctx_lens, a->att, a->batch, rows, a->max_q_len, a->hq,
                                   a->hkv, 128, 128, qkv_dim, att_dim, a->max_blocks, a->num_blocks, a->scale, a->window, 0, nullptr, nullptr, 0, 128, 0, 0.f,
                                   nullptr, 0, a->status, s)) return r;
    if (int r = product(a->att, l.wo, a->o, hidden, att_dim)) return r;
    if (int r = ff_add_rmsnorm(a->o, a->x, l.post_ln, a->n, nullptr, 0, rows, hidden, hidden, a->eps, 0, a->status, s)) return r;
    if (int r = ff_gemm_skinny_swiglu(a->n, l.wgu, a->mid, rows, 2 * ffn, hidden, hidden, hidden, ffn, gu, a->scratch, a->counters, 0, 0.f, a->status, s)) return r;
    if (int r = product(a->mid, l.wdown, a->o, hidden, ffn)) return r;
    if (int r = ff_add_rmsnorm(a->o, a->x, l.next_ln, a->n, nullptr, 0, rows, hidden, hidden, a->eps, 0, a->status, s)) return r;
  }
  return FF_HOST_OK;
}
