// One decoder layer of a training step, forward or backward, as a single native call: the launches of the schedule in models/llama.py for
// whole weights on one GPU.  From Python a launch costs 10 to 20 us, which bounds steps of small models (two layers of width 256 over 1024 tokens:
// 1520 us of host work for 450 us of kernels); from here about 3.  Nothing is kept between calls: the caller owns every buffer.
// The reference drives its layers from C++ modules too (src/nn/parallel_linear.cpp:31-106).
#include "kernels/lt_cuda.h"
#include "kernels/common/host.h"

#include <math.h>

extern "C" {

// M = B * T rows; all matrices row-major and dense.  bf16 but for rstd, lse, delta, dq_acc, part (fp32) and the tables.
struct LtLlamaLayer {
  int B, T, width, heads, kv_heads, head_dim, ffn, accumulate;
  float eps;
  const float *cos_t, *sin_t;                                            // [>= T, head_dim / 2]
  const void *attn_norm, *wqkv, *wo, *mlp_norm, *w_gu, *w_down;          // weights
  void *g_attn_norm, *g_wqkv, *g_wo, *g_mlp_norm, *g_w_gu, *g_w_down;    // their gradients: written, or added to with `accumulate`
  // forward: x -> x2; the others are kept for the way back
  const void* x;
  void *h1, *qkv, *o, *x1, *h2, *gu, *hm, *x2;
  float *rstd1, *rstd2, *lse;
  // backward: dx2 -> dx; gu becomes its own gradient, the others are scratch
  const void* dx2;
  void *dx, *dhm, *dh, *dx1, *d_o, *dqkv;
  float *delta, *dq_acc, *part;
};

#define LT_STEP(call)       \
  do {                      \
    const int _r = (call);  \
    if (_r) return _r;      \
  } while (0)

static int product(const void* a, const void* b, void* c, int M, int N, int K, int a_major, int b_major, const void* residual, int accumulate, void* st) {
  return lt_gemm_bf16(a, b, c, M, N, K, a_major ? M : K, b_major ? N : K, N, a_major, b_major, 0, nullptr, residual, residual ? N : 0, 0, accumulate, 1.f, 0, 0,
                      st);
}

static const void* at(const void* p, long long elements) { return static_cast<const char*>(p) + elements * 2; }
static void* into(void* p, long long elements) { return static_cast<char*>(p) + elements * 2; }

int lt_llama_layer_fwd(const LtLlamaLayer* a, void* stream) {
  const int M = a->B * a->T, W = a->width, F = a->ffn, D = a->head_dim, q = a->heads * D, kv = a->kv_heads * D, Q = q + 2 * kv;
  const long long row = Q, seq = (long long)a->T * Q, orow = q, oseq = (long long)a->T * q;
  LT_STEP(lt_norm_fwd(0, a->x, nullptr, a->attn_norm, nullptr, a->h1, nullptr, nullptr, a->rstd1, M, W, a->eps, stream));
  LT_STEP(product(a->h1, a->wqkv, a->qkv, M, Q, W, 0, 0, nullptr, 0, stream));
  LT_STEP(lt_rope(a->qkv, a->cos_t, a->sin_t, nullptr, M, a->T, a->heads + a->kv_heads, D, Q, 0, stream));
  LT_STEP(lt_flash_fwd(a->qkv, at(a->qkv, q), at(a->qkv, q + kv), a->o, a->lse, a->B, a->T, a->T, a->heads, a->kv_heads, D, seq, row, seq, row, seq, row, oseq,
                       orow, float(1.0 / sqrt(double(D))), 1, stream));
  LT_STEP(product(a->o, a->wo, a->x1, M, W, q, 0, 0, a->x, 0, stream));
  LT_STEP(lt_norm_fwd(0, a->x1, nullptr, a->mlp_norm, nullptr, a->h2, nullptr, nullptr, a->rstd2, M, W, a->eps, stream));
  LT_STEP(lt_gemm_glu_keep(a->h2, a->w_gu, a->hm, a->gu, M, F, W, W, W, F, 2ll * F, 2, stream));
  return product(a->hm, a->w_down, a->x2, M, W, F, 0, 0, a->x1, 0, stream);
}

int lt_llama_layer_bwd(const LtLlamaLayer* a, void* stream) {
  const int M = a->B * a->T, W = a->width, F = a->ffn, D = a->head_dim, q = a->heads * D, kv = a->kv_heads * D, Q = q + 2 * kv, acc = a->accumulate;
  const long long row = Q, seq = (long long)a->T * Q, orow = q, oseq = (long long)a->T * q;
  // feed-forward
  LT_STEP(product(a->dx2, a->w_down, a->dhm, M, F, W, 0, 1, nullptr, 0, stream));
  LT_STEP(product(a->dx2, a->hm, a->g_w_down, W, F, M, 1, 1, nullptr, acc, stream));
  LT_STEP(lt_swiglu_bwd(a->gu, a->dhm, a->gu, M, F, stream));
  LT_STEP(product(a->gu, a->w_gu, a->dh, M, W, 2 * F, 0, 1, nullptr, 0, stream));
  LT_STEP(product(a->gu, a->h2, a->g_w_gu, 2 * F, W, M, 1, 1, nullptr, acc, stream));
  LT_STEP(lt_norm_bwd(0, a->dh, a->x1, a->mlp_norm, nullptr, a->rstd2, a->dx2, a->dx1, a->part, nullptr, a->g_mlp_norm, nullptr, 0, acc, M, W, stream));
  // attention
  LT_STEP(product(a->dx1, a->wo, a->d_o, M, q, W, 0, 1, nullptr, 0, stream));
  LT_STEP(product(a->dx1, a->o, a->g_wo, W, q, M, 1, 1, nullptr, acc, stream));
  LT_STEP(lt_flash_bwd_rope(a->qkv, at(a->qkv, q), at(a->qkv, q + kv), a->o, a->lse, a->d_o, a->dqkv, into(a->dqkv, q), into(a->dqkv, q + kv), a->delta, a->dq_acc,
                            a->B, a->T, a->T, a->heads, a->kv_heads, D, seq, row, seq, row, seq, row, oseq, orow, oseq, orow, seq, row, seq, row,
                            float(1.0 / sqrt(double(D))), 1, a->cos_t, a->sin_t, stream));
  LT_STEP(product(a->dqkv, a->wqkv, a->dh, M, W, Q, 0, 1, nullptr, 0, stream));
  LT_STEP(product(a->dqkv, a->h1, a->g_wqkv, Q, W, M, 1, 1, nullptr, acc, stream));
  return lt_norm_bwd(0, a->dh, a->x, a->attn_norm, nullptr, a->rstd1, a->dx1, a->dx, a->part, nullptr, a->g_attn_norm, nullptr, 0, acc, M, W, stream);
}

}  // extern "C"
