// The two halves of a pre-norm decoder block at inference, each as one call: the launches are those of the single
// operators, but a block costs the host two calls and a handful of allocations instead of a Python operator (autograd
// node, argument checks, stream look-up, call) per launch. With ~30 us per operator the host was what bounded decoding:
// 0.93 ms per token for two layers and the head of a 1024-wide model whose kernels take 0.18 ms.
// Nothing is kept between calls; every buffer belongs to the caller.
#include "sm100.cuh"
#include "tpb_api.h"

namespace tpb {
thread_local bool t_chained = false;
namespace {
struct Chain {   // the launches of this thread follow one another early, until the end of the scope
  Chain() { t_chained = true; }
  ~Chain() { t_chained = false; }
};
}  // namespace
}  // namespace tpb

#define TPB_TRY(call)          \
  do {                         \
    const int r_ = (call);     \
    if (r_) return r_;         \
  } while (0)

// h = rmsnorm(x) ; qkv = h Wqkv^T ; qk = rotated query and key heads of qkv.
// x, h [rows, hidden]; qkv [rows, (Hq + 2 Hkv) D]; qk [rows, (Hq + Hkv) D]; all contiguous bf16. pos: int64 [rows], or
// null for positions pos0 + (row % T).
extern "C" int tpb_block_pre(const void* x, const void* norm_w, float eps, const void* w_qkv, void* h, void* qkv,
                             void* qk, const float* cos_t, const float* sin_t, const long long* pos, long long pos0,
                             int rows, int T, int hidden, int Hq, int Hkv, int D, uint32_t* status, void* stream) {
  TPB_NVTX("tpb_block_pre");
  const int tot = Hq + 2 * Hkv;
  TPB_TRY(tpb_rmsnorm_fwd(x, nullptr, norm_w, h, nullptr, nullptr, rows, hidden, hidden, hidden, eps, stream));
  TPB_TRY(tpb_gemm_bf16(h, w_qkv, qkv, nullptr, rows, tot * D, hidden, hidden, hidden, tot * D, 0, 0, 0, 0, 0, 1.f,
                        status, stream));
  const long long skip = pos ? 0 : pos0 * (D / 2);
  return tpb_rope_out(qkv, qk, cos_t + skip, sin_t + skip, pos, rows, Hq + Hkv, D, (long long)tot * D, D,
                      (long long)(Hq + Hkv) * D, D, T, 0, 0, stream);
}

// o = attn Wo^T ; x2 = o + x, h = rmsnorm(x2) ; gu = h Wgu^T ; act = silu(gate) * up ; y (+)= act Wdown^T.
// With accumulate the last product is added to y (which the caller then makes x2 itself).
extern "C" int tpb_block_post(const void* attn, const void* w_o, void* o, const void* x, const void* norm_w, float eps,
                              void* x2, void* h, const void* w_gu, void* gu, void* act, const void* w_down, void* y,
                              int accumulate, int rows, int hidden, int attn_width, int inter, uint32_t* status,
                              void* stream) {
  TPB_NVTX("tpb_block_post");
  TPB_TRY(tpb_gemm_bf16(attn, w_o, o, nullptr, rows, hidden, attn_width, attn_width, attn_width, hidden, 0, 0, 0, 0, 0,
                        1.f, status, stream));
  TPB_TRY(tpb_rmsnorm_fwd(o, x, norm_w, h, x2, nullptr, rows, hidden, hidden, hidden, eps, stream));
  TPB_TRY(tpb_gemm_bf16(h, w_gu, gu, nullptr, rows, 2 * inter, hidden, hidden, hidden, 2 * inter, 0, 0, 0, 0, 0, 1.f,
                        status, stream));
  TPB_TRY(tpb_swiglu_fwd(gu, static_cast<const __nv_bfloat16*>(gu) + inter, act, rows, inter, 2LL * inter, stream));
  return tpb_gemm_bf16(act, w_down, y, nullptr, rows, hidden, inter, inter, inter, hidden, 0, 0, 0, 0, accumulate, 1.f,
                       status, stream);
}

// A forward pass of a whole decoder over a few rows (at most 128) with contiguous caches [B, Hkv, capacity, D]: embedding,
// layers, final norm and logits by the launches that the pass makes operator by operator, issued by one call. A step of a
// small model has some 25 kernels of 2-7 us, which the operators' Python takes three times as long to issue (one sequence,
// 2 layers of 1024, a prompt of 37 tokens and 8 steps: 3160 us operator by operator, of which kernels 1000).
// a: the words below, then 9 per layer.
enum LlamaWord {
  kLwTokens, kLwEmbed, kLwFinalNorm, kLwHead, kLwLogits, kLwCos, kLwSin, kLwPos, kLwStatus, kLwScratch, kLwPart, kLwPartLse,
  kLwLse, kLwLseStride, kLwSplits, kLwFewRows, kLwBatch, kLwT, kLwPast, kLwHidden, kLwHq, kLwHkv, kLwD, kLwInter, kLwVocab,
  kLwLayers, kLwHeader
};
enum LayerWord { kLyAttnNorm, kLyQkv, kLyO, kLyFfnNorm, kLyGateUp, kLyDown, kLyK, kLyV, kLyCap, kLyWords };

// bf16 elements of scratch for `rows` rows: two residual streams, h, o, qkv, qk, attention, gate / up, activation.
extern "C" long long tpb_llama_cached_scratch(int rows, int hidden, int Hq, int Hkv, int D, int inter) {
  return (long long)rows * (4LL * hidden + (Hq + 2LL * Hkv) * D + (Hq + (long long)Hkv) * D + (long long)Hq * D + 3LL * inter);
}

extern "C" int tpb_llama_cached(const long long* a, float eps, float scale, void* stream) {
  TPB_NVTX("tpb_llama_cached");
  const int B = (int)a[kLwBatch], T = (int)a[kLwT], H = (int)a[kLwHidden], Hq = (int)a[kLwHq], Hkv = (int)a[kLwHkv];
  const int D = (int)a[kLwD], I = (int)a[kLwInter], V = (int)a[kLwVocab], layers = (int)a[kLwLayers], rows = B * T;
  const long long past = a[kLwPast];
  const int Tk = (int)past + T, tot = Hq + 2 * Hkv;
  if (rows <= 0 || rows > 128 || layers < 0) return -2;
  auto in = [&](long long w) { return reinterpret_cast<const void*>(w); };
  auto out = [&](long long w) { return reinterpret_cast<void*>(w); };
  uint32_t* status = reinterpret_cast<uint32_t*>(a[kLwStatus]);
  const float *cos_t = reinterpret_cast<const float*>(a[kLwCos]), *sin_t = reinterpret_cast<const float*>(a[kLwSin]);
  const long long* pos = reinterpret_cast<const long long*>(a[kLwPos]);
  float* lse = reinterpret_cast<float*>(a[kLwLse]);
  __nv_bfloat16* next = reinterpret_cast<__nv_bfloat16*>(a[kLwScratch]);
  auto take = [&](long long n) { __nv_bfloat16* p = next; next += rows * n; return p; };
  __nv_bfloat16 *x = take(H), *x2 = take(H), *h = take(H), *o = take(H), *qkv = take((long long)tot * D);
  __nv_bfloat16 *qk = take((long long)(Hq + Hkv) * D), *attn = take((long long)Hq * D), *gu = take(2LL * I), *act = take(I);
  TPB_TRY(tpb_embedding_fwd(reinterpret_cast<const long long*>(a[kLwTokens]), in(a[kLwEmbed]), x, rows, H, V, stream));
  // From here on each kernel starts while the one before still runs, and the products request their weights meanwhile. The
  // kernels without a part in this (products of more rows, prompts' attention) are launched and waited for as usual.
  // The pass of the figures above took 1340 us with launches that wait for one another, 955 so, of which the host 950.
  const tpb::Chain chain;
  for (int l = 0; l < layers; ++l) {
    const long long* w = a + kLwHeader + l * kLyWords;
    TPB_TRY(tpb_block_pre(x, in(w[kLyAttnNorm]), eps, in(w[kLyQkv]), h, qkv, qk, cos_t, sin_t, pos, past, rows, T, H, Hq, Hkv,
                          D, status, stream));
    const long long cap = w[kLyCap], qt = (long long)(Hq + Hkv) * D, vt = (long long)tot * D;   // token strides
    TPB_TRY(tpb_kv_append2(qk + (long long)Hq * D, qkv + (long long)(Hq + Hkv) * D, out(w[kLyK]), out(w[kLyV]), (int)past, B,
                           T, Hkv, D, T * qt, qt, D, T * vt, vt, D, Hkv * cap * D, D, cap * D, stream));
    if (a[kLwFewRows])
      TPB_TRY(tpb_flash_decode(qk, in(w[kLyK]), in(w[kLyV]), attn, lse, reinterpret_cast<float*>(a[kLwPart]),
                               reinterpret_cast<float*>(a[kLwPartLse]), B, T, Tk, Hq, Hkv, D, qt, D, T * qt, D, cap * D,
                               Hkv * cap * D, D, cap * D, Hkv * cap * D, (long long)Hq * D, D, (long long)T * Hq * D,
                               (int)a[kLwLseStride], 1, scale, 0, (int)a[kLwSplits], stream));
    else
      TPB_TRY(tpb_flash_fwd_ex(qk, in(w[kLyK]), in(w[kLyV]), attn, lse, B, T, Tk, Hq, Hkv, D, qt, D, T * qt, D, cap * D,
                               Hkv * cap * D, D, cap * D, Hkv * cap * D, (long long)Hq * D, D, (long long)T * Hq * D,
                               (int)a[kLwLseStride], 1, scale, status, stream, nullptr, 1, 0, 0, 0, nullptr, nullptr));
    TPB_TRY(tpb_block_post(attn, in(w[kLyO]), o, x, in(w[kLyFfnNorm]), eps, x2, h, in(w[kLyGateUp]), gu, act, in(w[kLyDown]),
                           x2, 1, rows, H, Hq * D, I, status, stream));
    __nv_bfloat16* t = x;
    x = x2;
    x2 = t;
  }
  TPB_TRY(tpb_rmsnorm_fwd(x, nullptr, in(a[kLwFinalNorm]), h, nullptr, nullptr, rows, H, H, H, eps, stream));
  return tpb_gemm_bf16(h, in(a[kLwHead]), out(a[kLwLogits]), nullptr, rows, V, H, H, H, V, 0, 0, 0, 0, 0, 1.f, status, stream);
}
