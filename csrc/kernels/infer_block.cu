// The two halves of a pre-norm decoder block at inference, each as one call: the launches are those of the single
// operators, but a block costs the host two calls and a handful of allocations instead of a Python operator (autograd
// node, argument checks, stream look-up, call) per launch. With ~30 us per operator the host was what bounded decoding:
// 0.93 ms per token for two layers and the head of a 1024-wide model whose kernels take 0.18 ms.
// Nothing is kept between calls; every buffer belongs to the caller.
#include "sm100.cuh"
#include "tpb_api.h"

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
