// Memory-bound row kernels for sm_100a: RMSNorm / LayerNorm forward+backward, RoPE, SwiGLU / GELU,
// fused cross-entropy forward+backward. All use 16-byte vector accesses and fp32 math on bf16
// storage; each is sized so that one pass over HBM is the cost.
//
// Counterparts in the reference: p10/src/backend/cuda/norm/RMSNormKernels.cu:147-486,
// norm/LayerNormKernels.cu:172-1053, transformers/AttentionRopeKernels.cu:141-272,
// ActivationKernels.cu:420-520, SoftmaxKernels.cu + LossFillKernels.cu:354-470.
#include "sm100.cuh"
#include "tpb_api.h"

namespace tpb {

constexpr int kRowThreads = 256;
constexpr int kMaxVec = 8;  // 16-byte vectors per thread kept in registers

union Vec8 {
  uint4 u;
  __nv_bfloat162 h[4];
};

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  Vec8 v;
  v.u = u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(v.h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  Vec8 v;
#pragma unroll
  for (int i = 0; i < 4; ++i) v.h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return v.u;
}

// Sum over the TPR threads that share a row (TPR is a power of two, 8..256).
template <int TPR>
__device__ __forceinline__ float row_sum(float v, float* scratch /* kRowThreads/32 floats */) {
  constexpr int W = TPR < 32 ? TPR : 32;
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, W);
  if constexpr (TPR > 32) {
    const int warp = threadIdx.x >> 5;
    const int wpr = TPR / 32;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[warp] = v;
    __syncthreads();
    const int first = (warp / wpr) * wpr;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < wpr; ++i) s += scratch[first + i];
    v = s;
  }
  return v;
}
template <int TPR>
__device__ __forceinline__ float row_max(float v, float* scratch) {
  constexpr int W = TPR < 32 ? TPR : 32;
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o, W));
  if constexpr (TPR > 32) {
    const int warp = threadIdx.x >> 5;
    const int wpr = TPR / 32;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[warp] = v;
    __syncthreads();
    const int first = (warp / wpr) * wpr;
    float s = -INFINITY;
#pragma unroll
    for (int i = 0; i < wpr; ++i) s = fmaxf(s, scratch[first + i]);
    v = s;
  }
  return v;
}

// One partial row per CTA from the column sums of its RPB row groups: [sub][H] through shared memory, added in order.
template <int TPR, int VPT>
__device__ __forceinline__ void fold_row_groups(const float (&acc)[VPT][8], float* __restrict__ out, int H, float* sm) {
  constexpr int RPB = kRowThreads / TPR;
  const int t = threadIdx.x % TPR, sub = threadIdx.x / TPR, nvec = H / 8;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = t + i * TPR;
    if (v < nvec) {
      // Single stores: vector stores want the sums in register quads throughout the loop above, at the price of its
      // loads in flight. LayerNorm backward, us with vector / single stores: 65536 x 4096 603 / 416, 32768 x 8192
      // 836 / 562, 65536 x 1024 203 / 135, 87381 x 768 127 / 131; RMSNorm 131072 x 2048 525 / 366, others within 3 %.
#pragma unroll
      for (int j = 0; j < 8; ++j) (RPB == 1 ? out : sm + sub * H)[v * 8 + j] = acc[i][j];
    }
  }
  if constexpr (RPB > 1) {
    __syncthreads();
    for (int c = threadIdx.x; c < H; c += kRowThreads) {
      float s = 0.f;
#pragma unroll
      for (int r = 0; r < RPB; ++r) s += sm[r * H + c];
      out[c] = s;
    }
    __syncthreads();
  }
}
// Floats of shared memory that fold_row_groups needs: RPB groups of at most TPR * VPT vectors of 8.
template <int TPR, int VPT>
constexpr int fold_floats() { return TPR == kRowThreads ? 4 : kRowThreads * VPT * 8; }

// A load of what an earlier kernel of a chain may have written. Outside of a chain it is an ordinary one, which the compiler orders
// more freely: RMSNorm of 30001 rows of 768 18.7 us against 20.6, RoPE of 4096 x 40 heads of 128 12.30 against 12.44, SwiGLU of
// 8192 x 28672 229.0 against 230.3.
template <bool CHAINED>
__device__ __forceinline__ uint4 row_ld(const uint4* p) {
  if constexpr (CHAINED) return chain_ld(p);
  else return *p;
}

// ------------------------------------------------------------------ RMSNorm forward
// y = (x [+ res]) * rstd * w ; optionally writes the summed residual stream back (res_out).
template <int TPR, int VPT, bool CHAINED>
__global__ void __launch_bounds__(kRowThreads)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd_out, int rows,
                   int H, long long x_stride, long long y_stride, float eps) {
  __shared__ float scratch[kRowThreads / 32];
  constexpr int RPB = kRowThreads / TPR;
  const int t = threadIdx.x % TPR;
  const int nvec = H / 8;
  if (CHAINED) {
    chain_next();
    chain_wait();
  }
  for (long long row0 = (long long)blockIdx.x * RPB; row0 < rows; row0 += (long long)gridDim.x * RPB) {
    const long long row = row0 + threadIdx.x / TPR;
    const bool live = row < rows;
    uint4 xv[VPT];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = t + i * TPR;
      if (live && v < nvec) {
        uint4 a = row_ld<CHAINED>(reinterpret_cast<const uint4*>(x + row * x_stride) + v);
        float f[8];
        unpack8(a, f);
        if (res) {
          float g[8];
          unpack8(row_ld<CHAINED>(reinterpret_cast<const uint4*>(res + row * (long long)H) + v), g);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] += g[j];
          a = pack8(f);
          unpack8(a, f);  // the normalised value is computed from the rounded stream
          if (res_out) reinterpret_cast<uint4*>(res_out + row * (long long)H)[v] = a;
        }
        xv[i] = a;
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
      }
    }
    ss = row_sum<TPR>(ss, scratch);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (live && t == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = t + i * TPR;
      if (live && v < nvec) {
        float f[8], g[8];
        unpack8(xv[i], f);
        unpack8(reinterpret_cast<const uint4*>(w)[v], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
        reinterpret_cast<uint4*>(y + row * y_stride)[v] = pack8(f);
      }
    }
  }
}

// ------------------------------------------------------------------ RMSNorm backward
// dx = rstd * (w*dy - xhat * mean(w*dy*xhat)) [+ dres]; dw partials per CTA in `dw_part`
// ([gridDim.x, H] fp32), reduced by colsum_kernel.
template <int TPR, int VPT>
__global__ void __launch_bounds__(kRowThreads)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_part, int rows, int H, long long x_stride,
                   long long dy_stride, long long dx_stride) {
  __shared__ float scratch[kRowThreads / 32];
  constexpr int RPB = kRowThreads / TPR;
  const int t = threadIdx.x % TPR;
  const int sub = threadIdx.x / TPR;
  const int nvec = H / 8;
  float dwacc[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;

  for (long long row0 = (long long)blockIdx.x * RPB; row0 < rows; row0 += (long long)gridDim.x * RPB) {
    const long long row = row0 + sub;
    const bool live = row < rows;
    const float rstd = live ? rstd_in[row] : 0.f;
    uint4 xv[VPT], gv[VPT];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = t + i * TPR;
      if (live && v < nvec) {
        xv[i] = reinterpret_cast<const uint4*>(x + row * x_stride)[v];
        gv[i] = reinterpret_cast<const uint4*>(dy + row * dy_stride)[v];
        float xf[8], gf[8], wf[8];
        unpack8(xv[i], xf);
        unpack8(gv[i], gf);
        unpack8(reinterpret_cast<const uint4*>(w)[v], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float xh = xf[j] * rstd;
          dot += wf[j] * gf[j] * xh;
          dwacc[i][j] += gf[j] * xh;
        }
      }
    }
    dot = row_sum<TPR>(dot, scratch) / (float)H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = t + i * TPR;
      if (live && v < nvec) {
        float xf[8], gf[8], wf[8], o[8];
        unpack8(xv[i], xf);
        unpack8(gv[i], gf);
        unpack8(reinterpret_cast<const uint4*>(w)[v], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rstd * (wf[j] * gf[j] - xf[j] * rstd * dot);
        if (dres) {
          float r[8];
          unpack8(reinterpret_cast<const uint4*>(dres + row * (long long)H)[v], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += r[j];
        }
        reinterpret_cast<uint4*>(dx + row * dx_stride)[v] = pack8(o);
      }
    }
  }
  __shared__ __align__(16) float fold[fold_floats<TPR, VPT>()];
  fold_row_groups<TPR, VPT>(dwacc, dw_part + (size_t)blockIdx.x * H, H, fold);
}

// out[c] = sum_r part[r, c] for one or two (blockIdx.y) fp32 matrices [nrows, H] that a kernel before left as
// per-block partial rows. A few hundred rows are too few bytes to matter and many dependent steps if one thread
// walks a column (30 us at 592 x 4096): here a block owns 32 columns and its 32 warps take every 32nd row, eight
// loads in flight each, so a column is three round trips deep (4 us).
struct ColsumArgs {
  const float* part[2];
  float* out_f32[2];
  __nv_bfloat16* out_bf16[2];
};
constexpr int kColsumThreads = 1024;
__global__ void __launch_bounds__(kColsumThreads)
colsum_kernel(const ColsumArgs a, int nrows, int H, int accumulate) {
  __shared__ float sm[32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* __restrict__ part = a.part[blockIdx.y];
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < H) {
    for (int r0 = warp; r0 < nrows; r0 += 32 * 8) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = (r0 + 32 * j < nrows) ? part[(size_t)(r0 + 32 * j) * H + c] : 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) s += v[j];
    }
  }
  sm[warp][lane] = s;
  __syncthreads();
  // warp w sums column w of the block
  float t = sm[lane][warp];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  const int co = blockIdx.x * 32 + warp;
  if (lane == 0 && co < H) {
    float* of = a.out_f32[blockIdx.y];
    __nv_bfloat16* ob = a.out_bf16[blockIdx.y];
    if (of) of[co] = accumulate ? of[co] + t : t;
    if (ob) ob[co] = __float2bfloat16(accumulate ? __bfloat162float(ob[co]) + t : t);
  }
}
static void launch_colsum(const ColsumArgs& a, int n, int nrows, int H, int accumulate, cudaStream_t stream) {
  colsum_kernel<<<dim3((H + 31) / 32, n), kColsumThreads, 0, stream>>>(a, nrows, H, accumulate);
}

// Column sums of a bf16 matrix [rows, N] (the gradient of a bias): one partial row of fp32 sums per block, then
// colsum_kernel. Bound by reading the matrix once; a block is 256 columns (16 bytes a lane) by a slice of rows.
constexpr int kBiasRowsMin = 32;   // rows per block below which more blocks no longer pay
__global__ void __launch_bounds__(256)
bias_grad_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ part, int rows, int N, long long ld,
                 int rows_per_block) {
  __shared__ float sm[8][256 + 8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 256 + lane * 8;
  const int r1 = min(rows, ((int)blockIdx.y + 1) * rows_per_block);
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (c < N) {
    for (int r = blockIdx.y * rows_per_block + warp; r < r1; r += 32) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        v[u] = (r + 8 * u < r1) ? __ldg(reinterpret_cast<const uint4*>(x + (size_t)(r + 8 * u) * ld + c))
                                : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float f[8];
        unpack8(v[u], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += f[j];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) sm[warp][lane * 8 + j] = acc[j];
  __syncthreads();
  const int co = blockIdx.x * 256 + threadIdx.x;
  if (co < N) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += sm[w][threadIdx.x];
    part[(size_t)blockIdx.y * N + co] = s;
  }
}
static int bias_grad_chunks(int rows, int N) {
  const int cols = (N + 255) / 256;
  int n = (sm_count() * 8 + cols - 1) / cols;
  const int most = (rows + kBiasRowsMin - 1) / kBiasRowsMin;
  if (n > most) n = most;
  return n < 1 ? 1 : n;
}

// ------------------------------------------------------------------ LayerNorm
template <int TPR, int VPT>
__global__ void __launch_bounds__(kRowThreads)
layernorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                     const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ y,
                     float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int H,
                     float eps) {
  __shared__ float scratch[kRowThreads / 32];
  constexpr int RPB = kRowThreads / TPR;
  const int t = threadIdx.x % TPR;
  const int nvec = H / 8;
  for (long long row0 = (long long)blockIdx.x * RPB; row0 < rows; row0 += (long long)gridDim.x * RPB) {
    const long long row = row0 + threadIdx.x / TPR;
    const bool live = row < rows;
    uint4 xv[VPT];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = t + i * TPR;
      if (live && v < nvec) {
        xv[i] = reinterpret_cast<const uint4*>(x + row * (long long)H)[v];
        float f[8];
        unpack8(xv[i], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += f[j];
      }
    }
    const float mean = row_sum<TPR>(s, scratch) / (float)H;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = t + i * TPR;
      if (live && v < nvec) {
        float f[8];
        unpack8(xv[i], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += (f[j] - mean) * (f[j] - mean);
      }
    }
    const float rstd = rsqrtf(row_sum<TPR>(ss, scratch) / (float)H + eps);
    if (live && t == 0) {
      if (mean_out) mean_out[row] = mean;
      if (rstd_out) rstd_out[row] = rstd;
    }
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = t + i * TPR;
      if (live && v < nvec) {
        float f[8], g[8], bb[8];
        unpack8(xv[i], f);
        unpack8(reinterpret_cast<const uint4*>(w)[v], g);
        if (b) unpack8(reinterpret_cast<const uint4*>(b)[v], bb);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = (f[j] - mean) * rstd * g[j] + (b ? bb[j] : 0.f);
        reinterpret_cast<uint4*>(y + row * (long long)H)[v] = pack8(f);
      }
    }
  }
}

// dx = rstd * (g - mean(g) - xhat * mean(g*xhat)), g = w*dy; dw/db partial rows per CTA.
template <int TPR, int VPT>
__global__ void __launch_bounds__(kRowThreads)
layernorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                     const __nv_bfloat16* __restrict__ w, const float* __restrict__ mean_in,
                     const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
                     float* __restrict__ dw_part, float* __restrict__ db_part, int rows, int H) {
  __shared__ float scratch[kRowThreads / 32];
  constexpr int RPB = kRowThreads / TPR;
  const int t = threadIdx.x % TPR;
  const int sub = threadIdx.x / TPR;
  const int nvec = H / 8;
  float dwacc[VPT][8], dbacc[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = dbacc[i][j] = 0.f;
  for (long long row0 = (long long)blockIdx.x * RPB; row0 < rows; row0 += (long long)gridDim.x * RPB) {
    const long long row = row0 + sub;
    const bool live = row < rows;
    const float mean = live ? mean_in[row] : 0.f;
    const float rstd = live ? rstd_in[row] : 0.f;
    uint4 xv[VPT], gv[VPT];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = t + i * TPR;
      if (live && v < nvec) {
        xv[i] = reinterpret_cast<const uint4*>(x + row * (long long)H)[v];
        gv[i] = reinterpret_cast<const uint4*>(dy + row * (long long)H)[v];
        float xf[8], gf[8], wf[8];
        unpack8(xv[i], xf);
        unpack8(gv[i], gf);
        unpack8(reinterpret_cast<const uint4*>(w)[v], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float xh = (xf[j] - mean) * rstd;
          float g = wf[j] * gf[j];
          s1 += g;
          s2 += g * xh;
          dwacc[i][j] += gf[j] * xh;
          dbacc[i][j] += gf[j];
        }
      }
    }
    s1 = row_sum<TPR>(s1, scratch) / (float)H;
    s2 = row_sum<TPR>(s2, scratch) / (float)H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = t + i * TPR;
      if (live && v < nvec) {
        float xf[8], gf[8], wf[8], o[8];
        unpack8(xv[i], xf);
        unpack8(gv[i], gf);
        unpack8(reinterpret_cast<const uint4*>(w)[v], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float xh = (xf[j] - mean) * rstd;
          o[j] = rstd * (wf[j] * gf[j] - s1 - xh * s2);
        }
        reinterpret_cast<uint4*>(dx + row * (long long)H)[v] = pack8(o);
      }
    }
  }
  __shared__ __align__(16) float fold[fold_floats<TPR, VPT>()];
  fold_row_groups<TPR, VPT>(dwacc, dw_part + (size_t)blockIdx.x * H, H, fold);
  fold_row_groups<TPR, VPT>(dbacc, db_part + (size_t)blockIdx.x * H, H, fold);
}

// ------------------------------------------------------------------ RoPE (in place capable)
// x viewed as [tokens, heads, D] with explicit token/head strides (elements), y likewise with its
// own strides (y == x rotates in place: each thread reads all it needs before it writes). cos/sin
// tables are fp32 [max_pos, D/2]; pos[token] optional (else token % seq_len). sign = -1 for backward.
// Idx: 32-bit indices wherever they suffice; the three divisions that take an index apart were most of the kernel's
// instructions in 64 bits.
template <typename Idx, bool CHAINED>
__global__ void __launch_bounds__(256)
rope_kernel(const __nv_bfloat16* x, __nv_bfloat16* y, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, const long long* __restrict__ pos,
                            long long tokens, int heads, int D, long long tok_stride,
                            long long head_stride, long long y_tok_stride, long long y_head_stride,
                            int seq_len, int interleaved, float sign) {
  const int half = D / 2;
  const int vec_per_head = half / 8;  // NeoX: 8 pairs per thread from both halves
  const Idx idx = (Idx)blockIdx.x * 256 + threadIdx.x;
  const Idx total = (Idx)tokens * heads * vec_per_head;
  if (CHAINED) {
    chain_next();
    chain_wait();
  }
  if (idx >= total) return;
  const Idx th = idx / (Idx)vec_per_head;
  const int v = (int)(idx - th * vec_per_head);
  const Idx tk = th / (Idx)heads;
  const int h = (int)(th - tk * heads);
  const long long tok = (long long)tk;
  const long long p = pos ? pos[tok] : (long long)(tk % (Idx)seq_len);
  const __nv_bfloat16* base = x + tok * tok_stride + (long long)h * head_stride;
  __nv_bfloat16* obase = y + tok * y_tok_stride + (long long)h * y_head_stride;
  const float* c = cos_t + p * half;
  const float* s = sin_t + p * half;
  if (!interleaved) {
    uint4 a = row_ld<CHAINED>(reinterpret_cast<const uint4*>(base) + v);
    uint4 b = row_ld<CHAINED>(reinterpret_cast<const uint4*>(base + half) + v);
    float af[8], bf[8], oa[8], ob[8];
    unpack8(a, af);
    unpack8(b, bf);
    // cos / sin of this thread's eight pairs as four 16-byte loads (half is a multiple of 8 floats, the tables
    // are 16-byte aligned rows)
    const float4 c0 = __ldg(reinterpret_cast<const float4*>(c + v * 8)), c1 = __ldg(reinterpret_cast<const float4*>(c + v * 8) + 1);
    const float4 s0 = __ldg(reinterpret_cast<const float4*>(s + v * 8)), s1 = __ldg(reinterpret_cast<const float4*>(s + v * 8) + 1);
    const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn8[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float cc = cs[j], sn = sign * sn8[j];
      oa[j] = af[j] * cc - bf[j] * sn;
      ob[j] = bf[j] * cc + af[j] * sn;
    }
    reinterpret_cast<uint4*>(obase)[v] = pack8(oa);
    reinterpret_cast<uint4*>(obase + half)[v] = pack8(ob);
  } else {
    // 16 consecutive elements = 8 (even, odd) pairs: two vectors per thread
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint4 a = row_ld<CHAINED>(reinterpret_cast<const uint4*>(base) + v * 2 + q);
      float f[8], o[8];
      unpack8(a, f);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int pi = v * 8 + q * 4 + j;
        float cc = c[pi], sn = sign * s[pi];
        o[2 * j] = f[2 * j] * cc - f[2 * j + 1] * sn;
        o[2 * j + 1] = f[2 * j + 1] * cc + f[2 * j] * sn;
      }
      reinterpret_cast<uint4*>(obase)[v * 2 + q] = pack8(o);
    }
  }
}

// ------------------------------------------------------------------ SwiGLU / GELU
// out[r, i] = silu(gate[r, i]) * up[r, i]; gate/up given with a common row stride.
// Bound by memory. A thread takes kActVecs vectors of eight elements, one block's width apart, with all their loads in
// flight together; the vector index is 32 bits wide wherever that suffices (Idx), since the division that splits it into
// row and column costs some ninety instructions in 64 bits, more than the arithmetic of the eight elements.
constexpr int kActVecs = 2;
template <typename Idx, bool CHAINED>
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ up,
                  __nv_bfloat16* __restrict__ out, long long rows, int I, long long in_stride,
                  const int* __restrict__ rows_dev) {
  const Idx nvec = I / 8;
  if (CHAINED) {
    chain_next();
    chain_wait();
  }
  if (rows_dev) rows = min(rows, (long long)*rows_dev);  // row count known only on the device (ragged buffers)
  const Idx total = (Idx)rows * nvec;
  const Idx i0 = (Idx)blockIdx.x * (256 * kActVecs) + threadIdx.x;
  uint4 gv[kActVecs], uv[kActVecs];
#pragma unroll
  for (int k = 0; k < kActVecs; ++k) {
    const Idx idx = i0 + k * 256;
    if (idx >= total) break;
    const Idx r = idx / nvec;
    const int v = (int)(idx - r * nvec);
    gv[k] = row_ld<CHAINED>(reinterpret_cast<const uint4*>(gate + (long long)r * in_stride) + v);
    uv[k] = row_ld<CHAINED>(reinterpret_cast<const uint4*>(up + (long long)r * in_stride) + v);
  }
#pragma unroll
  for (int k = 0; k < kActVecs; ++k) {
    const Idx idx = i0 + k * 256;
    if (idx >= total) break;
    float g[8], u[8], o[8];
    unpack8(gv[k], g);
    unpack8(uv[k], u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    reinterpret_cast<uint4*>(out)[idx] = pack8(o);   // rows of out are contiguous
  }
}
template <typename Idx>
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ gate,
                  const __nv_bfloat16* __restrict__ up, __nv_bfloat16* __restrict__ dgate,
                  __nv_bfloat16* __restrict__ dup, long long rows, int I, long long in_stride, long long out_stride,
                  const int* __restrict__ rows_dev) {
  const Idx nvec = I / 8;
  if (rows_dev) rows = min(rows, (long long)*rows_dev);
  const Idx total = (Idx)rows * nvec;
  const Idx i0 = (Idx)blockIdx.x * (256 * kActVecs) + threadIdx.x;
  uint4 gv[kActVecs], uv[kActVecs], dv[kActVecs];
  Idx row[kActVecs];
  int col[kActVecs];
#pragma unroll
  for (int k = 0; k < kActVecs; ++k) {
    const Idx idx = i0 + k * 256;
    if (idx >= total) break;
    row[k] = idx / nvec;
    col[k] = (int)(idx - row[k] * nvec);
    gv[k] = reinterpret_cast<const uint4*>(gate + (long long)row[k] * in_stride)[col[k]];
    uv[k] = reinterpret_cast<const uint4*>(up + (long long)row[k] * in_stride)[col[k]];
    dv[k] = reinterpret_cast<const uint4*>(dy)[idx];
  }
#pragma unroll
  for (int k = 0; k < kActVecs; ++k) {
    const Idx idx = i0 + k * 256;
    if (idx >= total) break;
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(gv[k], g);
    unpack8(uv[k], u);
    unpack8(dv[k], d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float sg = 1.f / (1.f + __expf(-g[j]));
      float silu = g[j] * sg;
      du[j] = d[j] * silu;
      dg[j] = d[j] * u[j] * (sg + silu * (1.f - sg));
    }
    reinterpret_cast<uint4*>(dgate + (long long)row[k] * out_stride)[col[k]] = pack8(dg);
    reinterpret_cast<uint4*>(dup + (long long)row[k] * out_stride)[col[k]] = pack8(du);
  }
}

// GELU; approx = 1 selects the tanh form, evaluated as x * sigmoid(2u) with u = sqrt(2/pi) (x + 0.044715 x^3): the
// same function as 0.5 x (1 + tanh u), without the cancellation of 1 + tanh for negative u, and one exponential and one
// division where tanhf takes some thirty instructions. The pass was bound by those: 54 us forward and 68 us backward at
// 16384 x 3072 against 30 and 45 us of memory time.
__device__ __forceinline__ float sigmoid_2u(float u) { return __fdividef(1.f, 1.f + __expf(-2.f * u)); }
__device__ __forceinline__ float gelu_f(float x, int approx) {
  if (approx) return x * sigmoid_2u(0.7978845608028654f * (x + 0.044715f * x * x * x));
  return 0.5f * x * (1.f + erff(x * 0.7071067811865476f));
}
__device__ __forceinline__ float gelu_grad_f(float x, int approx) {
  if (approx) {
    const float s = sigmoid_2u(0.7978845608028654f * (x + 0.044715f * x * x * x));
    const float du2 = 2.f * 0.7978845608028654f * (1.f + 3.f * 0.044715f * x * x);
    return s + x * (s * (1.f - s)) * du2;
  }
  float cdf = 0.5f * (1.f + erff(x * 0.7071067811865476f));
  float pdf = 0.3989422804014327f * __expf(-0.5f * x * x);
  return cdf + x * pdf;
}
__global__ void gelu_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                                long long nvec, int approx) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nvec) return;
  float f[8];
  unpack8(reinterpret_cast<const uint4*>(x)[idx], f);
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = gelu_f(f[j], approx);
  reinterpret_cast<uint4*>(y)[idx] = pack8(f);
}
__global__ void gelu_bwd_kernel(const __nv_bfloat16* __restrict__ dy,
                                const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ dx,
                                long long nvec, int approx) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nvec) return;
  float f[8], d[8];
  unpack8(reinterpret_cast<const uint4*>(x)[idx], f);
  unpack8(reinterpret_cast<const uint4*>(dy)[idx], d);
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = d[j] * gelu_grad_f(f[j], approx);
  reinterpret_cast<uint4*>(dx)[idx] = pack8(f);
}

// ------------------------------------------------------------------ cross-entropy (fwd + bwd fused)
// One CTA per row. Pass 1: online max / sum-exp over the vocabulary. Pass 2 (if dlogits):
// dlogits = (softmax - onehot) * gscale, written in place or to a separate buffer.
// loss[row] = lse - logit[target]; rows whose target == ignore_index get loss 0 / grad 0.
// The forward pass reads the logits once; what bounds it is that and the instructions of each logit, one exponential
// (16 per cycle and SM: 117 us of 160 us of memory time at 4096 x 128256) and those around it. A thread requests four
// 16-byte vectors before it needs the first, takes the maximum of their 32 values on packed bf16 pairs, rescales its
// running sum once for all of them, and subtracts, scales and adds two logits at a time; vectors past the end of the row,
// most of the last round, are left out. Blocks of 256 threads, eight to an SM, have another row to read while one ends.
// With the loss's reduction, 16384 x 50257 / 4096 x 128256 / 4000 x 8000 took 428 / 238 / 81 us with 512 threads and one
// logit at a time; two at a time 368 / 204 / 73, and with 256 threads 298 / 194 / 56. Requesting the next round ahead costs
// half of the resident warps: 459 / 257 / 91.
// Few long rows leave SMs with one block or two, and a block's rounds are what takes the time: 512 threads (ce_threads).
// Two fp32 numbers in a register pair: one instruction adds or multiplies both.
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  return ((unsigned long long)__float_as_uint(y) << 32) | __float_as_uint(x);
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  return make_float2(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// Below 2^-126 the result is zero, which a sum that holds a term of one does not notice.
__device__ __forceinline__ float exp2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The sum of exp(x - mu) over eight bf16 numbers, as two halves.
__device__ __forceinline__ unsigned long long exp8_sum(const uint4& u, unsigned long long minus_mu) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  const float log2e = 1.4426950408889634f;
  unsigned long long acc = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const unsigned long long x = ((unsigned long long)(w[j] & 0xffff0000u) << 32) | (w[j] << 16);
    const float2 e = unpack2(mul2(add2(x, minus_mu), pack2(log2e, log2e)));
    acc = add2(acc, pack2(exp2_ftz(e.x), exp2_ftz(e.y)));
  }
  return acc;
}
constexpr int kCeVec = 4;
template <int kCeThreads>
__global__ void __launch_bounds__(kCeThreads)
cross_entropy_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ target,
                     float* __restrict__ loss, float* __restrict__ lse_out,
                     __nv_bfloat16* __restrict__ dlogits, int V, long long stride,
                     long long ignore_index, float gscale) {
  __shared__ float sm[kCeThreads / 32];
  __shared__ float ss[kCeThreads / 32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* lr = logits + row * stride;
  const long long tgt = target[row];
  const int nvec = V / 8;
  float m = -INFINITY, s = 0.f;
  for (int v0 = threadIdx.x; v0 < nvec; v0 += kCeThreads * kCeVec) {
    uint4 u[kCeVec];
#pragma unroll
    for (int k = 0; k < kCeVec; ++k) {
      const int v = v0 + k * kCeThreads;
      u[k] = v < nvec ? reinterpret_cast<const uint4*>(lr)[v]
                      : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);   // -inf: adds nothing
    }
    __nv_bfloat162 mx = *reinterpret_cast<__nv_bfloat162*>(&u[0].x);
#pragma unroll
    for (int k = 0; k < kCeVec; ++k) {
      const __nv_bfloat162* hp = reinterpret_cast<const __nv_bfloat162*>(&u[k]);
#pragma unroll
      for (int j = 0; j < 4; ++j) mx = __hmax2(mx, hp[j]);
    }
    const float2 m2 = __bfloat1622float2(mx);
    const float nm = fmaxf(m, fmaxf(m2.x, m2.y));
    const float mu = nm == -INFINITY ? 0.f : nm;   // nothing but -inf so far
    const unsigned long long mu2 = pack2(-mu, -mu);
    unsigned long long acc = 0;
#pragma unroll
    for (int k = 0; k < kCeVec; ++k) {
      if (k > 0 && v0 + k * kCeThreads >= nvec) break;   // most of a last round
      acc = add2(acc, exp8_sum(u[k], mu2));
    }
    const float2 a2 = unpack2(acc);
    s = s * __expf(m - mu) + (a2.x + a2.y);
    m = nm;
  }
  for (int i = nvec * 8 + threadIdx.x; i < V; i += kCeThreads) {
    float f = __bfloat162float(lr[i]);
    float nm = fmaxf(m, f);
    const float mu = nm == -INFINITY ? 0.f : nm;
    s = s * __expf(m - mu) + __expf(f - mu);
    m = nm;
  }
  // block combine of (m, s)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float om = __shfl_xor_sync(0xffffffffu, m, o);
    float os = __shfl_xor_sync(0xffffffffu, s, o);
    float nm = fmaxf(m, om);
    s = (nm == -INFINITY) ? 0.f : s * __expf(m - nm) + os * __expf(om - nm);
    m = nm;
  }
  if ((threadIdx.x & 31) == 0) { sm[threadIdx.x >> 5] = m; ss[threadIdx.x >> 5] = s; }
  __syncthreads();
  float gm = -INFINITY;
#pragma unroll
  for (int i = 0; i < kCeThreads / 32; ++i) gm = fmaxf(gm, sm[i]);
  float gs = 0.f;
#pragma unroll
  for (int i = 0; i < kCeThreads / 32; ++i)
    gs += (sm[i] == -INFINITY) ? 0.f : ss[i] * __expf(sm[i] - gm);
  const float lse = gm + __logf(gs);
  const bool ignored = (tgt == ignore_index) || !TPB_DBG_CHECK(tgt >= 0 && tgt < V, 43);
  if (threadIdx.x == 0) {
    if (lse_out) lse_out[row] = lse;
    if (loss) loss[row] = ignored ? 0.f : lse - __bfloat162float(lr[tgt]);
  }
  if (!dlogits) return;
  __nv_bfloat16* dr = dlogits + row * stride;
  const float gsc = ignored ? 0.f : gscale;
  for (int v = threadIdx.x; v < nvec; v += kCeThreads) {
    float f[8];
    unpack8(reinterpret_cast<const uint4*>(lr)[v], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float pr = __expf(f[j] - lse);
      if ((long long)(v * 8 + j) == tgt) pr -= 1.f;
      f[j] = pr * gsc;
    }
    reinterpret_cast<uint4*>(dr)[v] = pack8(f);
  }
  for (int i = nvec * 8 + threadIdx.x; i < V; i += kCeThreads) {
    float pr = __expf(__bfloat162float(lr[i]) - lse);
    if (i == tgt) pr -= 1.f;
    dr[i] = __float2bfloat16(pr * gsc);
  }
}

// Backward from a saved log-sum-exp: dlogits = (exp(l - lse) - onehot) * g, where
// g = g_scalar[0] * scale[0] (either may be null) or g_rows[row]. Grid (chunks, rows).
__global__ void __launch_bounds__(256)
cross_entropy_bwd_kernel(const __nv_bfloat16* __restrict__ logits,
                         const long long* __restrict__ target, const float* __restrict__ lse_in,
                         __nv_bfloat16* __restrict__ dlogits, const float* __restrict__ g_scalar,
                         const float* __restrict__ scale, const float* __restrict__ g_rows, int V,
                         long long stride, long long ignore_index) {
  const long long row = blockIdx.y;
  const long long tgt = target[row];
  const bool ignored = (tgt == ignore_index) || !TPB_DBG_CHECK(tgt >= 0 && tgt < V, 43);
  float g = g_rows ? g_rows[row] : 1.f;
  if (g_scalar) g *= *g_scalar;
  if (scale) g *= *scale;
  if (ignored) g = 0.f;
  const float lse = lse_in[row];
  const __nv_bfloat16* lr = logits + row * stride;
  __nv_bfloat16* dr = dlogits + row * stride;
  const int nvec = V / 8;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += gridDim.x * blockDim.x) {
    float f[8];
    unpack8(reinterpret_cast<const uint4*>(lr)[v], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float pr = __expf(f[j] - lse);
      if ((long long)(v * 8 + j) == tgt) pr -= 1.f;
      f[j] = pr * g;
    }
    reinterpret_cast<uint4*>(dr)[v] = pack8(f);
  }
  if (blockIdx.x == 0) {
    for (int i = nvec * 8 + threadIdx.x; i < V; i += blockDim.x) {
      float pr = __expf(__bfloat162float(lr[i]) - lse);
      if (i == tgt) pr -= 1.f;
      dr[i] = __float2bfloat16(pr * g);
    }
  }
}

// ------------------------------------------------------------------ launch helpers
// Threads per row. Rows of up to 1024 take one warp each: the row sums are shuffles only, so the eight rows of a CTA run
// without a block barrier (with 128 threads per row, 768 columns left a quarter of them idle and every row paid two to
// four barriers: LayerNorm 21 us forward and 30 us backward at 16384 x 768).
static int pick_tpr(int H) {
  int nvec = H / 8;
  return nvec <= 16 ? 16 : (nvec <= 128 ? 32 : (nvec <= 256 ? 128 : 256));
}
static int pick_vpt(int H, int tpr) {
  int need = (H / 8 + tpr - 1) / tpr;
  if (tpr == 32) return need;   // 1..4
  int v = 1;
  while (v < need) v <<= 1;
  return v;
}
int row_grid(int rows, int tpr) {
  int rpb = kRowThreads / tpr;
  long long blocks = ((long long)rows + rpb - 1) / rpb;
  long long cap = (long long)sm_count() * 8;
  return (int)(blocks < cap ? blocks : cap);
}

#define TPB_VPT_SWITCH(vpt, ...)                          \
  switch (vpt) {                                          \
    case 1: { constexpr int VPT = 1; __VA_ARGS__; } break; \
    case 2: { constexpr int VPT = 2; __VA_ARGS__; } break; \
    case 4: { constexpr int VPT = 4; __VA_ARGS__; } break; \
    case 8: { constexpr int VPT = 8; __VA_ARGS__; } break; \
    default: return -2;                                   \
  }
#define TPB_ROW_SWITCH(tpr, vpt, ...)                                          \
  switch (tpr) {                                                               \
    case 16: { constexpr int TPR = 16; constexpr int VPT = 1; __VA_ARGS__; } break; \
    case 32: {                                                                 \
      constexpr int TPR = 32;                                                  \
      switch (vpt) {                                                           \
        case 1: { constexpr int VPT = 1; __VA_ARGS__; } break;                 \
        case 2: { constexpr int VPT = 2; __VA_ARGS__; } break;                 \
        case 3: { constexpr int VPT = 3; __VA_ARGS__; } break;                 \
        default: { constexpr int VPT = 4; __VA_ARGS__; } break;                \
      }                                                                        \
    } break;                                                                   \
    case 128: {                                                                \
      constexpr int TPR = 128;                                                 \
      constexpr int VPT = 2;                                                   \
      __VA_ARGS__;                                                             \
    } break;                                                                   \
    case 256: { constexpr int TPR = 256; TPB_VPT_SWITCH(vpt, __VA_ARGS__) } break; \
    default: return -2;                                                        \
  }

}  // namespace tpb

using namespace tpb;

extern "C" int tpb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* res_out,
                               float* rstd, int rows, int H, long long x_stride,
                               long long y_stride, float eps, void* stream) {
  TPB_NVTX("tpb_rmsnorm_fwd");
  if (H % 8 || H > 256 * kMaxVec * 8) return -2;
  if (rows <= 0) return 0;
  int tpr = pick_tpr(H);
  int grid = ((long long)rows + kRowThreads / tpr - 1) / (kRowThreads / tpr);
  cudaError_t e = cudaSuccess;
  TPB_ROW_SWITCH(tpr, pick_vpt(H, tpr), (e = launch_chained(
                          t_chained ? rmsnorm_fwd_kernel<TPR, VPT, true> : rmsnorm_fwd_kernel<TPR, VPT, false>, dim3(grid), kRowThreads, (cudaStream_t)stream,
                          (const __nv_bfloat16*)x, (const __nv_bfloat16*)res,
                          (const __nv_bfloat16*)w, (__nv_bfloat16*)y, (__nv_bfloat16*)res_out, rstd,
                          rows, H, x_stride, y_stride, eps)));
  return (int)e;
}

extern "C" int tpb_rmsnorm_bwd_grid(int rows, int H) {
  if (H % 8 || H > 256 * kMaxVec * 8) return -2;
  int tpr = pick_tpr(H);
  int g = row_grid(rows, tpr);
  // 4 CTAs of 62-64 registers x 256 threads fit an SM; each CTA works through its rows one after the
  // other (load, row reduction, store), so resident CTAs are what hides the memory latency
  int cap = sm_count() * 4;
  return g < cap ? g : cap;
}

// dw_part must hold tpb_rmsnorm_bwd_grid(rows, H) * H floats.
extern "C" int tpb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd,
                               const void* dres, void* dx, float* dw_part, float* dw_f32,
                               void* dw_bf16, int dw_accumulate, int rows, int H,
                               long long x_stride, long long dy_stride, long long dx_stride,
                               void* stream) {
  TPB_NVTX("tpb_rmsnorm_bwd");
  if (H % 8 || H > 256 * kMaxVec * 8) return -2;
  if (rows <= 0) return 0;
  int tpr = pick_tpr(H);
  int grid = tpb_rmsnorm_bwd_grid(rows, H);
  TPB_ROW_SWITCH(tpr, pick_vpt(H, tpr), (rmsnorm_bwd_kernel<TPR, VPT><<<grid, kRowThreads, 0, (cudaStream_t)stream>>>(
                          (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,
                          (const __nv_bfloat16*)w, rstd, (const __nv_bfloat16*)dres,
                          (__nv_bfloat16*)dx, dw_part, rows, H, x_stride, dy_stride, dx_stride)));
  launch_colsum({{dw_part, nullptr}, {dw_f32, nullptr}, {(__nv_bfloat16*)dw_bf16, nullptr}}, 1, grid, H, dw_accumulate,
                (cudaStream_t)stream);
  return (int)cudaGetLastError();
}

extern "C" int tpb_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean,
                                 float* rstd, int rows, int H, float eps, void* stream) {
  TPB_NVTX("tpb_layernorm_fwd");
  if (H % 8 || H > 256 * kMaxVec * 8) return -2;
  if (rows <= 0) return 0;
  int tpr = pick_tpr(H);
  int grid = ((long long)rows + kRowThreads / tpr - 1) / (kRowThreads / tpr);
  TPB_ROW_SWITCH(tpr, pick_vpt(H, tpr), (layernorm_fwd_kernel<TPR, VPT><<<grid, kRowThreads, 0, (cudaStream_t)stream>>>(
                          (const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
                          (const __nv_bfloat16*)b, (__nv_bfloat16*)y, mean, rstd, rows, H, eps)));
  return (int)cudaGetLastError();
}

// dw_part / db_part: tpb_rmsnorm_bwd_grid(rows, H) * H floats each.
extern "C" int tpb_layernorm_bwd(const void* dy, const void* x, const void* w, const float* mean,
                                 const float* rstd, void* dx, float* dw_part, float* db_part,
                                 float* dw_f32, void* dw_bf16, float* db_f32, void* db_bf16,
                                 int accumulate, int rows, int H, void* stream) {
  TPB_NVTX("tpb_layernorm_bwd");
  if (H % 8 || H > 256 * kMaxVec * 8) return -2;
  if (rows <= 0) return 0;
  int tpr = pick_tpr(H);
  int grid = tpb_rmsnorm_bwd_grid(rows, H);
  TPB_ROW_SWITCH(tpr, pick_vpt(H, tpr), (layernorm_bwd_kernel<TPR, VPT><<<grid, kRowThreads, 0, (cudaStream_t)stream>>>(
                          (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,
                          (const __nv_bfloat16*)w, mean, rstd, (__nv_bfloat16*)dx, dw_part, db_part,
                          rows, H)));
  launch_colsum({{dw_part, db_part}, {dw_f32, db_f32}, {(__nv_bfloat16*)dw_bf16, (__nv_bfloat16*)db_bf16}}, 2, grid, H,
                accumulate, (cudaStream_t)stream);
  return (int)cudaGetLastError();
}

// Column sums of a bf16 matrix: `part` holds tpb_bias_grad_chunks(rows, N) * N floats.
extern "C" int tpb_bias_grad_chunks(int rows, int N) { return bias_grad_chunks(rows, N); }
extern "C" int tpb_bias_grad(const void* x, float* part, void* out_bf16, int rows, int N, long long ld, void* stream) {
  TPB_NVTX("tpb_bias_grad");
  if (N % 8 || ld % 8 || (reinterpret_cast<uintptr_t>(x) & 15)) return -2;
  if (rows <= 0 || N <= 0) return 0;
  const int chunks = bias_grad_chunks(rows, N);
  bias_grad_kernel<<<dim3((N + 255) / 256, chunks), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, part, rows, N, ld, (rows + chunks - 1) / chunks);
  launch_colsum({{part, nullptr}, {nullptr, nullptr}, {(__nv_bfloat16*)out_bf16, nullptr}}, 1, chunks, N, 0,
                (cudaStream_t)stream);
  return (int)cudaGetLastError();
}

extern "C" int tpb_rope_out(const void* x, void* y, const float* cos_t, const float* sin_t,
                            const long long* pos, long long tokens, int heads, int D,
                            long long tok_stride, long long head_stride, long long y_tok_stride,
                            long long y_head_stride, int seq_len, int interleaved, int backward,
                            void* stream) {
  TPB_NVTX("tpb_rope_out");
  if (D % 16 || tok_stride % 8 || head_stride % 8 || y_tok_stride % 8 || y_head_stride % 8) return -2;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(cos_t) |
       reinterpret_cast<uintptr_t>(sin_t)) & 15)
    return -2;
  long long total = tokens * heads * (D / 16);
  if (total <= 0) return 0;
  int grid = (int)((total + 255) / 256);
  auto kern = t_chained ? (total < 0x7ff00000LL ? rope_kernel<unsigned, true> : rope_kernel<unsigned long long, true>)
                        : (total < 0x7ff00000LL ? rope_kernel<unsigned, false> : rope_kernel<unsigned long long, false>);
  return (int)launch_chained(kern, dim3(grid), 256, (cudaStream_t)stream,
      (const __nv_bfloat16*)x, (__nv_bfloat16*)y, cos_t, sin_t, pos, tokens, heads, D, tok_stride,
      head_stride, y_tok_stride, y_head_stride, seq_len, interleaved, backward ? -1.f : 1.f);
}
extern "C" int tpb_rope(void* x, const float* cos_t, const float* sin_t, const long long* pos,
                        long long tokens, int heads, int D, long long tok_stride,
                        long long head_stride, int seq_len, int interleaved, int backward,
                        void* stream) {
  TPB_NVTX("tpb_rope");
  return tpb_rope_out(x, x, cos_t, sin_t, pos, tokens, heads, D, tok_stride, head_stride, tok_stride,
                      head_stride, seq_len, interleaved, backward, stream);
}

// rows_dev (optional): device word with the number of rows actually in use (<= rows); rows beyond it
// are neither read nor written (expert buffers are sized for the worst case, filled to a
// data-dependent row).
extern "C" int tpb_swiglu_fwd_n(const void* gate, const void* up, void* out, long long rows, int I,
                                long long in_stride, const int* rows_dev, void* stream) {
  TPB_NVTX("tpb_swiglu_fwd_n");
  if (I % 8 || in_stride % 8) return -2;
  long long total = rows * (I / 8);
  if (total <= 0) return 0;
  auto kern = t_chained ? (total < 0x7ff00000LL ? swiglu_fwd_kernel<unsigned, true> : swiglu_fwd_kernel<unsigned long long, true>)
                        : (total < 0x7ff00000LL ? swiglu_fwd_kernel<unsigned, false> : swiglu_fwd_kernel<unsigned long long, false>);
  return (int)launch_chained(kern, dim3((unsigned)((total + 256 * kActVecs - 1) / (256 * kActVecs))), 256, (cudaStream_t)stream,
      (const __nv_bfloat16*)gate, (const __nv_bfloat16*)up, (__nv_bfloat16*)out, rows, I,
      in_stride, rows_dev);
}
extern "C" int tpb_swiglu_fwd(const void* gate, const void* up, void* out, long long rows, int I,
                              long long in_stride, void* stream) {
  TPB_NVTX("tpb_swiglu_fwd");
  return tpb_swiglu_fwd_n(gate, up, out, rows, I, in_stride, nullptr, stream);
}
extern "C" int tpb_swiglu_bwd_n(const void* dy, const void* gate, const void* up, void* dgate,
                                void* dup, long long rows, int I, long long in_stride,
                                long long out_stride, const int* rows_dev, void* stream) {
  TPB_NVTX("tpb_swiglu_bwd_n");
  if (I % 8 || in_stride % 8 || out_stride % 8) return -2;
  long long total = rows * (I / 8);
  if (total <= 0) return 0;
  auto kern = total < 0x7ff00000LL ? swiglu_bwd_kernel<unsigned> : swiglu_bwd_kernel<unsigned long long>;
  kern<<<(unsigned)((total + 256 * kActVecs - 1) / (256 * kActVecs)), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)gate, (const __nv_bfloat16*)up,
      (__nv_bfloat16*)dgate, (__nv_bfloat16*)dup, rows, I, in_stride, out_stride, rows_dev);
  return (int)cudaGetLastError();
}
extern "C" int tpb_swiglu_bwd(const void* dy, const void* gate, const void* up, void* dgate,
                              void* dup, long long rows, int I, long long in_stride,
                              long long out_stride, void* stream) {
  TPB_NVTX("tpb_swiglu_bwd");
  return tpb_swiglu_bwd_n(dy, gate, up, dgate, dup, rows, I, in_stride, out_stride, nullptr, stream);
}
extern "C" int tpb_gelu_fwd(const void* x, void* y, long long n, int approx, void* stream) {
  TPB_NVTX("tpb_gelu_fwd");
  if (n % 8) return -2;
  if (n <= 0) return 0;
  gelu_fwd_kernel<<<(unsigned)((n / 8 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, (__nv_bfloat16*)y, n / 8, approx);
  return (int)cudaGetLastError();
}
extern "C" int tpb_gelu_bwd(const void* dy, const void* x, void* dx, long long n, int approx,
                            void* stream) {
  TPB_NVTX("tpb_gelu_bwd");
  if (n % 8) return -2;
  if (n <= 0) return 0;
  gelu_bwd_kernel<<<(unsigned)((n / 8 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (__nv_bfloat16*)dx, n / 8, approx);
  return (int)cudaGetLastError();
}

// Threads of a block, by the rows that an SM has at once and the rounds of 256 threads that a row takes (8192 logits each). us with
// 256 / 512: 64 x 128256 18.2 / 12.3, 296 x 128256 21.2 / 17.8, 900 x 128256 48.5 / 46.5, 2400 x 128256 98 / 105; 148 x 50304
// 9.7 / 7.9, 296 x 50304 10.9 / 10.6, 592 x 50304 14.8 / 17.6; 148 x 32000 6.7 / 5.9, 200 x 32000 7.4 / 7.5; 64 x 8000 2.7 / 3.1.
static int ce_threads(long long rows, int V) {
  const long long sms = sm_count();
  return (rows <= sms && V > 2 * 8192) || (rows <= 2 * sms && V > 5 * 8192) ? 512 : 256;
}

extern "C" int tpb_cross_entropy(const void* logits, const long long* target, float* loss,
                                 float* lse, void* dlogits, long long rows, int V, long long stride,
                                 long long ignore_index, float gscale, void* stream) {
  TPB_NVTX("tpb_cross_entropy");
  if (stride % 8) return -2;
  if (rows <= 0) return 0;
  const int threads = ce_threads(rows, V);
  auto kern = threads == 512 ? cross_entropy_kernel<512> : cross_entropy_kernel<256>;
  kern<<<(unsigned)rows, threads, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)logits, target, loss, lse,
                                                             (__nv_bfloat16*)dlogits, V, stride, ignore_index, gscale);
  return (int)cudaGetLastError();
}

extern "C" int tpb_cross_entropy_bwd(const void* logits, const long long* target, const float* lse,
                                     void* dlogits, const float* g_scalar, const float* scale,
                                     const float* g_rows, long long rows, int V, long long stride,
                                     long long ignore_index, void* stream) {
  TPB_NVTX("tpb_cross_entropy_bwd");
  if (stride % 8) return -2;
  if (rows <= 0) return 0;
  int chunks = (V / 8 + 256 * 4 - 1) / (256 * 4);
  if (chunks < 1) chunks = 1;
  dim3 grid(chunks, (unsigned)rows);
  cross_entropy_bwd_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)logits, target, lse, (__nv_bfloat16*)dlogits, g_scalar, scale, g_rows,
      V, stride, ignore_index);
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------ allocation-free variant
#include "tpb_noalloc.h"

// Scratch for tpb_rmsnorm_bwd_noalloc: per-block partial sums of dw. Lives in every device
// that loads this library for the life of the process.
static __device__ __align__(256) float g_noalloc_rms_scratch[TPB_NOALLOC_RMSNORM_MAX_FLOATS];

namespace {
constexpr int kNoAllocMaxDevices = 64;
float* g_noalloc_scratch_ptr[kNoAllocMaxDevices] = {};
}  // namespace

extern "C" const char* tpb_noalloc_strerror(int code) {
  switch (code) {
    case 0: return "ok";
    case TPB_NOALLOC_TOO_LARGE:
      return "problem exceeds the built-in scratch (H <= 8192 and at most 296 blocks are supported)";
    case TPB_NOALLOC_BAD_ARGS: return "H must be a positive multiple of 8 and strides multiples of 8";
    case TPB_NOALLOC_NO_SYMBOL: return "could not obtain the device address of the built-in scratch";
    default: return code > 0 ? "CUDA error (see cudaGetErrorString)" : "unknown error";
  }
}

extern "C" int tpb_rmsnorm_bwd_noalloc(const void* dy, const void* x, const void* w,
                                       const float* rstd, const void* dres, void* dx, float* dw_f32,
                                       void* dw_bf16, int dw_accumulate, int rows, int H,
                                       long long x_stride, long long dy_stride, long long dx_stride,
                                       void* stream) {
  TPB_NVTX("tpb_rmsnorm_bwd_noalloc");
  if (H <= 0 || H % 8 || x_stride % 8 || dy_stride % 8 || dx_stride % 8) return TPB_NOALLOC_BAD_ARGS;
  if (H > TPB_NOALLOC_RMSNORM_MAX_H) return TPB_NOALLOC_TOO_LARGE;
  if (rows <= 0) return 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kNoAllocMaxDevices) return TPB_NOALLOC_NO_SYMBOL;
  // First call on this device: the array's name is only a host-side handle, the kernel needs
  // the address the symbol has on the current device.
  float* scratch = g_noalloc_scratch_ptr[dev];
  if (!scratch) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_rms_scratch);
    if (e != cudaSuccess || !p) return TPB_NOALLOC_NO_SYMBOL;
    scratch = static_cast<float*>(p);
    g_noalloc_scratch_ptr[dev] = scratch;
  }
  const int tpr = pick_tpr(H);
  int grid = tpb_rmsnorm_bwd_grid(rows, H);
  if (grid > TPB_NOALLOC_RMSNORM_MAX_BLOCKS) grid = TPB_NOALLOC_RMSNORM_MAX_BLOCKS;
  if ((long long)grid * H > (long long)TPB_NOALLOC_RMSNORM_MAX_FLOATS) return TPB_NOALLOC_TOO_LARGE;
  TPB_ROW_SWITCH(tpr, pick_vpt(H, tpr), (rmsnorm_bwd_kernel<TPR, VPT><<<grid, kRowThreads, 0, (cudaStream_t)stream>>>(
                          (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,
                          (const __nv_bfloat16*)w, rstd, (const __nv_bfloat16*)dres,
                          (__nv_bfloat16*)dx, scratch, rows, H, x_stride, dy_stride, dx_stride)));
  launch_colsum({{scratch, nullptr}, {dw_f32, nullptr}, {(__nv_bfloat16*)dw_bf16, nullptr}}, 1, grid, H, dw_accumulate,
                (cudaStream_t)stream);
  return (int)cudaGetLastError();
}
