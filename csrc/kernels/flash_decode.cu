// Attention of a few query rows over a long key/value sequence (decoding, speculative verification) for sm_100a.
//
// The work is reading K and V once: 2 * Tk * D * Hkv values per sequence against 4 * R flops a value, R = query rows
// that share a KV head (Tq * Hq / Hkv). The 128-row tiles of flash_fwd_kernel read every KV head once per QUERY head
// and leave all but B * Hq CTAs idle: 437 us at B = 8, Tk = 16381, 32/8 heads of 128 (0.54 GB). Here
//   * all query rows of a KV head form the 16-row operand of one warp MMA (m16n8k16), so K and V are read once per
//     16 rows; with at most 16 rows there is no tile that would amortise TMEM and a shared-memory operand pipeline;
//   * a warp works on steps of 16 keys and copies its own later steps with cp.async into a ring of its own (no barrier
//     between warps): K of a step is replaced once its scores are there, V once its product is. The chain of a step
//     (scores, maximum, exponentials, second product) takes some 1 000 cycles in which a warp's registers cannot also
//     be loading; with the fragments of the next step in registers (204 of them, eight warps per SM) warps spent 60 % of
//     the time in that chain and 4.8 TB/s came in. The ring leaves room for twelve (D = 128) or sixteen warps;
//   * the keys are split over CTAs; partial sums stay fp32. Up to eight splits of a row tile are one cluster that merges
//     them through distributed shared memory, in rank order; more go through memory and a second kernel.
// The same case takes 82 us (6.6 TB/s; 112 before the ring); 32 x 8000 keys 151 (6.9 TB/s; 215), 16 x 1006 keys 15.7
// (20), D = 64 with 8 x 16381 keys 44 (52).
// Scores, running maximum, sums and output accumulate in fp32; probabilities are rounded to bf16 for the second
// product, as in flash_fwd_kernel. With at most eight rows to a KV head the other eight rows of the operand carry what that
// rounding cuts off (FINE).
#include "sm100.cuh"
#include "tpb_api.h"

namespace tpb {

constexpr int kDecWarps = 4;
constexpr int kDecRows = 16;   // query rows per CTA
constexpr int kDecKeys = 16;   // keys per warp and step
constexpr int kDecCluster = 8; // splits that one cluster can hold (the portable size)

struct DecodeParams {
  const __nv_bfloat16 *q, *k, *v;
  __nv_bfloat16* o;
  float* lse;
  float* part_o;    // [n_splits][B * Hkv * R][D]; null when n_splits == 1 or the splits of a row tile are one cluster
  float* part_lse;  // [n_splits][B * Hkv * R], log2 domain
  int B, Tq, Tk, Hq, Hkv, group, R, row_tiles, causal, window, lse_stride, n_splits, keys_per_split;
  float scale_log2e;
  long long q_tok, q_head, q_batch, k_tok, k_head, k_batch, v_tok, v_head, v_batch, o_tok, o_head, o_batch;
};

__device__ __forceinline__ float dec_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t dec_pack(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
// 16 bytes to shared memory, zeros where `in` is false.
__device__ __forceinline__ void dec_cp(uint32_t dst, const __nv_bfloat16* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void dec_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void dec_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
template <bool TRANS>
__device__ __forceinline__ void dec_ldm(uint32_t (&r)[4], uint32_t a) {
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

constexpr int dec_stages(int d) { return d == 128 ? 2 : 3; }   // steps that a warp's ring holds
constexpr int dec_ctas(int d) { return d == 128 ? 3 : 4; }     // CTAs that fit an SM
constexpr int dec_smem(int d) {
  const int ring = kDecWarps * dec_stages(d) * 2 * kDecKeys * d * 2, rows = kDecWarps * kDecRows * d * 4;
  return ring > rows ? ring : rows;
}

// FINE: at most eight rows. The operand's rows 8..15 are then nobody's; in the second product they hold P - bf16(P) of rows 0..7,
// and their sums are added in the end. The largest probability of a warp's keys is exactly one and has no rounding error, so
// that the error grew with longer runs of keys to a warp: of the norm, against 64 bits, 2.21e-3 at 8 x 16381 keys, 32/8 heads of
// 128 (2.16e-3 in twice as many parts), 1.66e-3 so, which is the rounding of the result. It saves the exponentials of the rows that
// are not there: the same case 82.3 -> 81.6 us, 16 x 1006 keys 15.9 -> 15.3, one sequence of 9000 18.1 -> 17.6.
template <int D, bool FINE>
__global__ void __launch_bounds__(kDecWarps * 32, dec_ctas(D))
flash_decode_kernel(const DecodeParams p) {
  constexpr int S = dec_stages(D);
  constexpr int NR = FINE ? 1 : 2;          // rows of a lane
  constexpr int kTile = kDecKeys * D * 2;   // bytes of a step's K (or V) of a warp
  extern __shared__ __align__(128) uint8_t dec_sm[];   // the warps' rings, later their partial rows
  __shared__ float sm_m[kDecWarps][kDecRows], sm_l[kDecWarps][kDecRows], sm_lse[kDecRows];
  float (&sm_o)[kDecWarps][kDecRows][D] = *reinterpret_cast<float (*)[kDecWarps][kDecRows][D]>(dec_sm);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gq = lane >> 2, t = lane & 3;
  const int split = blockIdx.x, hk = blockIdx.y / p.row_tiles, rt = blockIdx.y % p.row_tiles, b = blockIdx.z;

  chain_next();
  chain_wait();
  int k_begin = split * p.keys_per_split;
  const int k_end = min(p.Tk, k_begin + p.keys_per_split);
  if (p.window > 0) {
    // the CTA's first row has the lowest bound
    const int first = (rt * kDecRows) / p.group + p.Tk - p.Tq - p.window + 1;
    if (first > k_begin) k_begin += (first - k_begin) / kDecKeys * kDecKeys;
  }

  // A lane copies one 16-byte piece of every LR-th row. Pieces are swizzled by their row, so that the eight rows of a
  // matrix lie in different banks.
  constexpr int LR = 256 / D;   // rows per copy of a warp
  const int piece = lane % (D / 8), row0 = lane / (D / 8);
  const uint32_t ring = smem_u32(dec_sm) + warp * (S * 2 * kTile);
  const __nv_bfloat16* kp = p.k + b * p.k_batch + (long long)hk * p.k_head + piece * 8;
  const __nv_bfloat16* vp = p.v + b * p.v_batch + (long long)hk * p.v_head + piece * 8;
  // keys past the end are zero-filled: their probability is zero, but zero times whatever lies there need not be
  auto load = [&](const __nv_bfloat16* src, long long tok, int base, uint32_t dst) {
    if (base < k_end) {
#pragma unroll
      for (int i = 0; i < kDecKeys / LR; ++i) {
        const int r = row0 + i * LR, key = base + r;
        dec_cp(dst + r * (D * 2) + ((piece ^ (r & 7)) << 4), src + (key < k_end ? key : 0) * tok, key < k_end);
      }
    }
    dec_commit();
  };
  constexpr int kStep = kDecWarps * kDecKeys;
  const int base0 = k_begin + warp * kDecKeys;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    load(kp, p.k_tok, base0 + s * kStep, ring + s * 2 * kTile);
    load(vp, p.v_tok, base0 + s * kStep, ring + s * 2 * kTile + kTile);
  }

  // this lane's two rows: r0 (fragment row gq) and r0 + 8
  const int r0 = rt * kDecRows + gq;
  int lim[2], low[2], all_lim = p.Tk - 1, all_low = 0;   // of the lane's rows that exist
  uint32_t qf[D / 16][4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = r0 + 8 * i;
    const int tq = r / p.group, h = hk * p.group + r % p.group;
    const bool in = r < p.R;
    lim[i] = in ? (p.causal ? min(p.Tk - 1, tq + p.Tk - p.Tq) : p.Tk - 1) : -1;
    low[i] = p.window > 0 ? tq + p.Tk - p.Tq - p.window + 1 : 0;
    if (in) { all_lim = min(all_lim, lim[i]); all_low = max(all_low, low[i]); }
    const __nv_bfloat16* qr = p.q + b * p.q_batch + (long long)tq * p.q_tok + (long long)h * p.q_head;
#pragma unroll
    for (int c = 0; c < D / 16; ++c)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        qf[c][i + 2 * e] = in ? *reinterpret_cast<const uint32_t*>(qr + c * 16 + e * 8 + 2 * t) : 0u;
  }
  // steps that lie inside every row's bounds take the path without masks (rows past the last one are not stored)
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    all_lim = min(all_lim, __shfl_xor_sync(0xffffffffu, all_lim, o));
    all_low = max(all_low, __shfl_xor_sync(0xffffffffu, all_low, o));
  }
  all_lim = min(all_lim, k_end - 1);

  float acc[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[n][j] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};

  // rows and piece halves of this lane's matrix addresses: K matrices (8 keys x 8 of d) side by side along d, V ones
  // (transposed) two key halves by two along d
  const int krow = lane & 7, kpc = lane >> 3;
  const int vrow = lane & 15, vpc = lane >> 4;
  int slot = 0;
  for (int base = base0; base < k_end; base += kStep) {
    const uint32_t sk = ring + slot * 2 * kTile, sv = sk + kTile;
    dec_wait<2 * S - 1>();
    __syncwarp();
    float s[2][4], s2[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
      for (int j = 0; j < 4; ++j) s[u][j] = s2[u][j] = 0.f;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t kf[4];
        dec_ldm<false>(kf, sk + (u * 8 + krow) * (D * 2) + (((c * 4 + kpc) ^ krow) << 4));
        mma_bf16_16816(s[u], qf[2 * c][0], qf[2 * c][1], qf[2 * c][2], qf[2 * c][3], kf[0], kf[1]);
        mma_bf16_16816(s2[u], qf[2 * c + 1][0], qf[2 * c + 1][1], qf[2 * c + 1][2], qf[2 * c + 1][3], kf[2], kf[3]);
      }
    }
    __syncwarp();   // every lane has read K
    load(kp, p.k_tok, base + S * kStep, sk);
    // s[u][2 i + j]: row i, key base + 8 u + 2 t + j
    float mx[2] = {-INFINITY, -INFINITY};
    const bool inside = base >= all_low && base + kDecKeys - 1 <= all_lim;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int i = 0; i < NR; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float& x = s[u][2 * i + j];
          x = (x + s2[u][2 * i + j]) * p.scale_log2e;
        }
    if (!inside) {
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int key = base + u * 8 + 2 * t + j;
            float& x = s[u][2 * i + j];
            x = (key <= lim[i] && key >= low[i] && key < k_end) ? x : -INFINITY;
          }
    }
    float alpha[2], mu[2];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      mx[i] = fmaxf(fmaxf(s[0][2 * i], s[0][2 * i + 1]), fmaxf(s[1][2 * i], s[1][2 * i + 1]));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
      const float mn = fmaxf(m[i], mx[i]);
      mu[i] = mn == -INFINITY ? 0.f : mn;   // no key yet: every exponent below is -inf
      alpha[i] = dec_exp2(m[i] - mu[i]);
      m[i] = mn;
      l[i] *= alpha[i];
    }
    if (FINE) alpha[1] = alpha[0];
    if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
      for (int n = 0; n < D / 8; ++n) {
        acc[n][0] *= alpha[0]; acc[n][1] *= alpha[0];
        acc[n][2] *= alpha[1]; acc[n][3] *= alpha[1];
      }
    }
    uint32_t pa[4];   // A fragment of the second product: (row, key half)
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const float e0 = dec_exp2(s[u][2 * i] - mu[i]), e1 = dec_exp2(s[u][2 * i + 1] - mu[i]);
        l[i] += e0 + e1;
        const uint32_t w = dec_pack(e0, e1);
        pa[2 * u + i] = w;
        if (FINE) pa[2 * u + 1] = dec_pack(e0 - __uint_as_float(w << 16), e1 - __uint_as_float(w & 0xffff0000u));
      }
    dec_wait<2 * S - 1>();
    __syncwarp();
#pragma unroll
    for (int c = 0; c < D / 16; ++c) {
      uint32_t vf[4];
      dec_ldm<true>(vf, sv + vrow * (D * 2) + (((c * 2 + vpc) ^ (vrow & 7)) << 4));
      mma_bf16_16816(acc[2 * c], pa[0], pa[1], pa[2], pa[3], vf[0], vf[1]);
      mma_bf16_16816(acc[2 * c + 1], pa[0], pa[1], pa[2], pa[3], vf[2], vf[3]);
    }
    __syncwarp();   // every lane has read V
    load(vp, p.v_tok, base + S * kStep, sv);
    slot = slot + 1 == S ? 0 : slot + 1;
  }
  dec_wait<0>();
  __syncthreads();   // the rings become the partial rows

  // ---- the four warps' partial rows
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    if (t == 0) { sm_m[warp][gq + 8 * i] = m[i]; sm_l[warp][gq + 8 * i] = l[i]; }
#pragma unroll
    for (int n = 0; n < D / 8; ++n) {
      float2 v = make_float2(acc[n][2 * i], acc[n][2 * i + 1]);
      if (FINE) {   // an infinite V gives infinities of either sign in the second part
        if (fabsf(v.x) < INFINITY) v.x += acc[n][2];
        if (fabsf(v.y) < INFINITY) v.y += acc[n][3];
      }
      *reinterpret_cast<float2*>(&sm_o[warp][gq + 8 * i][n * 8 + 2 * t]) = v;
    }
  }
  __syncthreads();
  constexpr int VEC = D / 4;   // float4 per row
  auto store = [&](int r, int d, const float4& o, float lse2) {
    const int tq = r / p.group, h = hk * p.group + r % p.group;
    uint2 w;
    w.x = dec_pack(o.x, o.y);
    w.y = dec_pack(o.z, o.w);
    *reinterpret_cast<uint2*>(p.o + b * p.o_batch + (long long)tq * p.o_tok + (long long)h * p.o_head + d) = w;
    if (d == 0) p.lse[((long long)b * p.Hq + h) * p.lse_stride + tq] = lse2 * 0.6931471805599453f;
  };
  for (int x = threadIdx.x; x < kDecRows * VEC; x += kDecWarps * 32) {
    const int rr = x / VEC, d = (x % VEC) * 4;
    const int r = rt * kDecRows + rr;
    if (r >= p.R) break;
    // Whether this split holds a key of the row is asked of the bounds: a maximum of -inf may also mean scores that are
    // all NaN, which have to reach the output, and V at keys that are masked for the row may hold anything.
    const int at_q = r / p.group + p.Tk - p.Tq;
    const int last = min(k_end - 1, p.causal ? at_q : p.Tk - 1);
    const int first = max(split * p.keys_per_split, p.window > 0 ? at_q - p.window + 1 : 0);
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) M = fmaxf(M, sm_m[w][rr]);
    const float mu = M == -INFINITY ? 0.f : M;
    float L = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (first <= last) {
#pragma unroll
      for (int w = 0; w < kDecWarps; ++w) {
        const float f = dec_exp2(sm_m[w][rr] - mu);
        L += f * sm_l[w][rr];
        const float4 a = *reinterpret_cast<const float4*>(&sm_o[w][rr][d]);
        o.x += f * a.x; o.y += f * a.y; o.z += f * a.z; o.w += f * a.w;
      }
    }
    const float inv = L > 0.f ? 1.f / L : 0.f;
    o.x *= inv; o.y *= inv; o.z *= inv; o.w *= inv;
    const float lse2 = L > 0.f ? M + log2f(L) : (L == 0.f || p.n_splits == 1 ? -INFINITY : L);   // NaN stays NaN in a partial row
    if (p.part_o) {
      const long long row = (long long)(b * p.Hkv + hk) * p.R + r;
      const long long at = (long long)split * p.B * p.Hkv * p.R + row;
      *reinterpret_cast<float4*>(p.part_o + at * D + d) = o;
      if (d == 0) p.part_lse[at] = lse2;
    } else if (p.n_splits > 1) {
      *reinterpret_cast<float4*>(&sm_o[0][rr][d]) = o;   // only this thread has read that place
      if (d == 0) sm_lse[rr] = lse2;
    } else {
      store(r, d, o, lse2);
    }
  }
  if (p.n_splits > 1 && !p.part_o) {
    // the splits are the CTAs of a cluster: each merges a slice of the rows, read in rank order
    __syncthreads();
    cluster_sync_all();
    const int items = min(kDecRows, p.R - rt * kDecRows) * VEC;
    const uint32_t o_sa = smem_u32(&sm_o[0][0][0]), l_sa = smem_u32(sm_lse);
    for (int x = split * kDecWarps * 32 + threadIdx.x; x < items; x += p.n_splits * kDecWarps * 32) {
      const int rr = x / VEC, d = (x % VEC) * 4;
      float w[kDecCluster];
      float4 v[kDecCluster];
#pragma unroll
      for (int s = 0; s < kDecCluster; ++s) {
        w[s] = s < p.n_splits ? ld_cluster_f32(l_sa + rr * 4, s) : -INFINITY;
        v[s] = s < p.n_splits ? ld_cluster_f4(o_sa + (rr * D + d) * 4, s) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      float M = -INFINITY;
#pragma unroll
      for (int s = 0; s < kDecCluster; ++s) M = fmaxf(M, w[s]);
      const float mu = M == -INFINITY ? 0.f : M;
      float den = 0.f;
      float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int s = 0; s < kDecCluster; ++s) {
        const float f = dec_exp2(w[s] - mu);
        den += f;
        o.x += f * v[s].x; o.y += f * v[s].y; o.z += f * v[s].z; o.w += f * v[s].w;
      }
      const float inv = den > 0.f ? 1.f / den : 0.f;
      o.x *= inv; o.y *= inv; o.z *= inv; o.w *= inv;
      store(rt * kDecRows + rr, d, o, den > 0.f ? M + log2f(den) : -INFINITY);
    }
    __syncthreads();
    cluster_sync_all();   // nobody leaves while a peer may read its rows
  }
}

// o = sum_s w_s o_s / sum_s w_s with w_s = 2^(lse_s - max); one warp per row, the splits' rows requested eight at a time.
template <int D>
__global__ void __launch_bounds__(128)
flash_decode_merge_kernel(const DecodeParams p) {
  constexpr int E = D / 32;   // floats per lane
  const int lane = threadIdx.x & 31;
  const long long rows = (long long)p.B * p.Hkv * p.R;
  const long long row = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  float M = -INFINITY;
  for (int s = lane; s < p.n_splits; s += 32) M = fmaxf(M, p.part_lse[s * rows + row]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  const float mu = M == -INFINITY ? 0.f : M;
  float acc[E], den = 0.f;
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.f;
  for (int s0 = 0; s0 < p.n_splits; s0 += 8) {
    float v[8][E], w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const bool in = s0 + j < p.n_splits;
      const long long at = (s0 + j) * rows + row;
      w[j] = in ? p.part_lse[at] : -INFINITY;
#pragma unroll
      for (int e = 0; e < E; ++e) v[j][e] = in ? p.part_o[at * D + lane + 32 * e] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float f = dec_exp2(w[j] - mu);
      den += f;
#pragma unroll
      for (int e = 0; e < E; ++e) acc[e] += f * v[j][e];
    }
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
  const int r = (int)(row % p.R);
  const int hk = (int)(row / p.R % p.Hkv), b = (int)(row / p.R / p.Hkv);
  const int tq = r / p.group, h = hk * p.group + r % p.group;
  __nv_bfloat16* o = p.o + b * p.o_batch + (long long)tq * p.o_tok + (long long)h * p.o_head;
#pragma unroll
  for (int e = 0; e < E; ++e) o[lane + 32 * e] = __float2bfloat16(acc[e] * inv);
  if (lane == 0)
    p.lse[((long long)b * p.Hq + h) * p.lse_stride + tq] = den > 0.f ? (M + log2f(den)) * 0.6931471805599453f : -INFINITY;
}

typedef void (*DecodeKernel)(DecodeParams);
static DecodeKernel decode_kernel(int D, bool fine) {
  return D == 64 ? (fine ? flash_decode_kernel<64, true> : flash_decode_kernel<64, false>)
                 : (fine ? flash_decode_kernel<128, true> : flash_decode_kernel<128, false>);
}

// More shared memory than a launch gets unasked.
static cudaError_t decode_configure(int dev, int D, bool fine) {
  static PerDevice done[2][2];
  return allow_smem(done[D == 64 ? 0 : 1][fine], dev, decode_kernel(D, fine), dec_smem(D));
}

// Clusters of n CTAs that fit the device at once, asked of the runtime once per size and device: the SMs of a GPC are not a
// multiple of every n (48 clusters of 8 CTAs of D = 128 fit, 142 of 3, although 444 CTAs do). Both forms take the same room.
static int decode_resident(int dev, int D, int n) {
  static PerDevice resident[2][kDecCluster + 1];
  return resident[D == 64 ? 0 : 1][n].get(dev, [&] {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = n;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(n, 4 * sm_count());
    cfg.blockDim = dim3(kDecWarps * 32);
    cfg.dynamicSmemBytes = dec_smem(D);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int fit = 0;
    decode_configure(dev, D, false);
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&fit, decode_kernel(D, false), &cfg);
    return e == cudaSuccess && fit > 0 ? fit : -1;
  });
}

// Splits of the keys and who merges them, by the time in ns that the launch takes. What resident CTAs take is what memory
// takes (7 TB/s; the row tiles of a head share its reads) or the keys of one times kKeyNs, which grows with the CTAs per
// SM: one alone reads 49 (D = 128) or 37 (64) GB/s and keeps an SM's share of the memory busy by itself. Clusters are not
// spread evenly: at 0.87 of an SM each, some SMs have two CTAs. A launch costs 4 us, each further round 1.8 us and a tail of
// 4 ns a key; a cluster's merge 1 us; a second kernel and scratch 3 us + 60 ns a split. The 5 us that they cost on the host are
// not counted: a launch that is waited for the host takes those whatever it does, and up to some 4000 keys the clusters are ahead
// anyway. (Counted, one sequence of 9000 keys and one KV head took 17.8 us for 11.6, two of 30000 and eight 56.8 for 44.7.)
// Measured, D x B x Hkv x Tk, splits: us (m: by two kernels): 128 x 8 x 8 x 16381, 1: 177, 2: 94, 3: 87, 4: 82, 5: 92, 8: 105,
// m9: 100, m12: 87; 128 x 32 x 8 x 8000, 1: 151, 2: 192, 3: 162, 8: 170; 128 x 3 x 16 x 5000, 1: 57, 3: 30, 5: 24, 8: 25;
// 128 x 1 x 8 x 3000, 8: 9.5, m16: 10.0; x 5500, 8: 13.0, m16: 12.0; x 10000, 8: 19.0, m16: 14.7; x 30000, 8: 44.8, m32: 27.3;
// 128 x 1 x 1 x 3000, 8: 8.7, m16: 8.2; x 7500, 8: 14.9, m40: 10.2; 64 x 1 x 8 x 5500, 8: 9.6, m16: 9.8; x 14000, 8: 16.6,
// m32: 12.9; 64 x 8 x 8 x 16381, 1: 115, 2: 62, 4: 44, 7: 51, 8: 47; 64 x 32 x 8 x 8000, 1: 80, 2: 89, 3: 97.
struct DecodePlan {
  int splits;
  bool memory;   // merged by the second kernel
};
static DecodePlan decode_plan(int dev, int B, int Hkv, int row_tiles, int Tk, int D, bool memory) {
  static const double kKeyNs[2][4] = {{7.0, 9.1, 13.0, 21.0}, {10.5, 15.0, 26.0, 26.0}};
  const int fit = dec_ctas(D), wide = D == 64 ? 0 : 1;
  const long long tiles = (long long)B * Hkv * row_tiles, sms = sm_count();
  const double read_ns = 4.0 * D / 7000.0 / row_tiles;   // of a key of a CTA
  DecodePlan best = {1, false};
  double best_cost = -1;
  // units are what is scheduled, clusters of `ctas` or single CTAs
  auto consider = [&](int n, bool mem, long long units, long long slots, int ctas) {
    const double keys = (double)((Tk + n - 1) / n);
    auto round = [&](double running) {   // CTAs
      const double per_sm = running * (ctas > 1 ? 1.15 : 1.0) / (double)sms;
      const int at = per_sm <= 1 ? 0 : per_sm <= 2 ? 1 : per_sm <= 3 || fit == 3 ? 2 : 3;
      const double read = running * read_ns, chain = kKeyNs[wide][at];
      return keys * (read > chain ? read : chain);
    };
    const long long full = units / slots, rest = units % slots, rounds = full + (rest > 0);
    double cost = full * round((double)(slots * ctas)) + (rest ? round((double)(rest * ctas)) : 0) + 4000 + 1800.0 * (rounds - 1);
    if (rounds > 1) cost += 4 * keys;
    cost += mem ? 3000 + 60 * n : (n > 1 ? 1000 : 0);
    if (best_cost < 0 || cost < best_cost) { best = {n, mem}; best_cost = cost; }
  };
  consider(1, false, tiles, fit * sms, 1);
  for (int n = 2; n <= kDecCluster && Tk / n >= 64; ++n) {
    const int clusters = decode_resident(dev, D, n);
    if (clusters > 0) consider(n, false, tiles, clusters, n);
  }
  for (int n = 2; memory && n <= 64 && Tk / n >= 64; ++n) consider(n, true, tiles * n, fit * sms, 1);
  return best;
}

}  // namespace tpb

using namespace tpb;

// 0 where tpb_flash_decode needs no memory for its splits (it then takes n_splits 0 and picks them itself, as it may
// anyway up to 2048 keys); else their number n: part_o has to hold n * B * Hq * Tq * D floats, part_lse n * B * Hq * Tq.
extern "C" int tpb_flash_decode_splits(int B, int Tq, int Tk, int Hq, int Hkv, int D) {
  if (B <= 0 || Tq <= 0 || Tk <= 0 || Hkv <= 0) return 0;
  const DecodePlan plan = decode_plan(current_device(), B, Hkv, (Tq * (Hq / Hkv) + kDecRows - 1) / kDecRows, Tk, D, true);
  return plan.memory ? plan.splits : 0;
}

// Arguments as in tpb_flash_fwd_ex; lse [B, Hq, lse_stride]. n_splits 0: the best number that needs no part_o. With
// part_o the splits are merged by a second kernel, without (eight at most) by clusters.
extern "C" int tpb_flash_decode(const void* q, const void* k, const void* v, void* o, float* lse, float* part_o,
                                float* part_lse, int B, int Tq, int Tk, int Hq, int Hkv, int D, long long q_tok,
                                long long q_head, long long q_batch, long long k_tok, long long k_head,
                                long long k_batch, long long v_tok, long long v_head, long long v_batch,
                                long long o_tok, long long o_head, long long o_batch, int lse_stride, int causal,
                                float scale, int window, int n_splits, void* stream) {
  TPB_NVTX("tpb_flash_decode");
  if (B <= 0 || Tq <= 0 || Hq <= 0) return 0;
  if ((D != 64 && D != 128) || Hkv <= 0 || Hq % Hkv || Tk <= 0 || n_splits < 0 || B > 65535) return -2;
  if ((q_tok | q_head | q_batch | k_tok | k_head | k_batch | v_tok | v_head | v_batch | o_tok | o_head | o_batch) % 8)
    return -2;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(o)) & 15)
    return -2;
  if ((n_splits > kDecCluster && !part_o) || (part_o && !part_lse)) return -2;
  const int dev = current_device();
  if (n_splits == 0) {
    part_o = part_lse = nullptr;
    n_splits = decode_plan(dev, B, Hkv, (Tq * (Hq / Hkv) + kDecRows - 1) / kDecRows, Tk, D, false).splits;
  }
  DecodeParams p;
  p.q = (const __nv_bfloat16*)q; p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v;
  p.o = (__nv_bfloat16*)o; p.lse = lse; p.part_o = n_splits > 1 ? part_o : nullptr; p.part_lse = part_lse;
  p.B = B; p.Tq = Tq; p.Tk = Tk; p.Hq = Hq; p.Hkv = Hkv; p.group = Hq / Hkv; p.R = Tq * p.group;
  p.row_tiles = (p.R + kDecRows - 1) / kDecRows;
  p.causal = causal; p.window = window > 0 ? window : 0; p.lse_stride = lse_stride; p.n_splits = n_splits;
  const int per = (Tk + n_splits - 1) / n_splits;
  p.keys_per_split = (per + kDecKeys - 1) / kDecKeys * kDecKeys;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.q_tok = q_tok; p.q_head = q_head; p.q_batch = q_batch; p.k_tok = k_tok; p.k_head = k_head; p.k_batch = k_batch;
  p.v_tok = v_tok; p.v_head = v_head; p.v_batch = v_batch; p.o_tok = o_tok; p.o_head = o_head; p.o_batch = o_batch;
  if ((long long)Hkv * p.row_tiles > 65535) return -2;
  const dim3 grid(n_splits, Hkv * p.row_tiles, B);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kDecWarps * 32);
  cfg.dynamicSmemBytes = dec_smem(D);
  cfg.stream = (cudaStream_t)stream;
  cfg.attrs = attr;
  if (t_chained) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (n_splits > 1 && !p.part_o) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = n_splits;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  const bool fine = p.R <= 8;
  cudaError_t e = decode_configure(dev, D, fine);
  if (e != cudaSuccess) return (int)e;
  e = cudaLaunchKernelEx(&cfg, decode_kernel(D, fine), p);
  if (e != cudaSuccess) return (int)e;
  if (p.part_o) {
    const long long rows = (long long)B * Hkv * p.R;
    const unsigned blocks = (unsigned)((rows + 3) / 4);
    if (D == 128) flash_decode_merge_kernel<128><<<blocks, 128, 0, (cudaStream_t)stream>>>(p);
    else flash_decode_merge_kernel<64><<<blocks, 128, 0, (cudaStream_t)stream>>>(p);
  }
  return (int)cudaGetLastError();
}
