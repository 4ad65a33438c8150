// Flash attention backward for sm_100a, the form with one tile of S and dP in TMEM: head dimension 128 with long streams,
// and head dimension 64, but for a dKV pass of few CTAs (flash_bwd.cu has the choice and the other form).
//
// Two passes as described there. Per streamed tile: S = X0 Y0^T and dP = X1 Y1^T into TMEM; eight warps turn S into
// P = exp2(..) and then dP into dS = P (dP - delta) * scale, each written as bf16 over the columns it came from, from
// where the accumulating MMAs take it as their A operand. The products of two tiles interleave on the tensor pipe,
//     dV(i)  S(i+1)  dK(i)  dP(i+1)      (dQ pass: S(i+1)  dQ(i)  dP(i+1)),
// and the warps compute dS(i) under dV(i) and S(i+1), and P(i+1) under dK(i) and dP(i+1). The dQ pass has no P product: S(i+1)
// is issued once S(i) is in registers and runs under P(i). The warps take 32 columns at a time and load the next ones under
// the math of the ones before, and read the statistics for P while they wait for S. With that and the passes overlapping
// (flash_bwd.cuh), in turn on one GPU, 32/8 heads, both passes: T = 8190 1910 -> 1706 us (at the power cap), T = 4096 514 -> 459;
// D = 64, T = 8190 1303 -> 1157, 16 x 1024 tokens of 12 heads 216 -> 188.
//
// D = 128: TMEM (S, dP and two accumulators of 128 columns) has no room for two tiles unless they have 64 rows; with 128
// rows there are half as many barriers and round trips (a tenth of the time at T = 4096 and 8190 when it was taken); the
// chip then runs at its power cap (1.7 GHz), at about 0.6 of what the MMAs alone would take.
// D = 64: 64-row tiles fit half of TMEM and of shared memory, so that two CTAs share an SM: starting and finishing a CTA
// takes about as long as the eight iterations it has at T = 1024, and one CTA's start, end and waits lie under the
// other's work (a ninth of the time at 16 x 1024 tokens of 12 heads when it was taken).
#include "flash_bwd.cuh"
#include "tpb_api.h"

namespace tpb {

constexpr int ctas_per_sm(int ks) { return ks == 64 ? 2 : 1; }

template <int D, int KS>
struct WideSmem {
  static constexpr int kStream = KS;
  static constexpr int kChunks = D / 64;
  static constexpr int kStatBytes = kStat * D * 2;      // one stationary tile
  static constexpr int kStreamBytes = kStream * D * 2;  // one streamed tile
  // One ring for the streamed tiles, Y0(0) Y1(0) Y0(1) Y1(1) ...: Y1 is released half an iteration before Y0.
  static constexpr int kRing = D == 128 ? 5 : 8;
  // Statistics of the streamed queries ride along with Y1. Y1(i + kStatSlots) is loaded into the ring only after the
  // slot of Y0(i) was released, which is after the P / dS warps were done with iteration i.
  static constexpr int kStatSlots = kRing / 2;
  static constexpr int kX0 = 0;
  static constexpr int kX1 = kX0 + kStatBytes;
  static constexpr int kY = kX1 + kStatBytes;
  static constexpr int kStats = kY + kRing * kStreamBytes;  // per slot: -lse * log2e [128] then -delta * scale [128]
  static constexpr int kBar = kStats + kStatSlots * 2 * kStream * 4;
  static constexpr int kUsed = kBar + (2 * kRing + 7) * 8 + 8;
  // Room to align the base to the swizzle atom (1024 bytes); what is left of it for D = 128 covers a base that is a
  // multiple of 256, and the kernel refuses any other.
  static constexpr int kTotal = kUsed + 1024 <= 227 * 1024 ? kUsed + 1024 : 227 * 1024;
  static_assert(kTotal - kUsed >= 768, "attention backward exceeds the shared memory of one CTA");
  static_assert(2 * kStatSlots + 1 >= kRing, "statistics would be overwritten while in use");
};

// P = exp2(S * scale_log2e - lse * log2e) of 32 columns of one row, in place (fp32). Straight-line code: the masked
// variant selects, it never branches.
//   DKV: per-column statistics of the streamed queries come from shared memory;
//   dQ : the row's own statistics are in registers.
// Both come negated and scaled from the pass that computes delta: scaling them here cost two of the ~eight instructions
// per element of the dK/dV pass.
template <bool DKV, bool MASKED>
__device__ __forceinline__ void p_math(uint32_t* sr, const float4* stats, float nlse2_row, int y0i, int y_lo, int y_hi,
                                       float scale_log2e) {
  const float2 sc2 = make_float2(scale_log2e, scale_log2e);
#pragma unroll
  for (int c = 0; c < 32; c += 4) {
    float4 l = make_float4(nlse2_row, nlse2_row, nlse2_row, nlse2_row);
    if (DKV) l = stats[c / 4];
    const float2 lo = __ffma2_rn(make_float2(__uint_as_float(sr[c]), __uint_as_float(sr[c + 1])), sc2, make_float2(l.x, l.y));
    const float2 hi = __ffma2_rn(make_float2(__uint_as_float(sr[c + 2]), __uint_as_float(sr[c + 3])), sc2, make_float2(l.z, l.w));
    float e[4] = {bwd_exp2(lo.x), bwd_exp2(lo.y), bwd_exp2(hi.x), bwd_exp2(hi.y)};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (MASKED) {
        const int yi = y0i + c + i;
        e[i] = ((yi >= y_lo) & (yi < y_hi)) ? e[i] : 0.f;
      }
      sr[c + i] = __float_as_uint(e[i]);
    }
  }
}

// dS = P * (dP * scale - delta * scale) of 32 columns, packed to bf16 pairs. `pr`: the P of these columns.
template <bool DKV, bool MASKED>
__device__ __forceinline__ void ds_math(const uint32_t* pr, const uint32_t (&dr)[32], uint32_t stats_sa, float ndsc_row,
                                        int y0i, int y_lo, int y_hi, float scale, uint32_t (&dw)[16]) {
  const float2 s2 = make_float2(scale, scale);
#pragma unroll
  for (int c = 0; c < 32; c += 4) {
    float4 d = make_float4(ndsc_row, ndsc_row, ndsc_row, ndsc_row);
    if (DKV)
      asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w) : "r"(stats_sa + c * 4));
    const float2 t0 = __ffma2_rn(make_float2(__uint_as_float(dr[c]), __uint_as_float(dr[c + 1])), s2, make_float2(d.x, d.y));
    const float2 t1 = __ffma2_rn(make_float2(__uint_as_float(dr[c + 2]), __uint_as_float(dr[c + 3])), s2, make_float2(d.z, d.w));
    float2 g0 = __fmul2_rn(make_float2(__uint_as_float(pr[c]), __uint_as_float(pr[c + 1])), t0);
    float2 g1 = __fmul2_rn(make_float2(__uint_as_float(pr[c + 2]), __uint_as_float(pr[c + 3])), t1);
    if (MASKED) {   // P is zero there, but the statistics past the last query may be anything
      const int yi = y0i + c;
      g0.x = ((yi >= y_lo) & (yi < y_hi)) ? g0.x : 0.f;
      g0.y = ((yi + 1 >= y_lo) & (yi + 1 < y_hi)) ? g0.y : 0.f;
      g1.x = ((yi + 2 >= y_lo) & (yi + 2 < y_hi)) ? g1.x : 0.f;
      g1.y = ((yi + 3 >= y_lo) & (yi + 3 < y_hi)) ? g1.y : 0.f;
    }
    __nv_bfloat162 b0 = __floats2bfloat162_rn(g0.x, g0.y), b1 = __floats2bfloat162_rn(g1.x, g1.y);
    dw[c / 2] = *reinterpret_cast<uint32_t*>(&b0);
    dw[c / 2 + 1] = *reinterpret_cast<uint32_t*>(&b1);
  }
}

// DKV = true : X = (K, V) stationary, Y = (Q, dO) streamed, rows are keys, columns queries.
// DKV = false: X = (Q, dO) stationary, Y = (K, V) streamed, rows are queries, columns keys.
template <int D, bool DKV, int KS>
__global__ void __launch_bounds__(kBwdThreads, ctas_per_sm(KS))
flash_bwd_wide_kernel(const __grid_constant__ CUtensorMap tmX0, const __grid_constant__ CUtensorMap tmX1,
                 const __grid_constant__ CUtensorMap tmY0, const __grid_constant__ CUtensorMap tmY1,
                 const AttnBwdParams p) {
  using L = WideSmem<D, KS>;
  constexpr int kStream = KS;
  constexpr int C = kStream / 2;   // columns of a P / dS warp
  // TMEM columns: S, dP, accumulators (and X0, X1 in the dQ pass of D = 128, which has one accumulator)
  constexpr int kTmemCols = 2 * kStream + 2 * D <= 256 ? 256 : 512;
  extern __shared__ uint8_t smem_raw[];
  bwd_overlap_start<DKV>();
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  if (smem + L::kUsed > smem_raw + L::kTotal) {   // see WideSmem::kTotal; the same for every thread
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0u, kStatusBadArgs | (20u << 8));
    bwd_overlap_end<DKV>();
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBar);
  constexpr int R = L::kRing;
  uint64_t* x_full = bars;              // 1
  uint64_t* y_full = bars + 1;          // R
  uint64_t* y_empty = y_full + R;       // R
  uint64_t* s_full = y_empty + R;       // 1: S of the iteration is in TMEM
  uint64_t* dp_full = s_full + 1;       // 1: dP
  uint64_t* p_full = dp_full + 1;       // 1 (one arrival per warp): S was read, and P is in TMEM (dKV pass)
  uint64_t* ds_full = p_full + 1;       // 1 (one arrival per warp): dS is in TMEM
  uint64_t* acc_done = ds_full + 1;     // 1
  uint64_t* x_ready = acc_done + 1;     // 1 (one arrival per warp): X0 / X1 are in TMEM (kXTmem)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(x_ready + 1);
  volatile uint32_t* abort_w = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int G = p.Hq / p.Hkv;
  const BwdTile tile = bwd_tile<DKV>(p);
  const int b = tile.b, hx = tile.hx, x0 = tile.x0;   // hx: KV head (DKV) or query head (dQ)
  int y_first, y_count;
  bwd_stream<DKV, kStream>(p, tile, y_first, y_count);
  const int n_it = DKV ? y_count * G : y_count;

  if (threadIdx.x == 0) {
    *abort_w = 0;
    mbar_init(x_full, 1);
    for (int i = 0; i < R; ++i) {
      mbar_init(&y_full[i], 1);
      mbar_init(&y_empty[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, kSoftThreads / 32);
    mbar_init(ds_full, kSoftThreads / 32);
    mbar_init(acc_done, 1);
    mbar_init(x_ready, kSoftThreads / 32);
    fence_barrier_init();
    prefetch_tmap(&tmX0);
    prefetch_tmap(&tmX1);
    prefetch_tmap(&tmY0);
    prefetch_tmap(&tmY1);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_acc0 = tmem_base + 2 * kStream;
  const uint32_t tmem_acc1 = tmem_acc0 + D;
  // A product of 128 x 128 x 16 reads 8 KB of operands in the 64 cycles it takes: all that shared memory delivers, and
  // the streamed tiles have to be written there too. The dQ pass has no second accumulator: with D = 128 the stationary
  // operands of S and dP move to its columns once, and only the streamed operand is read per product (756 -> 738 us at
  // T = 8190, 32/8 heads).
  constexpr bool kXTmem = !DKV && D == 128;
  const uint32_t tmem_x0 = tmem_acc0, tmem_x1 = tmem_x0 + D / 2;
  WaitCtx wc{abort_w, p.status, p.wait_ns};

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && n_it > 0) {
      mbar_arrive_expect_tx(x_full, 2 * L::kStatBytes);
      // DKV: X tiles are K/V of kv head hx ; dQ: X tiles are Q/dO of query head hx
#pragma unroll
      for (int c = 0; c < L::kChunks; ++c) {
        tma_load_4d(smem + L::kX0 + c * (kStat * 128), &tmX0, x_full, c * 64, hx, x0, b);
        tma_load_4d(smem + L::kX1 + c * (kStat * 128), &tmX1, x_full, c * 64, hx, x0, b);
      }
      for (int t = 0; t < 2 * n_it; ++t) {
        const int it = t >> 1, s = t % R;
        const bool second = t & 1;   // Y1
        if (!mbar_wait_relaxed(&y_empty[s], ((t / R) & 1) ^ 1, wc, 1)) break;
        trace_pt<DKV>(p, 0, it, 1);
        int hy, yb;
        if (DKV) { hy = hx * G + it / y_count; yb = y_first + it % y_count; }
        else { hy = hx / G; yb = y_first + it; }
        uint8_t* y = smem + L::kY + s * L::kStreamBytes;
        mbar_arrive_expect_tx(&y_full[s], L::kStreamBytes + (DKV && second ? 2 * kStream * 4 : 0));
        if (DKV && second) {
          // the per-query statistics of the streamed tile ride along with it
          const long long so = ((long long)b * p.Hq + hy) * p.stat_stride + (long long)yb * kStream;
          float* st = reinterpret_cast<float*>(smem + L::kStats) + (it % L::kStatSlots) * 2 * kStream;
          bulk_load_1d(st, p.nlse2 + so, kStream * 4, &y_full[s]);
          bulk_load_1d(st + kStream, p.ndsc + so, kStream * 4, &y_full[s]);
        }
#pragma unroll
        for (int c = 0; c < L::kChunks; ++c)
          tma_load_4d(y + c * (kStream * 128), second ? &tmY1 : &tmY0, &y_full[s], c * 64, hy, yb * kStream, b);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    // The whole warp runs the loop with uniform control flow and an elected lane issues: tcgen05
    // operands live in uniform registers, and a divergent `if (lane == 0)` region would move every
    // one of them there per instruction, which costs more than a 128 x 64 x 16 MMA takes to run.
    if (n_it > 0) {
      constexpr uint32_t idesc_s = make_idesc_f16(kStat, kStream, 1, 0, 0);
      constexpr uint32_t idesc_acc = make_idesc_f16(kStat, D, 1, 0, 1);
      constexpr uint32_t hi = smem_desc_hi(1024);
      const uint32_t x0_lo = smem_desc_lo(smem_u32(smem + L::kX0), 16);
      const uint32_t x1_lo = smem_desc_lo(smem_u32(smem + L::kX1), 16);
      const uint32_t yk_lo = smem_desc_lo(smem_u32(smem + L::kY), 16);               // streamed tiles, K-major view
      const uint32_t ym_lo = smem_desc_lo(smem_u32(smem + L::kY), kStream * 128);    // the same tiles, MN-major view
      constexpr uint32_t kTile = L::kStreamBytes >> 4;
      // S (second = 0) or dP (second = 1) of iteration it. The columns are free: every MMA that read the tile before as
      // P or dS was issued earlier by this warp and the tensor pipe executes in order, and the P / dS warps had read
      // it into registers when they arrived for those MMAs (p_full in the dQ pass, which has no P product).
      auto issue_in = [&](int it, int second) -> bool {
        const int t = 2 * it + second, s = t % R;
        if (!mbar_wait_warp(&y_full[s], (t / R) & 1, wc, 2)) return false;
        tc_fence_after_sync();
        const uint32_t x_lo = second ? x1_lo : x0_lo, y_lo = yk_lo + s * kTile;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t xo = ((kk / 4) * (kStat * 128) + (kk % 4) * 32) >> 4;
            const uint32_t yo = ((kk / 4) * (kStream * 128) + (kk % 4) * 32) >> 4;
            if (kXTmem)
              umma_f16_ts_w(tmem_base + second * kStream, (second ? tmem_x1 : tmem_x0) + kk * 8, y_lo + yo, hi, idesc_s, kk != 0);
            else
              umma_f16_ss_w(tmem_base + second * kStream, x_lo + xo, hi, y_lo + yo, hi, idesc_s, kk != 0);
          }
          umma_commit(second ? dp_full : s_full);
          if (!DKV && second) umma_commit(&y_empty[s]);   // V is not needed again
        }
        __syncwarp();
        return true;
      };
      // acc += (P or dS)^T-or-not * Y: the A operand is bf16 pairs in TMEM, the C streamed rows of each half in the first
      // C / 2 of its C columns
      auto issue_acc = [&](int it, uint32_t t_a, uint32_t t_acc, int second) {
        const int s = (2 * it + second) % R;
        const uint32_t y_lo = ym_lo + s * kTile;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kStream / 16; ++kk)
            umma_f16_ts_w(t_acc, t_a + (kk / (C / 16)) * C + (kk % (C / 16)) * 8, y_lo + kk * (2048 >> 4), hi, idesc_acc, (it | kk) != 0);
          umma_commit(&y_empty[s]);
        }
        __syncwarp();
      };
      bool ok = mbar_wait_warp(kXTmem ? x_ready : x_full, 0, wc, 4);
      tc_fence_after_sync();
      if (ok) ok = issue_in(0, 0) && issue_in(0, 1);
      for (int it = 0; it < n_it && ok; ++it) {
        if (!mbar_wait_warp(p_full, it & 1, wc, 5)) break;
        if (lane == 0) trace_pt<DKV>(p, 1, it, 3);
        tc_fence_after_sync();
        if (DKV) issue_acc(it, tmem_base, tmem_acc0, 1);                     // dV += P^T dO
        if (it + 1 < n_it && !issue_in(it + 1, 0)) break;
        if (!mbar_wait_warp(ds_full, it & 1, wc, 10)) break;
        tc_fence_after_sync();
        issue_acc(it, tmem_base + kStream, tmem_acc1, 0);                      // dK += dS^T Q  or  dQ += dS K
        if (it + 1 < n_it) {
          if (!issue_in(it + 1, 1)) break;
        } else {
          if (elect_one()) umma_commit(acc_done);
          __syncwarp();
        }
        if (lane == 0) trace_pt<DKV>(p, 1, it, 4);
      }
    }
  } else {
    // ---------------------------------------------------------------- P / dS warps
    const int qd = warp & 3;
    const int half = (warp - 2) >> 2;  // which C of the tile's columns this warp handles
    const int row = qd * 32 + lane;
    const int xi = x0 + row;  // key index (DKV) or query index (dQ)
    const uint32_t t_lane = ((uint32_t)(qd * 32) << 16);
    float lse_row = 0.f, delta_row = 0.f;
    if (!DKV) {
      if (xi < p.Tq) {
        long long o = ((long long)b * p.Hq + hx) * p.stat_stride + xi;
        lse_row = p.nlse2[o];
        delta_row = p.ndsc[o];
      }
    }
    int y_lo, y_hi;
    bwd_row_bounds<DKV>(p, b, xi, y_lo, y_hi);
    bool ok = true;
    if (kXTmem && n_it > 0) {
      // one group of four warps per operand, a row per thread: 16-byte pieces of the 128-byte-swizzled tile to bf16 pairs
      // in consecutive columns
      ok = mbar_wait_warp(x_full, 0, wc, 12);
      if (ok) {
        const uint32_t xs = smem_u32(smem + (half ? L::kX1 : L::kX0)) + row * 128;
#pragma unroll
        for (int c = 0; c < L::kChunks; ++c) {
          uint32_t w[32];
#pragma unroll
          for (int j = 0; j < 8; ++j)
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(w[4 * j]), "=r"(w[4 * j + 1]), "=r"(w[4 * j + 2]), "=r"(w[4 * j + 3])
                         : "r"(xs + c * (kStat * 128) + ((j ^ (row & 7)) << 4)));
          tmem_st_32x32b_x16((half ? tmem_x1 : tmem_x0) + t_lane + c * 32, &w[0]);
          tmem_st_32x32b_x16((half ? tmem_x1 : tmem_x0) + t_lane + c * 32 + 16, &w[16]);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(x_ready);
      }
    }
    const uint32_t t_s = tmem_base + t_lane + half * C, t_dp = t_s + kStream;
    for (int it = 0; it < n_it && ok; ++it) {
      int yb;
      if (DKV) yb = y_first + it % y_count;
      else yb = y_first + it;
      const int y0i = yb * kStream + half * C;  // first query (DKV) or key (dQ) of this warp's columns
      // Valid streamed indices of this thread's row form one interval [lo, hi): tiles that lie
      // entirely inside it take the predicate-free path (warp-uniform choice).
      const bool need_mask = __any_sync(0xffffffffu, (y0i < y_lo) || (y0i + C > y_hi));
      uint32_t lse_sa = 0;
      float4 st[C / 4];
      if (DKV) {
        // the statistics landed with Y1 (the wait orders the read)
        const int t = 2 * it + 1;
        if (!mbar_wait_warp(&y_full[t % R], (t / R) & 1, wc, 9)) { ok = false; break; }
        lse_sa = smem_u32(smem + L::kStats) + ((it % L::kStatSlots) * 2 * kStream + half * C) * 4;
#pragma unroll
        for (int c = 0; c < C / 4; ++c)
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(st[c].x), "=f"(st[c].y), "=f"(st[c].z), "=f"(st[c].w) : "r"(lse_sa + c * 16));
      }
      if (!mbar_wait_warp(s_full, it & 1, wc, 6)) { ok = false; break; }
      if (threadIdx.x == 64) trace_pt<DKV>(p, 2, it, 1);
      tc_fence_after_sync();
      // 32 columns at a time, the next ones loaded under the math of the ones before
      uint32_t sr[C / 32][32], dr[C / 32][32];
      tmem_ld_32x32b_x32(t_s, sr[0]);
#pragma unroll
      for (int q = 0; q < C / 32; ++q) {
        tmem_ld_wait(sr[q]);
        if (q + 1 < C / 32) tmem_ld_32x32b_x32(t_s + (q + 1) * 32, sr[q + 1]);
        if (!DKV && q + 1 == C / 32) {
          // S was read: its columns are free for the next tile, whose product runs under this tile's exponentials
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_full);   // one arrival per warp: 32 on one barrier are served one after the other
        }
        if (need_mask) p_math<DKV, true>(sr[q], st + q * 8, lse_row, y0i + q * 32, y_lo, y_hi, p.scale_log2e);
        else p_math<DKV, false>(sr[q], st + q * 8, lse_row, y0i + q * 32, y_lo, y_hi, p.scale_log2e);
        if (DKV) {
          // P (bf16 pairs) goes back over this warp's own S columns
          uint32_t pw[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(sr[q][2 * i]), __uint_as_float(sr[q][2 * i + 1]));
            pw[i] = *reinterpret_cast<uint32_t*>(&h);
          }
          tmem_st_32x32b_x16(t_s + q * 16, pw);
        }
      }
      if (DKV) {
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      if (threadIdx.x == 64) trace_pt<DKV>(p, 2, it, 3);
      if (!mbar_wait_warp(dp_full, it & 1, wc, 11)) { ok = false; break; }
      tc_fence_after_sync();
      if (threadIdx.x == 64) trace_pt<DKV>(p, 2, it, 4);
      // dS of 32 columns at a time goes over dP columns that were already read
      tmem_ld_32x32b_x32(t_dp, dr[0]);
#pragma unroll
      for (int q = 0; q < C / 32; ++q) {
        uint32_t dw[16];
        tmem_ld_wait(dr[q]);
        if (q + 1 < C / 32) tmem_ld_32x32b_x32(t_dp + (q + 1) * 32, dr[q + 1]);
        const uint32_t d_sa = lse_sa + (kStream + q * 32) * 4;
        if (need_mask) ds_math<DKV, true>(sr[q], dr[q], d_sa, delta_row, y0i + q * 32, y_lo, y_hi, p.scale, dw);
        else ds_math<DKV, false>(sr[q], dr[q], d_sa, delta_row, y0i + q * 32, y_lo, y_hi, p.scale, dw);
        tmem_st_32x32b_x16(t_dp + q * 16, dw);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
      if (threadIdx.x == 64) trace_pt<DKV>(p, 2, it, 5);
    }
    if (ok && n_it > 0) ok = mbar_wait_warp(acc_done, 0, wc, 8);
    if (ok) {
      tc_fence_after_sync();
      bwd_store<D, DKV>(p, tile, tmem_acc0 + t_lane, tmem_acc1 + t_lane, xi, half, n_it > 0);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_w) {
    unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  bwd_overlap_end<DKV>();
}

template <int D, bool DKV, int KS>
static int launch_wide(const CUtensorMap& x0, const CUtensorMap& x1, const CUtensorMap& y0,
                      const CUtensorMap& y1, const AttnBwdParams& p, dim3 grid,
                      cudaStream_t stream) {
  using L = WideSmem<D, KS>;
  auto kern = flash_bwd_wide_kernel<D, DKV, KS>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return bwd_launch(kern, !DKV, grid, L::kTotal, stream, x0, x1, y0, y1, p);
}

int launch_bwd_wide(int D, bool dkv, const CUtensorMap& x0, const CUtensorMap& x1, const CUtensorMap& y0,
                    const CUtensorMap& y1, const AttnBwdParams& p, dim3 grid, cudaStream_t stream) {
  if (D == 128)
    return dkv ? launch_wide<128, true, bwd_wide_rows(128)>(x0, x1, y0, y1, p, grid, stream)
               : launch_wide<128, false, bwd_wide_rows(128)>(x0, x1, y0, y1, p, grid, stream);
  return dkv ? launch_wide<64, true, bwd_wide_rows(64)>(x0, x1, y0, y1, p, grid, stream)
             : launch_wide<64, false, bwd_wide_rows(64)>(x0, x1, y0, y1, p, grid, stream);
}

}  // namespace tpb
