// Product with 4- or 8-bit weights for more rows than the GEMV takes: y = x dequant(W)^T (+ bias), the weights converted on
// their way to the tensor cores.
//
// Converting a weight matrix to bf16 in a pass of its own writes and reads two bytes per weight, four times what 4-bit
// weights take, and a second kernel multiplies. Here a CTA owns 128 weight rows (the 128-row operand) and NT rows of x (16 to
// 192, the column operand): TMA brings the packed weights and the x tile, eight warps turn 128 k of a weight row per pair of
// threads into bf16 and write them into TMEM, from where the MMA takes its A operand: the bf16 weights never touch shared
// memory, whose bandwidth is what a one-CTA tile is short of. Four warps store the previous tile meanwhile (two
// accumulators). Every weight is converted once per NT rows of x.
//
// The bf16 weight has the bits of the pass (code - zero) * scale in fp32, rounded: where the zero point is a whole number up to
// 127, as the quantiser makes it, code - zero is exact in bf16 and its product with the scale is rounded once.
//
// Bound by the conversion for few rows (0.42 us per 128 x 128 weights and SM: 16 warps' nibble extraction, waits and stores to
// TMEM, about twice the MMAs of 64 rows), by it and the MMAs alternating for many (0.68 us at 160 rows). 4 bits, M x N x K, us
// with the weights converted in a pass of their own / here: 777 x 14336 x 4096 114 / 86 (1 070 TFLOP/s), 128 x 14336 x 4096
// 60 / 26, 64 x 8192 x 8192 70 / 36, 333 x 28672 x 8192 285 / 179, 512 x 4096 x 4096 30 / 25; 8 bits 116 / 100, 55 / 26, 65 / 34,
// 275 / 184, 28 / 26.
#include "sm100.cuh"
#include "tpb_api.h"

namespace tpb {

int make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_elems,
                   const uint32_t* box, int swizzle128);
int make_tmap_2d_packed(CUtensorMap* out, const void* base, uint64_t inner, uint64_t rows, uint64_t pitch, uint32_t box_inner,
                        uint32_t box_rows);

namespace {

constexpr int kWqThreads = 704;     // warp 0 TMA, 1 MMA, 2..9 and 10..17 conversion, 18..21 results
constexpr int kWqMaxNT = 192;
constexpr int kWqMaxStages = 8;
constexpr int kWqMaxA = 4;

struct WqGemmParams {
  int M, N, K, NT, m_tiles, n_tiles, w_stages, x_stages;
  int a_stages;     // buffers of converted weights in TMEM: 2, or 4 beside accumulators of at most 128 columns
  int gpr;          // groups per weight row
  int kb_shift;     // k-blocks of 128 per group = 2^kb_shift, or 31 with one scale per row
  long long ldy;
  const __nv_bfloat16 *scale, *zero, *bias;
  __nv_bfloat16* y;
  uint32_t* status;
  unsigned long long wait_ns;
};

// (v & mask) | the bits of 128 in both halves: codes of up to 7 bits as the bf16 numbers 128 + code, exact.
__device__ __forceinline__ uint32_t wq_and_or(uint32_t v, uint32_t mask) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(v), "r"(mask), "r"(0x43004300u));
  return r;
}
__device__ __forceinline__ __nv_bfloat162 as_bf2(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ uint4 wq_lds(uint32_t a) {
  uint4 r;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a));
  return r;
}

template <int BITS>
__global__ void __launch_bounds__(kWqThreads, 1)
wq_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const WqGemmParams p) {
  constexpr int kWBytes = 128 * 128 * BITS / 8;   // packed weights of a k-block
  constexpr int kWRow = 128 * BITS / 8;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int x_bytes = p.NT * 256;                 // x tile of a k-block: two halves of 64 k
  uint8_t* w_sm = smem;
  uint8_t* x_sm = smem + p.w_stages * kWBytes;
  uint64_t* w_full = reinterpret_cast<uint64_t*>(x_sm + p.x_stages * x_bytes);
  uint64_t* w_empty = w_full + kWqMaxStages;
  uint64_t* x_full = w_empty + kWqMaxStages;
  uint64_t* x_empty = x_full + kWqMaxStages;
  uint64_t* a_full = x_empty + kWqMaxStages;
  uint64_t* a_empty = a_full + kWqMaxA;
  uint64_t* tfull = a_empty + kWqMaxA;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile uint32_t* abort_w = tmem_slot + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = p.n_tiles * p.m_tiles, kbs = p.K / 128;

  if (threadIdx.x == 0) {
    *abort_w = 0;
    for (int i = 0; i < kWqMaxStages; ++i) {
      mbar_init(&w_full[i], 1);
      mbar_init(&w_empty[i], 8);
      mbar_init(&x_full[i], 1);
      mbar_init(&x_empty[i], 1);
    }
    for (int i = 0; i < kWqMaxA; ++i) {
      mbar_init(&a_full[i], 8);
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);
    }
    fence_barrier_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const int acc_cols = p.a_stages == 2 ? kWqMaxNT : 128;
  const uint32_t tmem_a = tmem + 2 * acc_cols;    // k-blocks of bf16 weights, 64 columns each
  WaitCtx wc{abort_w, p.status, p.wait_ns};

  if (warp == 0) {
    // warp-uniform control flow, one elected lane issues: from a branch of lane 0 a copy takes twice as long to issue
    int ws = 0, xs = 0;
    uint32_t wph = 1, xph = 1;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      const int n0 = tile / p.m_tiles * 128, m0 = tile % p.m_tiles * p.NT;
      for (int kb = 0; kb < kbs; ++kb) {
        if (!mbar_wait_relaxed_warp(&w_empty[ws], wph, wc, 1)) { ok = false; break; }
        if (elect_one()) {
          mbar_arrive_expect_tx(&w_full[ws], kWBytes);
          tma_load_2d(w_sm + ws * kWBytes, &tmW, &w_full[ws], kb * kWRow, n0);
        }
        __syncwarp();
        if (++ws == p.w_stages) { ws = 0; wph ^= 1; }
        if (!mbar_wait_relaxed_warp(&x_empty[xs], xph, wc, 2)) { ok = false; break; }
        if (elect_one()) {
          mbar_arrive_expect_tx(&x_full[xs], x_bytes);
          uint8_t* dst = x_sm + xs * x_bytes;
          tma_load_2d(dst, &tmX, &x_full[xs], kb * 128, m0);
          tma_load_2d(dst + p.NT * 128, &tmX, &x_full[xs], kb * 128 + 64, m0);
        }
        __syncwarp();
        if (++xs == p.x_stages) { xs = 0; xph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // warp-uniform control flow, one elected lane issues (tcgen05 operands live in uniform registers)
    const uint32_t idesc = make_idesc_f16(128, p.NT, 1, 0, 0);
    constexpr uint32_t hi = smem_desc_hi(1024);
    const uint32_t x_lo0 = smem_desc_lo(smem_u32(x_sm), 16), half = (p.NT * 128) >> 4;
    int xs = 0, as = 0, lt = 0;
    uint32_t xph = 0, aph = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++lt) {
      const int acc = lt & 1;
      if (!mbar_wait_warp(&tempty[acc], ((lt >> 1) & 1) ^ 1, wc, 3)) break;
      tc_fence_after_sync();
      const uint32_t d = tmem + acc * acc_cols;
      for (int kb = 0; kb < kbs; ++kb) {
        if (!mbar_wait_warp(&x_full[xs], xph, wc, 4) || !mbar_wait_warp(&a_full[as], aph, wc, 5)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t x_lo = x_lo0 + xs * (x_bytes >> 4), a = tmem_a + as * 64;
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            umma_f16_ts_w(d, a + j * 8, x_lo + (j >> 2) * half + (j & 3) * (32 >> 4), hi, idesc, (kb | j) != 0);
          umma_commit(&a_empty[as]);
          umma_commit(&x_empty[xs]);
          if (kb == kbs - 1) umma_commit(&tfull[acc]);
        }
        __syncwarp();
        if (++xs == p.x_stages) { xs = 0; xph ^= 1; }
        if (++as == p.a_stages) { as = 0; aph ^= 1; }
      }
    }
  } else if (warp < 18) {
    // ---------------------------------------------------------------- conversion: half of a weight row's 128 k per thread
    // Two groups of eight warps take the k-blocks in turn, each with buffers of its own in TMEM: a block is some 1 000
    // cycles of waiting, loading, arithmetic and storing to a warp.
    const int grp = (warp - 2) >> 3, q = warp & 3, hf = ((warp - 2) >> 2) & 1, row = q * 32 + lane;
    const uint32_t t_a = tmem_a + ((uint32_t)(q * 32) << 16) + hf * 32;
    int ws = grp % p.w_stages, as = grp;
    uint32_t wph = 0, aph = 1;
    __nv_bfloat16 s_next, z_next = __float2bfloat16(BITS == 4 ? 8.f : 0.f);
    auto sz_row = [&](int tile) {   // where the thread's row of a tile has its scales (rows past the last: zero codes)
      return (size_t)min(tile / p.m_tiles * 128 + row, p.N - 1) * p.gpr;
    };
    auto load_sz = [&](size_t at) {   // of the group's next k-block
      s_next = p.scale[at];
      if (BITS == 4 && p.zero) z_next = p.zero[at];
    };
    int first = grp;   // the group's first k-block of the tile
    size_t sz_at = (int)blockIdx.x < tiles ? sz_row(blockIdx.x) : 0;
    if (first < kbs) load_sz(sz_at + (first >> p.kb_shift));
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      const int next_first = (first + kbs) & 1;   // blocks alternate across tiles, too
      const bool more = tile + (int)gridDim.x < tiles && next_first < kbs;
      const size_t sz_then = tile + (int)gridDim.x < tiles ? sz_row(tile + gridDim.x) : sz_at;
      if (first >= kbs && more) load_sz(sz_then + (next_first >> p.kb_shift));
      for (int kb = first; kb < kbs; kb += 2) {
        const __nv_bfloat16 s = s_next, z = z_next;
        if (kb + 2 < kbs) load_sz(sz_at + ((kb + 2) >> p.kb_shift));
        else if (more) load_sz(sz_then + (next_first >> p.kb_shift));
        if (!mbar_wait_warp(&w_full[ws], wph, wc, 6)) { ok = false; break; }
        constexpr int V = BITS / 2;   // 16-byte pieces of 64 weights
        uint4 v[V];
        const uint32_t base = smem_u32(w_sm + ws * kWBytes) + row * kWRow;
        // pieces lie where the copy's swizzle put them (64 or 128 bytes wide)
#pragma unroll
        for (int i = 0; i < V; ++i)
          v[i] = wq_lds(base + (((hf * V + i) ^ (BITS == 4 ? (row >> 1) & 3 : row & 7)) << 4));
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_empty[ws]);
        if ((ws += 2) >= p.w_stages) { ws -= p.w_stages; wph ^= 1; }
        uint32_t o[32];
        const __nv_bfloat162 s2 = __halves2bfloat162(s, s);
        if (BITS == 8) {
#pragma unroll
          for (int i = 0; i < V; ++i) {
            const uint32_t w4[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                // a byte = its low 7 bits - 128 * sign: (128 + 7 bits) - (128, or 256 with the sign)
                const uint32_t b = __byte_perm(w4[j], 0u, e == 0 ? 0x1100 : 0x3322);
                const __nv_bfloat162 c = __hsub2(as_bf2(wq_and_or(b, 0x007F007Fu)), as_bf2(wq_and_or(b, 0x00800080u)));
                o[i * 8 + j * 2 + e] = as_u32(__hmul2(c, s2));
              }
          }
        } else {
          const float zf = __bfloat162float(z);
          const bool whole = zf == rintf(zf) && zf >= 0.f && zf <= 127.f;
          if (__all_sync(0xffffffffu, whole)) {
            const __nv_bfloat16 zb = __float2bfloat16(128.f + zf);
            const __nv_bfloat162 z2 = __halves2bfloat162(zb, zb);
#pragma unroll
            for (int i = 0; i < V; ++i) {
              const uint32_t w4[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint32_t h = w4[j] >> 4;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const uint32_t b = wq_and_or(__byte_perm(w4[j], h, 0x4400 + e * 0x1111), 0x000F000Fu);
                  o[i * 16 + j * 4 + e] = as_u32(__hmul2(__hsub2(as_bf2(b), z2), s2));
                }
              }
            }
          } else {
            const float sf = __bfloat162float(s);
#pragma unroll
            for (int i = 0; i < V; ++i) {
              const uint32_t w4[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
              for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float f0 = (float)((w4[j] >> (8 * e)) & 15u), f1 = (float)((w4[j] >> (8 * e + 4)) & 15u);
                  o[i * 16 + j * 4 + e] = as_u32(__floats2bfloat162_rn((f0 - zf) * sf, (f1 - zf) * sf));
                }
            }
          }
        }
        if (!mbar_wait_warp(&a_empty[as], aph, wc, 7)) { ok = false; break; }
        tc_fence_after_sync();
        tmem_st_32x32b_x16(t_a + as * 64, &o[0]);
        tmem_st_32x32b_x16(t_a + as * 64 + 16, &o[16]);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[as]);
        if ((as += 2) >= p.a_stages) { as -= p.a_stages; aph ^= 1; }
      }
      first = next_first;
      sz_at = sz_then;
    }
  } else {
    // ---------------------------------------------------------------- results: a weight row (a column of y) per thread
    const int q = warp & 3;
    int lt = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++lt) {
      const int acc = lt & 1;
      if (!mbar_wait_warp(&tfull[acc], (lt >> 1) & 1, wc, 8)) break;
      tc_fence_after_sync();
      const int n = tile / p.m_tiles * 128 + q * 32 + lane, m0 = tile % p.m_tiles * p.NT;
      const int rows = min(p.NT, p.M - m0);
      const uint32_t t_row = tmem + ((uint32_t)(q * 32) << 16) + acc * acc_cols;
      const float b = p.bias && n < p.N ? __bfloat162float(p.bias[n]) : 0.f;
      // even lanes store the even row of x for their own column and the next, odd lanes the odd row for the one before
      // and their own: four bytes a lane (columns come in eights)
      const bool odd = lane & 1;
      __nv_bfloat16* dst = p.y + (size_t)(m0 + odd) * p.ldy + (n & ~1);
      for (int c = 0; c < rows; c += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(t_row + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float f0 = __uint_as_float(r[i]) + b, f1 = __uint_as_float(r[i + 1]) + b;
          const float got = __shfl_xor_sync(0xffffffffu, odd ? f0 : f1, 1);
          const __nv_bfloat162 o = odd ? __floats2bfloat162_rn(got, f1) : __floats2bfloat162_rn(f0, got);
          if (c + i + odd < rows && n < p.N) *reinterpret_cast<__nv_bfloat162*>(dst + (size_t)(c + i) * p.ldy) = o;
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_w) {
    // copies of this CTA may still be in flight: give them time before memory goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

constexpr int wq_smem(int bits, int nt, int w_stages, int x_stages) {
  return w_stages * 128 * 128 * bits / 8 + x_stages * nt * 256 + 1024 + 512;
}

template <int BITS>
int launch_wq_gemm(const CUtensorMap& tw, const CUtensorMap& tx, const WqGemmParams& p, cudaStream_t stream) {
  static PerDevice done;
  const cudaError_t e = allow_smem(done, current_device(), wq_gemm_kernel<BITS>, 227 * 1024);
  if (e != cudaSuccess) return (int)e;
  const int tiles = p.n_tiles * p.m_tiles;
  wq_gemm_kernel<BITS><<<tiles < sm_count() ? tiles : sm_count(), kWqThreads, wq_smem(BITS, p.NT, p.w_stages, p.x_stages), stream>>>(
      tw, tx, p);
  return (int)cudaGetLastError();
}

// Rows of x per tile, by rounds of tiles times what a k-block takes (measured: 0.45 us at 16 rows, 0.51 at 64, 0.66 at 128, 0.69
// at 176); also that time for one k-block of all tiles. Tried are the twelve sizes there are, the larger one first where two cost
// the same: trying every number of row tiles, M / 16 of them, took 20 us of the host at 65536 rows, twice a call.
int wq_pick_nt(int M, int n_tiles, double* us) {
  int best = 0;
  for (int nt = kWqMaxNT; nt >= 16; nt -= 16) {
    if (nt > 16 && nt - 16 >= M) continue;   // no row in its last 16
    const long long tiles = (long long)n_tiles * ((M + (long long)nt - 1) / nt), rounds = (tiles + sm_count() - 1) / sm_count();
    const double cost = rounds * (0.42 + 0.0016 * nt);
    if (!best || cost < *us) { best = nt; *us = cost; }
  }
  return best;
}

bool wq_gemm_fits(int N, int K, int bits, int group) {
  const int blocks = group / 128;
  return K % 128 == 0 && N % 8 == 0 && (bits == 4 || bits == 8) && (bits == 8 || group > 0) &&
         (group <= 0 || (group % 128 == 0 && K % group == 0 && !(blocks & (blocks - 1))));
}

}  // namespace
}  // namespace tpb

using namespace tpb;

// Whether tpb_wq_gemm takes this product and is the fastest way to it. Up to 16 rows belong to the GEMV, which does not round
// the weights (9 x 28672 x 8192 77 us there, 61 here). The other way: a pass that converts the weights (two launches, 5 TB/s
// of packed and bf16 bytes) and the bf16 product (6 TB/s of weights or 1.1 PFLOP/s, 1.5 from 1024 rows on); of that 0.81 for few
// rows, where the product finds the weights in L2 and splits K: up to 40 rows, or 128 of 8 bits. us there / here, 4 bits: 17 x
// 4096 x 4096 18 / 18, 22 x 1280 x 1536 8.7 / 8.9, 27 x 7560 x 1280 13.5 / 9.1, 200 x 1024 x 1024 12 / 9, 1024 x 28672 x 8192
// 445 / 430, 4096 x 14336 x 4096 351 / 449; 8 bits: 35 x 2216 x 1664 10.0 / 10.2, 73 x 2152 x 3200 13.5 / 15.4, 87 x 3800 x 2816
// 16.7 / 15.0, 128 x 4096 x 4096 20.8 / 19.9.
extern "C" int tpb_wq_gemm_pays(int M, int N, int K, int bits, int group) {
  if (M <= 16 || N <= 0 || K <= 0 || !wq_gemm_fits(N, K, bits, group)) return 0;
  double us = 0;
  wq_pick_nt(M, (N + 127) / 128, &us);
  const double here = 4.3 + us * (K / 128), weights = (double)N * K, packed = weights * bits / 8;
  const double read = weights * 2 / 6e6, math = 2.0 * M * weights / (M < 1024 ? 1.1e9 : 1.5e9);
  const double there = 9 + (packed + 2 * weights) / 5e6 + (read > math ? read : math);
  return here < (M <= 40 || (M <= 128 && bits == 8) ? 0.81 : 1.0) * there;
}

// Arguments as tpb_wq_gemv, any number of rows; K a multiple of 128, one scale per row (8 bits, group 0) or groups of 128 times
// a power of two, N a multiple of 8, 16-byte aligned x and w, even ldy. -3: not such a product.
extern "C" int tpb_wq_gemm(const void* x, const void* w, const void* scale, const void* zero, const void* bias, void* y, int M,
                           int N, int K, int bits, int group, long long ldx, long long ldy, uint32_t* status, void* stream) {
  TPB_NVTX("tpb_wq_gemm");
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  if ((bits != 8 && bits != 4) || (bits == 4 && group <= 0)) return -2;
  if (!wq_gemm_fits(N, K, bits, group) || ldx % 8 || ldy % 2 || (reinterpret_cast<uintptr_t>(x) & 15) ||
      (reinterpret_cast<uintptr_t>(w) & 15) || (reinterpret_cast<uintptr_t>(y) & 3))
    return -3;
  WqGemmParams p;
  p.M = M; p.N = N; p.K = K; p.ldy = ldy;
  p.n_tiles = (N + 127) / 128;
  double us = 0;
  p.NT = wq_pick_nt(M, p.n_tiles, &us);
  p.m_tiles = (M + p.NT - 1) / p.NT;
  p.a_stages = p.NT <= 128 ? 4 : 2;
  // as many blocks of weights as of x ahead, where they fit
  p.w_stages = p.x_stages = kWqMaxStages;
  while (wq_smem(bits, p.NT, p.w_stages, p.x_stages) > 227 * 1024) {
    if (p.x_stages > 3 && p.x_stages >= p.w_stages) --p.x_stages;
    else --p.w_stages;
  }
  p.gpr = group > 0 ? K / group : 1;
  p.kb_shift = 31;
  if (group > 0)
    for (p.kb_shift = 0; (128 << p.kb_shift) < group;) ++p.kb_shift;
  p.scale = (const __nv_bfloat16*)scale; p.zero = (const __nv_bfloat16*)zero; p.bias = (const __nv_bfloat16*)bias;
  p.y = (__nv_bfloat16*)y; p.status = status; p.wait_ns = kDefaultWaitNs;
  CUtensorMap tw, tx;
  const uint64_t inner = (uint64_t)K * bits / 8;
  int r = make_tmap_2d_packed(&tw, w, inner, N, inner, 128 * bits / 8, 128);
  if (r) return r;
  const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M}, strides[2] = {1, (uint64_t)ldx};
  const uint32_t box[2] = {64, (uint32_t)p.NT};
  if ((r = make_tmap_bf16(&tx, x, 2, dims, strides, box, 1))) return r;
  return bits == 4 ? launch_wq_gemm<4>(tw, tx, p, (cudaStream_t)stream) : launch_wq_gemm<8>(tw, tx, p, (cudaStream_t)stream);
}
