// Shared by the two forms of the attention backward (flash_bwd.cu, flash_bwd_wide.cu).
#pragma once
#include "sm100.cuh"

namespace tpb {

int make_tmap_bthd(CUtensorMap* out, const void* base, int B, int T, int H, int D,
                   long long tok_stride, long long head_stride, long long batch_stride, int rows);

constexpr int kBwdThreads = 320;  // TMA warp, MMA warp, 8 P/dS warps (two per TMEM lane quarter)
constexpr int kSoftThreads = 256;
constexpr int kStat = 128;        // rows of the stationary tiles
constexpr int kStatPad = 128;     // the statistics' rows are padded to this many queries (whole streamed tiles)

struct AttnBwdParams {
  int B, Tq, Tk, Hq, Hkv;
  int causal, kv_offset;
  // optional key bounds of a query, as in the forward: window > 0 = local attention; seg_start / seg_end
  // [B * Tq] = keys [start, end) of every query, which with Tq == Tk (packed self-attention, the only form
  // that takes them) are also the queries [start, end) of every key
  int window;
  const int* seg_start;
  const int* seg_end;
  float scale, scale_log2e;
  const float* nlse2;  // [B, Hq, stat_stride]: -lse * log2(e)
  const float* ndsc;   // [B, Hq, stat_stride]: -delta * scale
  int stat_stride;     // Tq rounded up to kStatPad
  __nv_bfloat16* out0;  // dKV: dV ; dQ: unused
  __nv_bfloat16* out1;  // dKV: dK ; dQ: dQ
  long long out_tok, out_head, out_batch;
  uint32_t* status;
  unsigned long long wait_ns;
  unsigned long long* trace;  // optional: cycle stamps of CTA (0,0,0), see tpb_flash_bwd_set_trace
};

// Debug aid: cycle stamps of block (0,0,0), trace[((pass * 3 + who) * 64 + it) * 8 + tag] with pass 0 = dKV, 1 = dQ and
// who 0 = TMA warp, 1 = MMA warp, 2 = first P / dS thread. Only in the debug build: each stamp is a branch, which the
// compiler schedules nothing across.
#ifdef TPB_KERNEL_DEBUG
constexpr bool kBwdTrace = true;
#else
constexpr bool kBwdTrace = false;
#endif
constexpr int kBwdTraceWords = 2 * 3 * 64 * 8;
template <bool DKV>
__device__ __forceinline__ void trace_pt(const AttnBwdParams& p, int who, int it, int tag) {
  if (kBwdTrace && p.trace && it < 64 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0)
    p.trace[(((DKV ? 0 : 3) + who) * 64 + it) * 8 + tag] = clock64();
}

__device__ __forceinline__ float bwd_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));  // pure: let the compiler schedule it
  return y;
}

// The dQ pass needs nothing of the dKV pass: its CTAs start as soon as those of the dKV pass have all started, and fill the
// SMs that run out of them (the dKV pass of 32/8 heads at T = 4096 has 256 CTAs of 4 to 128 tiles). The dQ launch is a
// programmatic dependent of the dKV launch; its last CTA waits for the dKV pass before it ends, so that what follows in the
// stream follows both.
// Both passes: 8 x 309 tokens, 16/4 heads 62 -> 46 us (D = 64: 46 -> 36), 2 x 4096 with a window of 512 198 -> 180, 2 x 2048
// without a mask 242 -> 216, T = 4096 with 32/8 heads 440 -> 413, T = 8190 1571 -> 1553.
template <bool DKV>
__device__ __forceinline__ void bwd_overlap_start() {
  if (DKV) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <bool DKV>
__device__ __forceinline__ void bwd_overlap_end() {
  if (!DKV && blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1 && blockIdx.z == gridDim.z - 1)
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... Params, typename... Args>
int bwd_launch(void (*kern)(Params...), bool overlap, dim3 grid, int smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kBwdThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return (int)cudaLaunchKernelEx(&cfg, kern, args...);
}

// What a CTA works on: batch, head (KV head for dKV, query head for dQ) and first row of its stationary tile.
// CTAs start in the order of their linear index; with a causal mask the tile index is the slowest coordinate, heaviest
// tile first (key tile 0 for dK/dV, the last query tile for dQ), heads and batches the fastest, so that the light CTAs of
// all heads fill the tail.
struct BwdTile {
  int b, hx, x0;
};
template <bool DKV>
__device__ __forceinline__ BwdTile bwd_tile(const AttnBwdParams& p) {
  int b = blockIdx.z, hx = blockIdx.y, xi = blockIdx.x;
  if (p.causal) {
    const int lin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    const int hb = gridDim.y * gridDim.z;
    xi = lin / hb;
    hx = (lin % hb) % gridDim.y;
    b = (lin % hb) / gridDim.y;
  }
  return {b, hx, ((DKV || !p.causal) ? xi : (int)gridDim.x - 1 - xi) * kStat};
}

// Streamed tiles of KS rows that the stationary tile at x0 may pair with: [first, first + count).
template <bool DKV, int KS>
__device__ __forceinline__ void bwd_stream(const AttnBwdParams& p, const BwdTile& t, int& first, int& count) {
  const long long seg_base = (long long)t.b * p.Tq;
  const int x0 = t.x0;
  first = 0;
  if (DKV) {
    // queries of this key tile: from the first key's lower bound to the last key's upper bound
    int q_hi = p.Tq;
    const int k_last = min(x0 + kStat - 1, p.Tk - 1);
    if (p.causal) {
      const int qmin = x0 - p.kv_offset;
      first = qmin > 0 ? qmin / KS : 0;
    }
    if (p.window > 0) q_hi = min(q_hi, k_last - p.kv_offset + p.window);
    if (p.seg_start && x0 < p.Tk) first = max(first, p.seg_start[seg_base + x0] / KS);
    if (p.seg_end && x0 < p.Tk) q_hi = min(q_hi, p.seg_end[seg_base + k_last]);
    count = max((max(q_hi, 0) + KS - 1) / KS - first, 0);
  } else {
    // keys of this query tile: from the first query's lower bound to the last query's upper bound
    int nkb = (p.Tk + KS - 1) / KS;
    const int q_last = min(x0 + kStat - 1, p.Tq - 1);
    if (p.causal) {
      const int last_key = x0 + kStat - 1 + p.kv_offset;
      nkb = min(nkb, last_key < 0 ? 0 : last_key / KS + 1);
    }
    if (p.seg_end && x0 < p.Tq) nkb = min(nkb, (p.seg_end[seg_base + q_last] + KS - 1) / KS);
    int lo_first = 0;
    if (p.window > 0) lo_first = max(lo_first, x0 + p.kv_offset - p.window + 1);
    if (p.seg_start && x0 < p.Tq) lo_first = max(lo_first, p.seg_start[seg_base + x0]);
    first = lo_first / KS;
    count = max(nkb - first, 0);
  }
}

// Streamed indices (queries for dKV, keys for dQ) that row xi (a key, a query) may pair with: [lo, hi).
template <bool DKV>
__device__ __forceinline__ void bwd_row_bounds(const AttnBwdParams& p, int b, int xi, int& lo, int& hi) {
  const long long seg_base = (long long)b * p.Tq;
  if (DKV) {
    lo = (xi < p.Tk) ? (p.causal ? max(xi - p.kv_offset, 0) : 0) : 0x3fffffff;
    hi = p.Tq;
    if (p.window > 0) hi = min(hi, xi - p.kv_offset + p.window);
  } else {
    lo = 0;
    hi = (xi < p.Tq) ? (p.causal ? min(p.Tk, xi + p.kv_offset + 1) : p.Tk) : 0;
    if (p.window > 0) lo = max(lo, xi + p.kv_offset - p.window + 1);
  }
  if (xi < (DKV ? p.Tk : p.Tq)) {
    if (p.seg_start) lo = max(lo, p.seg_start[seg_base + xi]);
    if (p.seg_end) hi = min(hi, p.seg_end[seg_base + xi]);
  }
}

// A warp's half of its accumulator rows (dV and dK, or dQ) to global memory; zeros where nothing was streamed.
template <int D, bool DKV>
__device__ __forceinline__ void bwd_store(const AttnBwdParams& p, const BwdTile& t, uint32_t t_acc0, uint32_t t_acc1, int xi,
                                          int half, bool streamed) {
  const long long obase = (long long)t.b * p.out_batch + (long long)xi * p.out_tok + (long long)t.hx * p.out_head;
#pragma unroll 1
  for (int a = DKV ? 0 : 1; a < 2; ++a) {
    __nv_bfloat16* orow = (a == 0 ? p.out0 : p.out1) + obase;
    const uint32_t t_acc = a == 0 ? t_acc0 : t_acc1;
#pragma unroll 1
    for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {
      uint32_t o[32];
      if (streamed) {
        tmem_ld_32x32b_x32(t_acc + c * 32, o);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0;
      }
      if (xi < (DKV ? p.Tk : p.Tq)) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 v;
          __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            h[i] = __floats2bfloat162_rn(__uint_as_float(o[g * 8 + 2 * i]), __uint_as_float(o[g * 8 + 2 * i + 1]));
          *reinterpret_cast<uint4*>(orow + c * 32 + g * 8) = v;
        }
      }
    }
  }
}

// The wide form, by head dimension 128 (128-row streamed tiles) or 64 (64-row tiles, two CTAs per SM): rows of its
// streamed tiles, and the launch of one pass.
constexpr int bwd_wide_rows(int d) { return d; }
int launch_bwd_wide(int D, bool dkv, const CUtensorMap& x0, const CUtensorMap& x1, const CUtensorMap& y0,
                    const CUtensorMap& y1, const AttnBwdParams& p, dim3 grid, cudaStream_t stream);

}  // namespace tpb
