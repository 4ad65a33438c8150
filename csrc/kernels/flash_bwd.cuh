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
  unsigned long long* trace;  // optional: timestamps of CTA (0,0,0), see tpb_flash_bwd_set_trace
  int trace_cap;
};

// Debug aid: records (role, iteration, phase, globaltimer) tuples of block (0,0,0).
__device__ __forceinline__ void trace_pt(const AttnBwdParams& p, int role, int it, int phase) {
  if (p.trace && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
    unsigned long long idx = atomicAdd(p.trace, 1ull);
    if ((int)idx < p.trace_cap) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
      p.trace[1 + idx * 2] = ((unsigned long long)role << 48) | ((unsigned long long)(it & 0xffffff) << 16) | (unsigned)phase;
      p.trace[2 + idx * 2] = t;
    }
  }
}

__device__ __forceinline__ float bwd_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));  // pure: let the compiler schedule it
  return y;
}

// The wide form, by head dimension 128 (128-row streamed tiles) or 64 (64-row tiles, two CTAs per SM): rows of its
// streamed tiles, and the launch of one pass.
constexpr int bwd_wide_rows(int d) { return d; }
int launch_bwd_wide(int D, bool dkv, const CUtensorMap& x0, const CUtensorMap& x1, const CUtensorMap& y0,
                    const CUtensorMap& y1, const AttnBwdParams& p, dim3 grid, cudaStream_t stream);

}  // namespace tpb
