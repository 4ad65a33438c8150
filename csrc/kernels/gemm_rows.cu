// bf16 GEMM for few rows of A (M <= 128, K-major: decoding, small batches) on clusters that split the reduction:
//   C[m, n] (+)= alpha * sum_k A(m, k) * B(n, k)  (+ bias[n])
// The product is bound by streaming B once. The weight rows are the 128-row operand of the MMA and the NT = 16..128
// rows of A its column operand, so a stage is 16 KB of weights plus 2..16 KB, and the two CTAs of an SM keep about
// 190 KB in flight. (With A as the 128-row operand, as in the one-CTA kernel, most rows of its tiles are empty and only
// N / 128 CTAs work.) A cluster of up to eight CTAs shares the k-blocks of one 128-column tile: every CTA drains its
// fp32 partial tile into its own shared memory, and after a cluster barrier each sums a slice of the tile over the
// cluster through distributed shared memory, in rank order, and stores it. The reduction needs no workspace, no flags
// and no second launch, so it is safe on any stream and under graph capture, and its result does not depend on timing.
//
// Measured against the other two kernels (operands beyond L2): M = 1, N = 4096, K = 14336: 70 -> 22 us; M = 16,
// N = K = 4096: 25 -> 11 us, N = 28672: 52 -> 41 us (5.7 TB/s), N = 128256: 190 -> 165 us (6.4 TB/s).
#include "sm100.cuh"
#include "tpb_api.h"

namespace tpb {

constexpr int kRowsThreads = 192;   // warp 0 TMA, warp 1 TMEM owner + MMA issue, warps 2..5 drain
constexpr int kRowsK = 64;
constexpr int kRowsBBytes = 128 * kRowsK * 2;

template <int NT>
struct RowsCfg {
  static constexpr int kStageBytes = kRowsBBytes + NT * kRowsK * 2;
  static constexpr int kStages = NT <= 32 ? 5 : (NT == 64 ? 4 : 3);
  static constexpr int kTmemCols = NT < 32 ? 32 : NT;
  static constexpr int kTileBytes = NT * 132 * 4;   // the partial tile reuses the ring: [NT][128 + 4] floats
  static_assert(kTileBytes <= kStages * kStageBytes, "the partial tile must fit the ring");
  static constexpr int kSmem = kStages * kStageBytes + 1024 + 256;   // two CTAs per SM
};

struct RowsParams {
  int M, N, K, ldc;
  void* C;
  const void* bias;
  int bias_f32, out_f32, accumulate;
  float alpha;
  uint32_t* status;
  unsigned long long wait_ns;
};

// CHAINED: launched while the kernel before may still run. On its own the form without that takes, with / without, 16 x 4096 x
// 4096 11.1 / 10.6 us, 128 x 4096 x 4096 15.4 / 14.7, 37 x 7184 x 1024 9.2 / 8.8.
template <int NT, bool B_MN, bool CHAINED>
__global__ void __launch_bounds__(kRowsThreads, 2)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmA,
                   const RowsParams p) {
  using Cfg = RowsCfg<NT>;
  constexpr int S = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * Cfg::kStageBytes);
  uint64_t* empty = full + S;
  uint64_t* done = empty + S;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile uint32_t* abort_w = tmem_slot + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank(), csize = (int)cluster_nctas();
  const int tile = blockIdx.x / csize;
  const int n0 = tile * 128;
  const int k_blocks = (p.K + kRowsK - 1) / kRowsK;
  const int per = k_blocks / csize, rem = k_blocks % csize;
  const int kb0 = rank * per + min(rank, rem);
  const int n_kb = per + (rank < rem ? 1 : 0);   // the host keeps csize <= k_blocks

  if (CHAINED) chain_next();
  if (threadIdx.x == 0) {
    *abort_w = 0;
    for (int i = 0; i < S; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(done, 1);
    fence_barrier_init();
    prefetch_tmap(&tmB);
    prefetch_tmap(&tmA);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  WaitCtx wc{abort_w, p.status, p.wait_ns};

  if (warp == 0) {
    // (warp-uniform control flow, one elected lane issues)
    auto load_b = [&](int it) {
      const int s = it % S, k = (kb0 + it) * kRowsK;
      uint8_t* sp = smem + s * Cfg::kStageBytes;
      mbar_arrive_expect_tx(&full[s], Cfg::kStageBytes);
      if (!B_MN) {
        tma_load_2d(sp, &tmB, &full[s], k, n0);
      } else {
#pragma unroll
        for (int c = 0; c < 2; ++c) tma_load_2d(sp + c * (kRowsK * 128), &tmB, &full[s], n0 + c * 64, k);
      }
    };
    // In a chain the weights are nobody's output: a ring of them is requested while the kernel before still runs. Otherwise the
    // first k-block would wait for all of that, so its rows of A are requested with it.
    const int ahead = min(S, n_kb);
    if (CHAINED) {
      for (int it = 0; it < ahead; ++it) {
        if (elect_one()) load_b(it);
        __syncwarp();
      }
      chain_wait();
    }
    for (int it = 0; it < n_kb; ++it) {
      const int s = it % S;
      if (it >= ahead && !mbar_wait_relaxed_warp(&empty[s], ((it / S) & 1) ^ 1, wc, 1)) break;
      if (elect_one()) {
        if (!CHAINED || it >= ahead) load_b(it);
        tma_load_2d(smem + s * Cfg::kStageBytes + kRowsBBytes, &tmA, &full[s], (kb0 + it) * kRowsK, 0);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    // warp-uniform control flow, one elected lane issues (tcgen05 operands live in uniform registers)
    if (CHAINED) chain_wait();
    constexpr uint32_t idesc = make_idesc_f16(128, NT, 1, B_MN ? 1 : 0, 0);
    constexpr uint32_t hi = smem_desc_hi(1024);
    const uint32_t p_lo0 = smem_desc_lo(smem_u32(smem), B_MN ? kRowsK * 128 : 16);
    const uint32_t q_lo0 = smem_desc_lo(smem_u32(smem + kRowsBBytes), 16);
    for (int it = 0; it < n_kb; ++it) {
      const int s = it % S;
      if (!mbar_wait_warp(&full[s], (it / S) & 1, wc, 2)) break;
      tc_fence_after_sync();
      const uint32_t p_lo = p_lo0 + s * (Cfg::kStageBytes >> 4), q_lo = q_lo0 + s * (Cfg::kStageBytes >> 4);
      if (elect_one()) {
#pragma unroll
        for (int j = 0; j < kRowsK / 16; ++j) {
          const uint32_t po = B_MN ? j * (2048 >> 4) : j * (32 >> 4);
          umma_f16_ss_w(tmem, p_lo + po, hi, q_lo + j * (32 >> 4), hi, idesc, (it | j) != 0);
        }
        umma_commit(&empty[s]);
        if (it == n_kb - 1) umma_commit(done);
      }
      __syncwarp();
    }
  } else {
    // drain the accumulator into the ring (every load has landed and every MMA has read it once `done` completes)
    const int q = warp & 3;
    if (CHAINED) chain_wait();
    if (mbar_wait_warp(done, 0, wc, 3)) {
      tc_fence_after_sync();
      const int row = q * 32 + lane;
      const uint32_t t_row = tmem + ((uint32_t)(q * 32) << 16);
      float* tile_s = reinterpret_cast<float*>(smem);
      constexpr int STEP = NT < 32 ? 16 : 32;
#pragma unroll 1
      for (int c = 0; c < NT; c += STEP) {
        uint32_t r[32];
        if constexpr (STEP == 16) {
          uint32_t r16[16];
          tmem_ld_32x32b_x16(t_row + c, r16);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = r16[i];
        } else {
          tmem_ld_32x32b_x32(t_row + c, r);
          tmem_ld_wait();
        }
#pragma unroll
        for (int i = 0; i < STEP; ++i) tile_s[(c + i) * 132 + row] = __uint_as_float(r[i]);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_w) {
    // copies of this CTA may still be in flight: give them time before memory is read or goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();   // every partial tile of the cluster is in shared memory
  if (!*abort_w)
    cluster_sum_store<128, 132, 1, 8>({p.C, p.ldc, p.N, p.bias, p.bias_f32, p.out_f32, p.accumulate, p.alpha}, smem_u32(smem), 0,
                                   p.M, n0, rank * kRowsThreads + (int)threadIdx.x, csize * kRowsThreads, 0, csize);
  cluster_sync_all();   // nobody leaves while a peer may read its tile
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, Cfg::kTmemCols);
  }
}

template <int NT, bool B_MN>
static cudaError_t rows_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int csize, unsigned tiles) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<NT, B_MN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         RowsCfg<NT>::kSmem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(gemm_rows_kernel<NT, B_MN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, RowsCfg<NT>::kSmem);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = csize;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg->gridDim = dim3(tiles * csize);
  cfg->blockDim = dim3(kRowsThreads);
  cfg->dynamicSmemBytes = RowsCfg<NT>::kSmem;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  return cudaSuccess;
}

// Cluster size for `tiles` tiles of `kb` k-blocks: rounds of resident clusters times the k-blocks of one CTA, plus
// six k-blocks a round for prologue and drain and two for the cluster's barriers and reduction. How many clusters of
// a size fit at once depends on how many SMs the device's GPCs have left (48 clusters of 6 do not, although 288 CTAs
// would: N = 6144 took 17 us with 6 against 10 us for N = 4096 with 8), so it is asked of the runtime, once per size.
template <int NT, bool B_MN>
static int rows_cluster(int tiles, int kb) {
  static int resident[9] = {0};
  long long best_cost = -1;
  int best = 1;
  for (int c = 1; c <= 8 && c <= kb; ++c) {
    if (resident[c] == 0) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      int n = 0;
      if (rows_config<NT, B_MN>(&cfg, attr, c, 2 * sm_count()) != cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&n, gemm_rows_kernel<NT, B_MN, false>, &cfg) != cudaSuccess || n <= 0)
        n = -1;
      resident[c] = n;
    }
    if (resident[c] < 0) continue;
    const long long rounds = (tiles + resident[c] - 1) / resident[c];
    const long long cost = rounds * ((kb + c - 1) / c + 6 + (c > 1 ? 2 : 0));
    if (best_cost < 0 || cost < best_cost) { best = c; best_cost = cost; }
  }
  return best;
}

template <int NT, bool B_MN>
static int launch_rows(const CUtensorMap& tb, const CUtensorMap& ta, const RowsParams& p, cudaStream_t stream) {
  const int tiles = (p.N + 127) / 128;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cudaError_t e = rows_config<NT, B_MN>(&cfg, attr, rows_cluster<NT, B_MN>(tiles, (p.K + kRowsK - 1) / kRowsK), tiles);
  if (e != cudaSuccess) return (int)e;
  cfg.stream = stream;
  if (t_chained) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  return (int)cudaLaunchKernelEx(&cfg, t_chained ? gemm_rows_kernel<NT, B_MN, true> : gemm_rows_kernel<NT, B_MN, false>, tb, ta, p);
}

// Which products of at most 128 rows go here; the others go to the persistent one-CTA kernel, which loads its next tile
// under the stores of the last. What this kernel gains is the split of K over a cluster while there are fewer tiles
// than CTAs that fit (two per SM), and the small column operand; what it pays is an epilogue of 3 us a round at 16 rows
// and 9 us at 128, under which nothing is loaded. Column tiles (N / 128) x K, us here / there, operands from memory:
//   M = 16: 64 x 4096 16.5 / 24.2, 296 x 4096 52.5 / 54.9, 393 x 1024 28.6 / 28.3, 393 x 2048 39.8 / 41.0
//   M = 32: 250 x 2048 26.4 / 26.6, 393 x 2048 42.0 / 41.6, 393 x 3072 57.8 / 59.9, 700 x 1024 48.0 / 39.8
//   M = 64: 72 x 1024 10.2 / 10.4, 72 x 4096 20.2 / 24.3, 78 x 2048 18.0 / 15.1, 78 x 3072 17.0 / 19.7, 96 x 4096 29.6 / 25.0
//   M = 128: 20 x 512 7.3 / 7.0, 30 x 512 7.7 / 7.0, 44 x 1024 10.7 / 10.2, 44 x 2048 13.3 / 14.8, 64 x 2048 16.6 / 15.1,
//            64 x 4096 23.4 / 24.2, 56 x 8192 35.8 / 42.2, 78 x 8192 35.3 / 42.7, 112 x 8192 62.3 / 46.7
// (the step between 72 and 78 tiles is that of the cluster size, two to three; M = 40 80 x 2560 14.3 / 17.4, M =
// 128 27 x 768 7.9 / 8.3). With results that the other kernel stores from its lanes one by one more stay here (`store`: 1
// accumulated, 2 fp32 with a bias). As 2: M = 16 393 x 1024 26.8 / 31.6, M = 32 29.7 / 32.9, 700 x 1024 47.0 / 45.8, M =
// 64 148 x 1536 19.3 / 23.1, 224 x 14336 153.5 / 142.7, 290 x 1024 24.4 / 28.3, 393 x 14336 266.8 / 282.8.
// A single row: 128256 x 2048 84 / 87, 50304 x 768 19.5 / 19.8, 128256 x 512 30 / 26. Over 1286 such products the choice
// takes 1.003 of the faster kernel on average and 1.16 at most.
bool gemm_rows_takes(int M, int N, int K, int a_mn, int store) {
  if (M > 128 || a_mn) return false;
  const long long tiles = (N + 127) / 128, sms = sm_count();
  if (M <= 32)
    return tiles <= 2 * sms || K >= (M <= 4 ? 768 : M <= 16 ? 2048 : 3072) || (store && (M <= 16 || tiles <= 3 * sms));
  if (K >= (M <= 100 ? 2560 : 3072) && tiles <= sms * 3 / 5) return true;
  if (M <= 64)
    return tiles <= sms / 2 || (store == 2 ? tiles >= sms : store && tiles > sms * 7 / 4 && tiles <= 2 * sms);
  return tiles <= sms / 7 || (K >= (tiles <= sms / 4 ? 768 : 1024) && tiles <= sms / 3);
}

// Same contract as gemm_bf16_dispatch for the plain product with a K-major A of at most 128 rows.
int gemm_rows_dispatch(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldb,
                       int ldc, int b_mn, int out_f32, int bias_f32, int accumulate, float alpha, uint32_t* status,
                       cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (M > 128 || K <= 0 || (lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) & 15) ||
      (reinterpret_cast<uintptr_t>(B) & 15))
    return -2;
  const int nt = M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128));
  CUtensorMap tb, ta;
  int r = !b_mn ? make_tmap_2d_bf16(&tb, B, K, N, ldb, 128) : make_tmap_2d_bf16(&tb, B, N, K, ldb, kRowsK);
  if (r) return r;
  if ((r = make_tmap_2d_bf16(&ta, A, K, M, lda, nt))) return r;
  RowsParams p;
  p.M = M; p.N = N; p.K = K; p.ldc = ldc;
  p.C = C; p.bias = bias; p.bias_f32 = bias_f32; p.out_f32 = out_f32; p.accumulate = accumulate; p.alpha = alpha;
  p.status = status; p.wait_ns = kDefaultWaitNs;
#define TPB_ROWS_CASE(NT) \
  if (nt == NT) return b_mn ? launch_rows<NT, true>(tb, ta, p, stream) : launch_rows<NT, false>(tb, ta, p, stream);
  TPB_ROWS_CASE(16)
  TPB_ROWS_CASE(32)
  TPB_ROWS_CASE(64)
  TPB_ROWS_CASE(128)
#undef TPB_ROWS_CASE
  return -3;
}

}  // namespace tpb
