// Thin inline-PTX wrappers for the Blackwell (sm_100a) execution model:
// mbarrier, TMA (cp.async.bulk.tensor, never with cluster multicast), tcgen05
// (TMEM alloc, UMMA issue, commit, TMEM loads) and bounded waits.
//
// Every wait in this file is bounded: a wait that runs out of time sets a
// shared abort word plus a global status word and returns false, so that the
// kernel can drain, free its TMEM and exit normally.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <nvtx3/nvToolsExt.h>

#include <atomic>

namespace tpb {

// NVTX ranges around the host side of every launching entry point, off unless tpb_nvtx_enable(1)
// was called (the profiler module does it inside `profiler.nvtx_kernels()`): a timeline then shows
// which library call queued which kernels. One global switch for all translation units.
extern int g_nvtx_on;
struct NvtxScope {
  bool on;
  explicit NvtxScope(const char* name) : on(g_nvtx_on != 0) { if (on) nvtxRangePushA(name); }
  ~NvtxScope() { if (on) nvtxRangePop(); }
  NvtxScope(const NvtxScope&) = delete;
  NvtxScope& operator=(const NvtxScope&) = delete;
};
#define TPB_NVTX(name) ::tpb::NvtxScope tpb_nvtx_scope_(name)

// Status codes written to the global status word (0 = ok).
enum : uint32_t {
  kStatusOk = 0,
  kStatusMbarTimeout = 1,
  kStatusFlagTimeout = 2,
  kStatusBadArgs = 3,
  kStatusBounds = 4,   // debug build: an index check failed (the access was skipped)
};

// Index checks of the debug build (-DTPB_KERNEL_DEBUG): TPB_DBG_CHECK(cond, site) evaluates to
// `cond`; when it is false the debug build also records kStatusBounds | site << 8 in the status
// word registered with tpb_debug_set_status, so that a guard which silently skips an access in the
// release build names its site in the debug build. Never traps: the caller skips the access.
#ifdef TPB_KERNEL_DEBUG
static __device__ uint32_t* g_dbg_status = nullptr;
__device__ __forceinline__ bool dbg_check(bool cond, uint32_t site) {
  if (!cond && g_dbg_status) atomicCAS(g_dbg_status, 0u, kStatusBounds | (site << 8));
  return cond;
}
#define TPB_DBG_CHECK(cond, site) ::tpb::dbg_check((cond), (site))
// Each translation unit has its own copy of g_dbg_status; it registers a setter here and
// tpb_debug_set_status calls them all.
typedef int (*DbgSetter)(uint32_t*);
void dbg_register_setter(DbgSetter fn);
static int dbg_set_local(uint32_t* p) { return (int)cudaMemcpyToSymbol(g_dbg_status, &p, sizeof(p)); }
namespace {
struct DbgRegistrar {
  DbgRegistrar() { dbg_register_setter(&dbg_set_local); }
};
static DbgRegistrar dbg_registrar_instance;
}  // namespace
#else
#define TPB_DBG_CHECK(cond, site) (cond)
#endif

// Default wait budget: 2 s of globaltimer. Host code may override per launch.
constexpr unsigned long long kDefaultWaitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Non-blocking probe: has the phase with this parity completed?
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// ---------------------------------------------------------------- launches that start early
// A chain of launches (see launch_chained) starts each kernel while the one before still runs. A kernel of a chain calls
// chain_next() at its start, which lets the next one's CTAs in as soon as all of its own have started, and chain_wait()
// in every thread before it touches what an earlier kernel of the chain reads or writes; what no kernel of the chain
// writes (weights, tables) it may load before. It then reads with chain_ld: a read-only load may be moved above the wait.
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ uint4 chain_ld(const void* p) {
  uint4 r;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}

// Host side: a value for each device of the process. What the runtime keeps per device (a kernel's shared-memory limit) or
// answers for one (how many clusters fit) is set or asked once on each; a process may launch on several, from several threads.
// 0 means not yet; devices past the last slot are set and asked on every call.
inline int current_device() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}
struct PerDevice {
  static constexpr int kDevices = 64;
  std::atomic<int> v[kDevices];
  template <typename F>
  int get(int dev, F&& ask) {
    if (dev < 0 || dev >= kDevices) return ask();
    int r = v[dev].load(std::memory_order_acquire);
    if (r == 0) {
      r = ask();
      v[dev].store(r, std::memory_order_release);
    }
    return r;
  }
};
// `kern` may have `bytes` of dynamic shared memory on the current device `dev` from then on.
template <typename K>
inline cudaError_t allow_smem(PerDevice& done, int dev, K kern, int bytes) {
  cudaError_t e = cudaSuccess;
  done.get(dev, [&] {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e == cudaSuccess ? 1 : 0;   // a failure is tried again
  });
  return e;
}

// Host side: whether the launches of this thread belong to a chain whose first kernel was launched; set for the extent of a
// native call that issues a chain.
extern thread_local bool t_chained;
template <typename... Params, typename... Args>
inline cudaError_t launch_chained(void (*kern)(Params...), dim3 grid, int threads, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = t_chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

// Shared per-CTA abort word + global status word used by all bounded waits.
struct WaitCtx {
  volatile uint32_t* abort_smem;  // set to 1 once any wait in the CTA gave up
  uint32_t* status_gmem;          // first failing code is kept (atomicCAS)
  unsigned long long limit_ns;
};

__device__ __forceinline__ void report_timeout(const WaitCtx& w, uint32_t code, uint32_t where) {
  *w.abort_smem = 1;
  if (w.status_gmem) atomicCAS(w.status_gmem, 0u, code | (where << 8));
}

// Bounded mbarrier wait. Returns false if the CTA is aborting.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const WaitCtx& w,
                                          uint32_t where) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0 = 0;
  uint32_t spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((++spins & 0xff) == 0) {
      if (*w.abort_smem) return false;
      unsigned long long t = globaltimer_ns();
      if (t0 == 0) t0 = t;
      else if (t - t0 > w.limit_ns) {
        report_timeout(w, kStatusMbarTimeout, where);
        return false;
      }
    }
  }
}

// Same bounded wait for threads that run far ahead of their consumers (TMA producers): it backs
// off between polls so that the spinning warp leaves the issue slots of its scheduler to the
// warps that do arithmetic.
__device__ __forceinline__ bool mbar_wait_relaxed(uint64_t* bar, uint32_t parity, const WaitCtx& w,
                                                  uint32_t where) {
  if (mbar_test(bar, parity)) return true;
  unsigned long long t0 = 0;
  uint32_t spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    __nanosleep(64);
    if ((++spins & 0x3f) == 0) {
      if (*w.abort_smem) return false;
      unsigned long long t = globaltimer_ns();
      if (t0 == 0) t0 = t;
      else if (t - t0 > w.limit_ns) {
        report_timeout(w, kStatusMbarTimeout, where);
        return false;
      }
    }
  }
}

// Warp-uniform form: every lane waits, and the warp proceeds only if all lanes succeeded, so
// that .sync.aligned instructions after the wait are never executed by a partial warp.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, const WaitCtx& w,
                                               uint32_t where) {
  bool ok = mbar_wait(bar, parity, w, where);
  return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ bool mbar_wait_relaxed_warp(uint64_t* bar, uint32_t parity, const WaitCtx& w, uint32_t where) {
  bool ok = mbar_wait_relaxed(bar, parity, w, where);
  return __all_sync(0xffffffffu, ok);
}

// Bounded wait on a 32-bit flag in global (possibly peer) memory reaching >= want.
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release_gpu(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_release_sys_add(uint32_t* p, uint32_t v) {
  asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_release_gpu_add(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Returns false on timeout (status word set). `sys` selects system scope (peer flags).
__device__ __forceinline__ bool flag_wait_ge(const uint32_t* flag, uint32_t want, bool sys,
                                             uint32_t* status_gmem, unsigned long long limit_ns,
                                             uint32_t where) {
  unsigned long long t0 = 0;
  uint32_t spins = 0;
  while (true) {
    uint32_t v = sys ? ld_acquire_sys(flag) : ld_acquire_gpu(flag);
    if ((int32_t)(v - want) >= 0) return true;
    if ((++spins & 0x3f) == 0) {
      unsigned long long t = globaltimer_ns();
      if (t0 == 0) t0 = t;
      else if (t - t0 > limit_ns) {
        if (status_gmem) atomicCAS(status_gmem, 0u, kStatusFlagTimeout | (where << 8));
        return false;
      }
      __nanosleep(64);
    }
  }
}

// ---------------------------------------------------------------- TMA
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar,
                                            int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
      "l"(m), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, uint64_t* bar,
                                            int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(m), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* m, uint64_t* bar,
                                            int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(dst)),
      "l"(m), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
// 1-D bulk copy global -> shared (16-byte aligned addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(m),
               "r"(smem_u32(src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait_all() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]; bf16/fp16 inputs, fp32 accumulate.
__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc].
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same two forms with the descriptors given as (low, high) 32-bit words. Within one operand
// tile only the start-address field (low word, units of 16 bytes) changes from one k-step to the
// next, so a caller keeps the high word and the base of the low word in registers and issues
// each MMA after a single 32-bit add: the issuing thread is one lane of one warp, and descriptor
// arithmetic redone per instruction (a chain of dependent 64-bit operations) costs more cycles
// than a 128 x 128 x 16 MMA takes to execute.
__device__ __forceinline__ void umma_f16_ss_w(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                              uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
      "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_f16_ts_w(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi,
                                              uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Words of a 128-byte-swizzle shared-memory descriptor (see make_smem_desc_sw128 below).
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t saddr, uint32_t lbo_bytes) {
  return ((saddr & 0x3FFFF) >> 4) | (((lbo_bytes >> 4) & 0x3FFF) << 16);
}
__host__ __device__ constexpr uint32_t smem_desc_hi(uint32_t sbo_bytes) {
  return ((sbo_bytes >> 4) & 0x3FFF) | (1u << 14) | (2u << 29);
}
// int8 x int8 -> int32
__device__ __forceinline__ void umma_i8_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on an mbarrier once all previously issued tcgen05.mma of this thread completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// The same as the definition of the 32 words that were loaded: nothing that uses them moves before it while later loads are
// in flight.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
      : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
        "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
        "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
        "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
      :
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// 32 lanes x 32 consecutive fp32 columns: thread i of the warp gets lane (base+i), cols c..c+31.
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 16 columns store (fp32 words / packed bf16x2) from registers into TMEM.
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15])
      : "memory");
}

// ---------------------------------------------------------------- descriptors
// Shared-memory matrix descriptor for 128-byte-swizzled tiles (tile base 1024-B aligned).
//   K-major  : rows of 64 bf16 (128 B); 8-row groups are `sbo` bytes apart (1024).
//   MN-major : 64-element (128 B) MN chunks, 8 k-rows per 1024-B atom;
//              `lbo` = bytes between 64-wide MN chunks, `sbo` = bytes between 8-k groups.
__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t saddr, uint32_t lbo_bytes,
                                                         uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version (Blackwell)
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}

// Instruction descriptor, kind::f16, fp32 accumulate.
//   ab_fmt: 0 = f16, 1 = bf16.  a_mn / b_mn: 1 if that operand is MN-major in smem.
__host__ __device__ constexpr uint32_t make_idesc_f16(int m, int n, int ab_fmt, int a_mn,
                                                      int b_mn) {
  return (1u << 4) | ((uint32_t)ab_fmt << 7) | ((uint32_t)ab_fmt << 10) |
         ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}
// kind::i8, int32 accumulate, signed int8 operands, both K-major.
__host__ __device__ constexpr uint32_t make_idesc_i8(int m, int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}

// ---------------------------------------------------------------- thread-block clusters
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_nctas() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Value at the same shared-memory offset in CTA `rank` of the cluster.
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t saddr, uint32_t rank) {
  float4 v;
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %4, %5;\n\t"
      "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n\t}"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "r"(saddr), "r"(rank)
      : "memory");
  return v;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t saddr, uint32_t rank) {
  float v;
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %1, %2;\n\t"
      "ld.shared::cluster.f32 %0, [ra];\n\t}"
      : "=f"(v)
      : "r"(saddr), "r"(rank)
      : "memory");
  return v;
}

// ---------------------------------------------------------------- warp MMA
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---------------------------------------------------------------- GEMM epilogues
// Where and how the sum of a split product leaves.
struct SumStore {
  void* C;
  int ldc, N;
  const void* bias;
  int bias_f32, out_f32, accumulate;
  float alpha;
};
// Sums the fp32 partial tiles of COLS columns (rows LD floats apart) that `parts` CTAs of a cluster hold at `base` in
// their shared memory, CTAs rank0, rank0 + STEP, .., in that order, and stores the result: `rows` rows from (row0, col0)
// on. Units of four columns are dealt out from u0 in steps of du. MOST: parts at most, all requested at once.
template <int COLS, int LD, int STEP, int MOST>
__device__ __forceinline__ void cluster_sum_store(const SumStore& p, uint32_t base, int row0, int rows, int col0, int u0,
                                                  int du, int rank0, int parts) {
  constexpr int UNITS = 2;   // in flight per thread
  for (int u = u0; u < rows * (COLS / 4); u += UNITS * du) {
    float4 t[UNITS][MOST];
    uint4 old[UNITS];
    uint8_t* o[UNITS];
    int cols[UNITS];   // of a unit that exist: 0 to 4
    bool vec[UNITS];
#pragma unroll
    for (int k = 0; k < UNITS; ++k) {
      const int uk = u + k * du, r = uk / (COLS / 4), j4 = (uk % (COLS / 4)) * 4, col = col0 + j4;
      cols[k] = r < rows ? max(0, min(4, p.N - col)) : 0;
      o[k] = reinterpret_cast<uint8_t*>(p.C) + ((size_t)(row0 + r) * p.ldc + col) * (p.out_f32 ? 4 : 2);
      vec[k] = cols[k] == 4 && (reinterpret_cast<uintptr_t>(o[k]) & (p.out_f32 ? 15 : 7)) == 0;
      // what is accumulated into is requested with the partial sums, and converted only where it is used: the warp
      // would wait for it here
      old[k] = make_uint4(0u, 0u, 0u, 0u);
      if (p.accumulate && vec[k]) {
        if (p.out_f32) {
          old[k] = *reinterpret_cast<const uint4*>(o[k]);
        } else {
          const uint2 w = *reinterpret_cast<const uint2*>(o[k]);
          old[k].x = w.x;
          old[k].y = w.y;
        }
      }
      const uint32_t at = base + (uint32_t)(r * LD + j4) * 4;
#pragma unroll
      for (int h = 0; h < MOST; ++h)
        t[k][h] = h < parts && cols[k] ? ld_cluster_f4(at, rank0 + STEP * h) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < UNITS; ++k) {
      const int col = col0 + ((u + k * du) % (COLS / 4)) * 4;
      float v[4] = {t[k][0].x, t[k][0].y, t[k][0].z, t[k][0].w};
#pragma unroll
      for (int h = 1; h < MOST; ++h) { v[0] += t[k][h].x; v[1] += t[k][h].y; v[2] += t[k][h].z; v[3] += t[k][h].w; }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i] *= p.alpha;
        if (p.bias && i < cols[k])
          v[i] += p.bias_f32 ? reinterpret_cast<const float*>(p.bias)[col + i]
                             : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[col + i]);
      }
      if (p.accumulate) {
        if (vec[k] && p.out_f32) {
          v[0] += __uint_as_float(old[k].x); v[1] += __uint_as_float(old[k].y);
          v[2] += __uint_as_float(old[k].z); v[3] += __uint_as_float(old[k].w);
        } else if (vec[k]) {
          const float2 f0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&old[k].x));
          const float2 f1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&old[k].y));
          v[0] += f0.x; v[1] += f0.y; v[2] += f1.x; v[3] += f1.y;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (i < cols[k])
              v[i] += p.out_f32 ? reinterpret_cast<const float*>(o[k])[i]
                                : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(o[k])[i]);
        }
      }
      if (vec[k] && p.out_f32) {
        *reinterpret_cast<float4*>(o[k]) = make_float4(v[0], v[1], v[2], v[3]);
      } else if (vec[k]) {
        uint2 w;
        *reinterpret_cast<__nv_bfloat162*>(&w.x) = __floats2bfloat162_rn(v[0], v[1]);
        *reinterpret_cast<__nv_bfloat162*>(&w.y) = __floats2bfloat162_rn(v[2], v[3]);
        *reinterpret_cast<uint2*>(o[k]) = w;
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < cols[k]) {
            if (p.out_f32) reinterpret_cast<float*>(o[k])[i] = v[i];
            else reinterpret_cast<__nv_bfloat16*>(o[k])[i] = __float2bfloat16(v[i]);
          }
      }
    }
  }
}

// The bias of 32 consecutive output columns, shared by all rows a warp drains. Every lane reads the same
// addresses, so the cost is the number of load instructions and their latency: four (bf16) or eight (fp32)
// 16-byte loads, issued by the caller before it waits for its TMEM load. As 32 two-byte loads inside the
// arithmetic the same bias made the CTA-pair kernel 3.3x slower at K = 768 (GPT-2-small, 16384 rows: 1.6 ->
// 5.4 ms over 17 products).
struct Bias32 {
  uint4 w[4];
};
// Whether the vector form applies: a whole 32-column chunk of a 16-byte aligned bf16 bias.
__device__ __forceinline__ bool bias32_vec_ok(const void* bias, int bias_f32, int col0, int N) {
  return bias && !bias_f32 && col0 + 32 <= N && ((reinterpret_cast<uintptr_t>(bias) & 15) == 0);
}
__device__ __forceinline__ void bias32_load(Bias32& b, const void* bias, int col0) {
  const uint4* s = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(bias) + col0);
#pragma unroll
  for (int i = 0; i < 4; ++i) b.w[i] = __ldg(s + i);
}
__device__ __forceinline__ void bias32_add(float (&v)[32], const Bias32& b) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(b.w);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] += f.x;
    v[2 * i + 1] += f.y;
  }
}
// Same for the other cases (fp32 or unaligned bias, last columns).
__device__ __forceinline__ void bias32_add_any(float (&v)[32], const void* bias, int bias_f32, int col0, int N) {
  if (bias_f32 && col0 + 32 <= N && ((reinterpret_cast<uintptr_t>(bias) & 15) == 0)) {
    const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(bias) + col0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 f = __ldg(s + i);
      v[4 * i] += f.x; v[4 * i + 1] += f.y; v[4 * i + 2] += f.z; v[4 * i + 3] += f.w;
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (col0 + i < N)
      v[i] += bias_f32 ? reinterpret_cast<const float*>(bias)[col0 + i]
                       : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[col0 + i]);
}

// The bias of a chunk of 32 columns in any of its forms.
__device__ __forceinline__ void bias32_apply(float (&v)[32], const void* bias, int bias_f32, int col0, int N) {
  if (bias32_vec_ok(bias, bias_f32, col0, N)) {
    Bias32 b;
    bias32_load(b, bias, col0);
    bias32_add(v, b);
  } else {
    bias32_add_any(v, bias, bias_f32, col0, N);
  }
}

// Plain bf16 results: 32 accumulator rows (the TMEM lanes of a warp) to `rows` valid rows of C, 64 columns at a time while
// `cols` lasts; returns the columns done. c: first row and column, 16-byte aligned like every row; bias: null, or
// 16-byte aligned bf16 at that column; stage: kDrainStage bytes of the warp's own.
// A lane holds 32 columns of one row. Stored from there, an instruction touches 32 rows by 16 bytes and takes 32 passes
// of the load/store unit, 4096 of the ~6000 cycles that the MMAs of a 256-row tile take at K = 768: the results go
// through shared memory (144-byte rows, free of conflicts both ways) and leave as 4 rows by 128 contiguous bytes. Both
// TMEM loads share one wait, and all of a chunk is read back before any of it is stored, which the compiler may not
// arrange by itself (the two could alias). CTA-pair kernel, 4096 x 4096, K = 64 / 1032 / 4096: 21.7 / 32.8 / 115.8 us
// with 32 columns at a time, 15.4 / 31.5 / 112.6 us so; stored from the lanes 21.1 / 35.3 / 119.5 us.
constexpr int kDrainStage = 32 * 144;
__device__ __forceinline__ int drain_bf16(uint32_t t_row, uint8_t* stage, __nv_bfloat16* c, size_t ldc, int rows, int cols,
                                          float alpha, const void* bias, int lane) {
  if (rows <= 0) return cols & ~63;
  int done = 0;
#pragma unroll 1
  for (; done + 64 <= cols; done += 64) {
    uint32_t r[2][32];
    tmem_ld_32x32b_x32(t_row + done, r[0]);
    tmem_ld_32x32b_x32(t_row + done + 32, r[1]);
    Bias32 b[2];
    if (bias) {
      bias32_load(b[0], bias, done);
      bias32_load(b[1], bias, done + 32);
    }
    tmem_ld_wait();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[h][i]) * alpha;
      if (bias) bias32_add(v, b[h]);
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint4 o;
        __nv_bfloat162* ob2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) ob2[j] = __floats2bfloat162_rn(v[i + 2 * j], v[i + 2 * j + 1]);
        *reinterpret_cast<uint4*>(stage + lane * 144 + h * 64 + i * 2) = o;
      }
    }
    __syncwarp();
    uint4 val[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      val[i] = *reinterpret_cast<const uint4*>(stage + (i * 4 + (lane >> 3)) * 144 + (lane & 7) * 16);
    __nv_bfloat16* dst = c + (size_t)(lane >> 3) * ldc + done + (lane & 7) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i * 4 + (lane >> 3) < rows) *reinterpret_cast<uint4*>(dst + (size_t)(i * 4) * ldc) = val[i];
    __syncwarp();
  }
  return done;
}

}  // namespace tpb
