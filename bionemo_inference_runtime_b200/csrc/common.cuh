// Shared host/device helpers for the sm_100a triangle-attention kernels.
//
// Device side: thin wrappers over the Blackwell PTX this library is built on
// (mbarrier, TMA bulk-tensor copies, tcgen05 MMA / TMEM access) plus the
// bounded waits every kernel uses.  Host side: status codes, the per-thread
// error string, the driver entry point for tensor-map encoding and the
// per-device status word kernels write when a wait runs out.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/b200ta.h"

namespace b200ta {

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

// Records a formatted message for b200ta_last_error() and returns `code`.
int fail(int code, const char* fmt, ...);

#define B200TA_CHECK_CUDA(expr)                                                        \
  do {                                                                                 \
    cudaError_t _e = (expr);                                                           \
    if (_e != cudaSuccess)                                                             \
      return ::b200ta::fail(B200TA_ERR_CUDA, "%s failed: %s", #expr,                   \
                            cudaGetErrorString(_e));                                   \
  } while (0)

#define B200TA_REQUIRE(cond, ...)                                                      \
  do {                                                                                 \
    if (!(cond)) return ::b200ta::fail(B200TA_ERR_INVALID, __VA_ARGS__);               \
  } while (0)

// Per-device state created on first use (a symbol-address lookup and a property query; no allocation).
// Callers are told to make their first call outside a stream capture.
struct DeviceState {
  int device = -1;
  int num_sms = 0;
  int* status_dev = nullptr;  // device word kernels write when they abandon a bounded wait
  std::atomic<uint32_t> configured{0};  // bit per KernelId: its shared-memory limit has been raised on this device
};
enum KernelId {
  kKernelPrologue, kKernelEpilogue, kKernelAttention, kKernelAttentionMasked, kKernelTransition, kKernelTransitionRelu,
  kKernelProject, kKernelContract, kKernelOutput, kKernelOutputF32, kKernelLinear, kKernelPairBias, kKernelRowStats,
  kKernelMaskRows
};
int get_device_state(DeviceState** out);

#ifdef __CUDACC__
// Launches a kernel that begins with pdl_wait(): the stream may start its blocks while the last blocks of the kernel
// before it still run (programmatic dependent launch), so that barrier and tensor-memory set-up and the launch latency
// itself hide behind them.  A block's set-up takes 2-3 us of the 5-12 us a kernel needs at small token counts.
template <typename... P, typename... A>
int launch_kernel(DeviceState* st, KernelId id, void (*kernel)(P...), dim3 grid, int threads, int smem_bytes, void* stream,
                  A&&... args) {
  const uint32_t bit = 1u << id;
  if (smem_bytes > 0 && !(st->configured.load(std::memory_order_relaxed) & bit)) {
    B200TA_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    st->configured.fetch_or(bit, std::memory_order_relaxed);
  }
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(unsigned(threads));
  config.dynamicSmemBytes = size_t(smem_bytes);
  config.stream = static_cast<cudaStream_t>(stream);
  config.attrs = &attr;
  config.numAttrs = 1;
  B200TA_CHECK_CUDA(cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...));
  return B200TA_OK;
}
#endif

// Encodes a tiled bf16/fp32 tensor map. `dims`, `strides_bytes` (rank-1 entries,
// for dims 1..rank-1) and `box` are innermost first.
enum SwizzleMode { SWZ_NONE = 0, SWZ_32 = 1, SWZ_64 = 2, SWZ_128 = 3 };
int encode_tensor_map(CUtensorMap* map, const void* base, int elem_bytes, int rank,
                      const uint64_t* dims, const uint64_t* strides_bytes,
                      const uint32_t* box, SwizzleMode swz, const char* what);

// ---------------------------------------------------------------------------
// Device side
// ---------------------------------------------------------------------------
#ifdef __CUDACC__

// A wait that has not completed after this long gives up, raises the CTA's
// abort flag and lets the kernel unwind (status word = B200TA_ERR_DEVICE_WAIT).
constexpr uint64_t kWaitLimitNs = 1000ull * 1000ull * 1000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// ---- programmatic dependent launch -------------------------------------------
// Lets the stream's next kernel start its blocks as soon as every block of this one has come here and there is room for
// them.  In a kernel with tensor memory the warp that allocates it calls this right behind the allocation: tcgen05.alloc
// waits without a limit, so a block of the next kernel that got the columns first would wait for this kernel (pdl_wait)
// while this kernel waits for the columns.  (Called by all threads behind the barrier that follows, a node's small
// kernels started 0.1 us later each.)
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Returns once the kernels before this one in the stream are complete and their writes visible.  Every thread calls it
// before its first access to global memory, except for reads of packed weights: the pack entry points end with an
// ordinary launch, behind which no kernel can start before the weights are complete.  Loading them early takes the
// 32-135 KB a block needs off the critical path of a small call.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The value in a register of its own, which the compiler cannot compute again from where it came from.
template <typename T>
__device__ __forceinline__ T keep_in_register(T v) {
  static_assert(sizeof(T) == 4, "one register");
  T out;
  asm volatile("mov.b32 %0, %1;" : "=r"(out) : "r"(v));
  return out;
}

// ---- mbarrier --------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait.  Returns false (and raises *abort_flag) when the barrier has
// not flipped within kWaitLimitNs or another thread of the CTA already gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 31u) == 0u) {
      if (*abort_flag) return false;
      if (global_timer_ns() - t0 > kWaitLimitNs) {
        *abort_flag = 1;
        return false;
      }
    }
  }
  return true;
}

// The same wait made by all 32 lanes of a converged warp; every decision is a vote, so the result is the same in
// every lane, the code after it stays warp-uniform, and a failed poll costs no divergence bookkeeping.
__device__ __forceinline__ bool mbar_wait_warp_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  uint64_t t0 = 0;
  for (uint32_t spins = 1;; ++spins) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((spins & 63u) == 0u) {
      if (t0 == 0) t0 = global_timer_ns();
      const bool late = global_timer_ns() - t0 > kWaitLimitNs;
      if (__any_sync(0xffffffffu, late || *abort_flag)) {
        if (late) *abort_flag = 1;
        return false;
      }
    }
  }
}
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return mbar_wait_warp_slow(bar, parity, abort_flag);
}
// Waits for two barriers at once (one vote for the usual case that both are complete already).
__device__ __forceinline__ bool mbar_wait2_warp(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1,
                                                volatile int* abort_flag) {
  const bool a = mbar_try_wait(bar0, parity0), b = mbar_try_wait(bar1, parity1);
  if (__all_sync(0xffffffffu, a && b)) return true;
  return mbar_wait_warp_slow(bar0, parity0, abort_flag) && mbar_wait_warp_slow(bar1, parity1, abort_flag);
}
// ---- proxies / fences --------------------------------------------------------
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ---- TMA -----------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* m, uint32_t bar,
                                            int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(m), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* m, uint32_t bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"(m), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* m, uint32_t bar,
                                            int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst),
      "l"(m), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(m),
               "r"(src), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, uint32_t src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(m), "r"(src),
               "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, uint32_t src, int c0, int c1,
                                             int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::
          "l"(m),
      "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void tma_store_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ---- TMEM / tcgen05 ----------------------------------------------------------------
// Warp-collective: allocates `cols` (power of two, >= 32) TMEM columns and writes
// the base address to *slot (shared memory).
__device__ __forceinline__ void tmem_alloc(uint32_t slot_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols)
               : "memory");
}

// Shared-memory matrix descriptor for tcgen05.mma operands.
//   layout_type: 2 = 128-byte swizzle, 4 = 64-byte swizzle, 6 = 32-byte swizzle.
//   lbo/sbo are byte offsets (multiples of 16).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes,
                                                   uint32_t sbo_bytes, uint32_t layout_type) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;  // descriptor version for sm_100
  d |= static_cast<uint64_t>(layout_type & 7u) << 61;
  return d;
}
// The same with lbo, sbo and layout known at compile time: only the address field is computed.
template <uint32_t LBO, uint32_t SBO, uint32_t LAYOUT>
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
  constexpr uint32_t hi = (SBO >> 4) | (1u << 14) | (LAYOUT << 29), lo = (LBO >> 4) << 16;
  return (static_cast<uint64_t>(hi) << 32) | ((saddr >> 4) | lo);  // shared-memory addresses are below 2^18
}
constexpr uint32_t kLayoutSw128 = 2, kLayoutSw64 = 4, kLayoutSw32 = 6;

// Instruction descriptor for kind::f16 with bf16 operands and fp32 accumulation.
//   b_mn_major: B operand is MN-major (N contiguous) instead of K-major.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int m, int n, bool a_mn_major = false,
                                                       bool b_mn_major = false) {
  return (1u << 4)                                   // D format: f32
         | (1u << 7)                                 // A format: bf16
         | (1u << 10)                                // B format: bf16
         | ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) |
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]; issued by one thread.
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                        uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Warp-collective forms (A in shared or in tensor memory): executed by all 32 lanes of a converged warp with the same
// operands; one elected lane issues.  A warp that stays converged lets the compiler keep descriptors and addresses in
// uniform registers: measured on B200, a thread inside an `if (lane == 0)` branch issues one tcgen05.mma every 45-80
// clocks whatever its size, the collective form one every 15 (N = 32) to 50 (N = 128) clocks, i.e. at the rate
// the tensor pipe retires them.  The elected lane is the same every time (the lowest one), so a later
// umma_commit_warp covers all MMAs of the warp.
__device__ __forceinline__ void umma_ss_warp(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, e;\nsetp.ne.b32 p, %4, 0;\nelect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_ts_warp(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, e;\nsetp.ne.b32 p, %4, 0;\nelect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit_warp(uint32_t bar) {
  asm volatile(
      "{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(bar)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_warp(uint32_t bar) {
  asm volatile(
      "{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n"
      "@e mbarrier.arrive.shared::cta.b64 _, [%0];\n}" ::"r"(bar)
      : "memory");
}
// An arrival that hands shared memory back right after it was read, before the values have been used: the fence makes
// the loads complete first (without it the next TMA write overtook them now and then).
__device__ __forceinline__ void mbar_arrive_warp_after_reads(uint32_t bar) {
  __threadfence_block();
  __syncwarp();
  mbar_arrive_warp(bar);
}
// Arrives on `bar` once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}

// Warp-collective TMEM loads: lane i of the warp receives columns
// [col, col+N) of TMEM lane (taddr.lane + i).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
      "%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// 64 columns into 64 floats.
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, float (&r)[64]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
      "%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,"
      "%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];"
      : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]),
        "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]), "=f"(r[16]),
        "=f"(r[17]), "=f"(r[18]), "=f"(r[19]), "=f"(r[20]), "=f"(r[21]), "=f"(r[22]), "=f"(r[23]), "=f"(r[24]),
        "=f"(r[25]), "=f"(r[26]), "=f"(r[27]), "=f"(r[28]), "=f"(r[29]), "=f"(r[30]), "=f"(r[31]), "=f"(r[32]),
        "=f"(r[33]), "=f"(r[34]), "=f"(r[35]), "=f"(r[36]), "=f"(r[37]), "=f"(r[38]), "=f"(r[39]), "=f"(r[40]),
        "=f"(r[41]), "=f"(r[42]), "=f"(r[43]), "=f"(r[44]), "=f"(r[45]), "=f"(r[46]), "=f"(r[47]), "=f"(r[48]),
        "=f"(r[49]), "=f"(r[50]), "=f"(r[51]), "=f"(r[52]), "=f"(r[53]), "=f"(r[54]), "=f"(r[55]), "=f"(r[56]),
        "=f"(r[57]), "=f"(r[58]), "=f"(r[59]), "=f"(r[60]), "=f"(r[61]), "=f"(r[62]), "=f"(r[63])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Warp-collective TMEM store, the mirror of tmem_ld32.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
      "%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
      "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
      "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st1(uint32_t taddr, uint32_t r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(r) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- small math ---------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }
// Packed fp32 pairs (one instruction for two lanes of data on sm_100).
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3_f32(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Byte offset of 16-byte chunk `chunk` of row `row` inside a tile whose rows are
// 128 bytes (128-byte swizzle) or 64 bytes (64-byte swizzle); tile base must be
// 1024-byte (resp. 512-byte) aligned.  Matches what TMA writes and tcgen05 reads.
__device__ __forceinline__ uint32_t sw128_offset(uint32_t row, uint32_t chunk) {
  return row * 128u + ((chunk ^ (row & 7u)) << 4);
}
__device__ __forceinline__ uint32_t sw64_offset(uint32_t row, uint32_t chunk) {
  return row * 64u + ((chunk ^ ((row >> 1) & 3u)) << 4);
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr));
  return v;
}
// 16 bytes as two packed fp32 pairs.
__device__ __forceinline__ void lds_f32x2(uint32_t addr, uint64_t& a, uint64_t& b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w)
               : "memory");
}

// LayerNorm statistics {rstd, -mean * rstd} of a row of 128 bf16 channels in shared memory (two 64-channel halves of
// 128-byte swizzled rows, 16 KiB apart).  One pass over the row in packed fp32 pairs: sums of (x - k) and (x - k)^2 with k
// the row's first channel.  (k - mean)^2 is at most 127 variances, so the variance formula E[d^2] - E[d]^2 loses no more
// than 1e-5 of it.
__device__ __forceinline__ float2 row_stats_128(uint32_t tile, int row, float eps) {
  const float k = bf16_lo(lds128(tile + sw128_offset(row, 0)).x);
  const uint64_t nk2 = pack_f32x2(-k, -k);
  uint64_t sa[4] = {0ull, 0ull, 0ull, 0ull}, sq[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 8
  for (int c = 0; c < 16; ++c) {
    const uint4 x = lds128(tile + (c >> 3) * 16384 + sw128_offset(row, c & 7));
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint64_t d = add_f32x2(pack_f32x2(bf16_lo(w[e]), bf16_hi(w[e])), nk2);
      sa[e] = add_f32x2(sa[e], d);
      sq[e] = fma_f32x2(d, d, sq[e]);
    }
  }
  float a0, a1, q0, q1;
  unpack_f32x2(add_f32x2(add_f32x2(sa[0], sa[1]), add_f32x2(sa[2], sa[3])), a0, a1);
  unpack_f32x2(add_f32x2(add_f32x2(sq[0], sq[1]), add_f32x2(sq[2], sq[3])), q0, q1);
  const float md = (a0 + a1) * (1.f / 128);  // mean of x - k
  const float var = fmaxf((q0 + q1) * (1.f / 128) - md * md, 0.f);
  const float rstd = rsqrtf(var + eps);
  return make_float2(rstd, -(md + k) * rstd);
}

#endif  // __CUDACC__

}  // namespace b200ta
