// Thin inline-PTX wrappers for the Blackwell (sm_100a) execution model:
// mbarrier, TMA (cp.async.bulk.tensor, never with cluster multicast), tcgen05
// (TMEM allocation, UMMA issue, commit, TMEM loads) and the descriptor
// encodings they need.  Every wait in here is bounded: it gives up after a
// clock budget and reports failure so the caller can set a status word and
// leave the kernel cleanly instead of spinning forever.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace ab {

// A kernel attribute (dynamic shared memory limit, carve-out) belongs to one device's copy of the
// kernel, so "already set" is kept per device: one bit per device ordinal in a mask that each call
// site owns.  first_use_on_device() returns true until mark_device() was called on this device.
struct PerDeviceOnce {
  std::atomic<unsigned long long> mask{0};
  unsigned long long bit() const {
    int dev = 0;
    cudaGetDevice(&dev);
    return 1ull << (dev & 63);
  }
  bool first_use_on_device() const { return !(mask.load(std::memory_order_acquire) & bit()); }
  void mark_device() { mask.fetch_or(bit(), std::memory_order_release); }
};

inline cudaError_t device_sms(int* n) {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  return e != cudaSuccess ? e : cudaDeviceGetAttribute(n, cudaDevAttrMultiProcessorCount, dev);
}

// ---------------------------------------------------------------- status ---
// Kernels report trouble through a device status word owned by the host
// wrapper (never by trapping).  0 means success.
enum StatusCode : int {
  ST_OK = 0,
  ST_TIMEOUT_FULL = 1,      // consumer waited too long for a TMA stage
  ST_TIMEOUT_EMPTY = 2,     // producer waited too long for a free stage
  ST_TIMEOUT_TMEM_FULL = 3, // epilogue waited too long for an accumulator
  ST_TIMEOUT_TMEM_EMPTY = 4,// MMA warp waited too long for a drained accumulator
  ST_TIMEOUT_PEER = 5,      // wait on a flag written by another GPU ran out
  ST_TIMEOUT_MISC = 6,
  ST_BAD_ARGUMENT = 7,
};

// Spin budget in SM clock cycles (about one second at 1.9 GHz).
#ifndef AB_SPIN_CYCLES
#define AB_SPIN_CYCLES (2000000000ll)
#endif

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// One lane of a converged warp.  Loads by TMA, MMAs and what goes with them are issued by warp-uniform code: the
// whole warp runs the loop and hands the `lead` that this returned to the instructions.  In code that one
// lane runs by itself the operands (descriptors, coordinates) lie in that lane's registers and go one by one
// to the uniform registers that these instructions read: a 64-wide step of a contraction over 128 x 64 tiles took 530
// clocks, 345 this way.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t"
      "}\n"
      : "=r"(pred));
  return pred;
}
// The warp's number, known to be the same for all lanes
__device__ __forceinline__ int warp_number() { return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0); }

// -------------------------------------------------------------- mbarrier ---
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes, uint32_t lead) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
               "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}\n"
               ::"r"(smem_u32(bar)), "r"(bytes), "r"(lead) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok;
}
// Same test, but the thread may stay suspended for up to `hint_ns` nanoseconds waiting for the
// phase to complete before the instruction returns (it wakes as soon as the phase completes), so a
// polling loop around it issues far fewer instructions.
__device__ __forceinline__ uint32_t mbar_try_wait_suspend(uint64_t* bar, uint32_t parity,
                                                          uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok;
}
#ifndef AB_MBAR_SUSPEND_NS
#define AB_MBAR_SUSPEND_NS 2000u
#endif
// Bounded wait.  Returns false when the budget ran out (or another thread of
// the CTA has already raised `*abort_flag`).  `sleep_ns` > 0 puts the thread to sleep between
// polls: for waits with slack (an epilogue waiting for the next accumulator, a producer waiting
// for a free stage) this keeps the polling warps out of the issue slots and the power budget.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          volatile int* abort_flag, uint32_t sleep_ns = 0) {
  if (mbar_try_wait(bar, parity)) return true;
  long long t0 = clock64();
  uint32_t spins = 0;
  while (!mbar_try_wait_suspend(bar, parity, AB_MBAR_SUSPEND_NS)) {
    if (sleep_ns) __nanosleep(sleep_ns);
    if ((++spins & 0x3f) == 0) {
      if (*abort_flag) return false;
      if (clock64() - t0 > AB_SPIN_CYCLES) return false;
    }
  }
  return true;
}

// The same for a whole warp, converged: one verdict for all lanes, so that a warp whose wait ran out leaves as one.  (Its
// instructions that are the whole warp's, TMEM's among them, would wait without a limit for lanes that had left.)
// Voting on every poll keeps the loop uniform: one game of 90 tokens 960 us with a vote on the lanes' verdicts, or with
// verdicts per lane, and 934 so; attention forward 64 x 512 x 16 heads 92.3 per lane and 92.9 so, with dropout 143.4
// and 145.3.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (!__all_sync(0xffffffffu, mbar_try_wait_suspend(bar, parity, AB_MBAR_SUSPEND_NS)))
    if ((++spins & 0x3f) == 0 && __any_sync(0xffffffffu, *abort_flag || clock64() - t0 > AB_SPIN_CYCLES)) return false;
  return true;
}

// The same for a copy that has to land before its shared memory is given up (a block on its way out):
// another thread's trouble does not end this wait, only the clock does.
__device__ __forceinline__ bool mbar_wait_landed(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try_wait_suspend(bar, parity, AB_MBAR_SUSPEND_NS))
    if (clock64() - t0 > AB_SPIN_CYCLES) return false;
  return true;
}

// Makes generic-proxy writes to shared memory visible to the async proxy
// (TMA, tcgen05.mma operand fetch).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---------------------------------------------- programmatic dependent launch ---
// A kernel launched with the programmatic-stream-serialization attribute may start while the
// kernel before it in the stream is still running (once that kernel has executed
// griddep_launch_dependents in every CTA, or has exited).  It must call griddep_wait before it
// touches anything the earlier kernel produces or still reads; what it does before that (barrier
// set-up, TMEM allocation, prefetch of weights) overlaps the earlier kernel.  Both instructions
// are no-ops in a kernel launched the ordinary way.
__device__ __forceinline__ void griddep_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void griddep_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// First statement of a kernel that can be a link of a programmatic chain (the captured training
// micro-step): lets the kernel behind it in the stream become resident as this one drains, then
// waits for the kernel before it.  Everything the kernel reads or writes comes after this.
__device__ __forceinline__ void griddep_enter() {
  if (threadIdx.x == 0) griddep_launch_dependents();
  griddep_wait();
}

// Host side: launches made through launch_chained carry the programmatic-stream-serialization
// attribute while g_pdl_chain is set (only around the capture of a training micro-step; defined in
// embed.cu).  Every kernel launched this way starts with griddep_enter() or, as the GEMMs and the attention
// forward, does its set-up first and then waits.
extern int g_pdl_chain;
template <typename... KArgs, typename... Args>
inline cudaError_t launch_chained(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                  cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  if (g_pdl_chain) {
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
  }
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// A programmatic dependent of the kernel before it in the stream, whatever g_pdl_chain says
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                    Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// ------------------------------------------------------------------- TMA ---
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 2-D tiled load global -> shared, completion counted on `bar` in bytes.
// x is the innermost (contiguous) coordinate and must be a multiple of
// 16 bytes / element size.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar,
                                            int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x),
      "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];\n\t}\n"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(lead)
      : "memory");
}
// 2-D tiled store shared -> global (bulk async group).
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)), "r"(x), "r"(y)
               : "memory");
}
// 2-D tiled reduction shared -> global: global[tile] += smem[tile] (fp32 add, bulk async group).
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* m, const void* src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)), "r"(x), "r"(y)
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
__device__ __forceinline__ void tma_store_wait() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// --------------------------------------------------------------- tcgen05 ---
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Whole-warp calls.  ncols: power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_result)),
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
// D[tmem] (+)= A[smem desc] * B[smem desc], bf16 inputs, fp32 accumulate; by the warp's elected lane.
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate, uint32_t lead) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
      : "memory");
}
// Same with A in TMEM (lane = row, two K-adjacent bf16 values per 32-bit column).
__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate, uint32_t lead) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
      : "memory");
}
// Arrive on `bar` once every tcgen05.mma issued so far by the elected lane is done.
__device__ __forceinline__ void umma_commit(uint64_t* bar, uint32_t lead) {
  asm volatile(
      "{\n\t"
      ".reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
      "}\n"
      ::"r"(smem_u32(bar)), "r"(lead)
      : "memory");
}
// Each thread of the warp reads 32 consecutive fp32 columns of its own TMEM
// lane (lane = 32 * (warp_id % 4) + lane_id, encoded in taddr bits 31..16).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
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
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// The counterpart of tmem_ld16: each thread writes 16 consecutive 32-bit columns of its own lane.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Asks for `bytes` (a multiple of 16) of global memory from a 16-byte aligned address into L2.
__device__ __forceinline__ void bulk_prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// ------------------------------------------------------------- grid scheduling ---
// A running block takes the place of one of its grid that has not started, and does its work: the set-up is paid
// once per resident block, loads for the next work go out under the current one, and blocks that run ahead take more.
// The answer (16 bytes) arrives at `bar` (expect 16 bytes); after a "none left" no block may be asked for again.
__device__ __forceinline__ void grid_take_block(uint4* answer, uint64_t* bar, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
      "@q clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];\n\t}\n"
      ::"r"(smem_u32(answer)), "r"(smem_u32(bar)), "r"(lead) : "memory");
}
// Whether there was one, and which.  Whole warp; before asking again: fence_proxy_async_smem() and __syncwarp().
__device__ __forceinline__ bool grid_taken_block(const uint4* answer, uint3& block) {
  uint32_t yes, x, y, z;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t.reg .b32 w;\n\t"
      "ld.shared.b128 h, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, w}, h;\n\t}\n"
      : "=r"(yes), "=r"(x), "=r"(y), "=r"(z) : "r"(smem_u32(answer)) : "memory");
  block = make_uint3(x, y, z);
  return __shfl_sync(0xffffffffu, yes, 0) != 0;
}

// ------------------------------------------------- CTA pairs (cta_group::2) ---
// Two CTAs of a cluster (ranks 0 and 1) act as one MMA unit: the leader (rank 0) issues
// tcgen05.mma for both, each CTA stages its own half of A (rows) and of B (columns) in its own
// shared memory and owns 128 lanes of the accumulator in its own TMEM.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t mapa_shared(uint32_t cta_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(cta_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 2-D tiled load into this CTA's shared memory whose completion bytes are counted on a barrier
// that may live in the partner CTA (`bar_cluster_addr` from mapa_shared).  Plain unicast load.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* m,
                                                 uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(x),
      "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* m, uint32_t bar_cluster_addr, int x, int y,
                                                 uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];\n\t}\n"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(lead)
      : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate, uint32_t lead) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
      : "memory");
}
// Arrive on the barrier at `bar_cluster_addr` (either CTA of the pair) once every pair MMA issued
// so far by the elected lane is done.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar_cluster_addr, uint32_t lead) {
  asm volatile(
      "{\n\t"
      ".reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
      "}\n"
      ::"r"(bar_cluster_addr), "r"(lead)
      : "memory");
}

// ----------------------------------------------------------- descriptors ---
// Shared-memory matrix descriptor for 128-byte-swizzled bf16 tiles (the layout
// a TMA load with CU_TENSOR_MAP_SWIZZLE_128B produces).  Field positions:
// start>>4 [0,14), LBO>>4 [16,30), SBO>>4 [32,46), version=1 [46,48),
// layout type [61,64) with 2 = SWIZZLE_128B, 4 = SWIZZLE_64B.
// For `base` + `off`, both multiples of 16: neighbouring descriptors differ by one addition to the low word (shared
// memory ends below 2^18, so nothing carries out of the address field).
template <uint32_t LAYOUT>
__device__ __forceinline__ uint64_t make_sdesc(uint32_t base, uint32_t off, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  const uint32_t lo = (base >> 4) + ((off >> 4) | (((lbo_bytes >> 4) & 0x3FFF) << 16));
  const uint32_t hi = ((sbo_bytes >> 4) & 0x3FFF) | (1u << 14) | (LAYOUT << 29);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}
__device__ __forceinline__ uint64_t make_sdesc_sw128(uint32_t base, uint32_t off, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return make_sdesc<2>(base, off, lbo_bytes, sbo_bytes);
}
// Instruction descriptor for kind::f16 with bf16 A/B and fp32 accumulator.
// a_mn / b_mn: operand is MN-major (1) rather than K-major (0).
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, int a_mn, int b_mn) {
  return (1u << 4)      // D format fp32
         | (1u << 7)    // A format bf16
         | (1u << 10)   // B format bf16
         | (static_cast<uint32_t>(a_mn) << 15) | (static_cast<uint32_t>(b_mn) << 16) |
         (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

// ------------------------------------------------------------------ misc ---
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// gelu_new (tanh form) and its derivative.
// GELU (tanh form) and its derivative, written for the fewest issue slots: the GEMM epilogues that
// use them are bound by instruction issue.  With u = k0 (x + k1 x^3) = x (k0 + k0 k1 x^2), t = tanh u:
//   gelu(x)  = 0.5 x (1 + t)                      = fma(h, t, h),  h = 0.5 x          (6 operations)
//   gelu'(x) = 0.5 (1 + t) + 0.5 x (1 - t^2) u'   with u' = k0 + 3 k0 k1 x^2          (10 operations)
constexpr float GELU_K0 = 0.7978845608028654f;
constexpr float GELU_K01 = 0.7978845608028654f * 0.044715f;
__device__ __forceinline__ float gelu_tanh(float x) {
  const float t = tanh_fast(x * fmaf(GELU_K01, x * x, GELU_K0));
  const float h = 0.5f * x;
  return fmaf(h, t, h);
}
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float x2 = x * x;
  const float t = tanh_fast(x * fmaf(GELU_K01, x2, GELU_K0));
  const float dt = fmaf(-t, t, 1.f) * fmaf(3.f * GELU_K01, x2, GELU_K0);
  return fmaf(0.5f * x, dt, fmaf(0.5f, t, 0.5f));
}
// both at once (they share x^2 and the tanh): returns gelu(x), stores gelu'(x)
__device__ __forceinline__ float gelu_tanh_with_grad(float x, float& grad) {
  const float x2 = x * x;
  const float t = tanh_fast(x * fmaf(GELU_K01, x2, GELU_K0));
  const float h = 0.5f * x;
  grad = fmaf(h, fmaf(-t, t, 1.f) * fmaf(3.f * GELU_K01, x2, GELU_K0), fmaf(0.5f, t, 0.5f));
  return fmaf(h, t, h);
}

// ------------------------------------------------------------ packed fp32 ---
// Two fp32 values in one 64-bit register pair; one instruction does both (sm_100a).
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_bcast(float v) { return f2_pack(v, v); }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint32_t f2_to_bf16x2(uint64_t v) {
  float lo, hi;
  f2_unpack(v, lo, hi);
  return pack_bf16x2(lo, hi);
}
// gelu_tanh / gelu_tanh_with_grad of two values (same formulas as above)
__device__ __forceinline__ uint64_t f2_gelu_tanh(uint64_t x) {
  const uint64_t u = f2_mul(x, f2_fma(f2_bcast(GELU_K01), f2_mul(x, x), f2_bcast(GELU_K0)));
  float u0, u1;
  f2_unpack(u, u0, u1);
  const uint64_t t = f2_pack(tanh_fast(u0), tanh_fast(u1));
  const uint64_t h = f2_mul(x, f2_bcast(0.5f));
  return f2_fma(h, t, h);
}
__device__ __forceinline__ uint64_t f2_gelu_tanh_with_grad(uint64_t x, uint64_t& grad) {
  const uint64_t x2 = f2_mul(x, x);
  const uint64_t u = f2_mul(x, f2_fma(f2_bcast(GELU_K01), x2, f2_bcast(GELU_K0)));
  float u0, u1;
  f2_unpack(u, u0, u1);
  const uint64_t t = f2_pack(tanh_fast(u0), tanh_fast(u1));
  const uint64_t h = f2_mul(x, f2_bcast(0.5f));
  const uint64_t sech2 = f2_fma(f2_mul(t, f2_bcast(-1.f)), t, f2_bcast(1.f));
  const uint64_t du = f2_fma(f2_bcast(3.f * GELU_K01), x2, f2_bcast(GELU_K0));
  grad = f2_fma(h, f2_mul(sech2, du), f2_fma(f2_bcast(0.5f), t, f2_bcast(0.5f)));
  return f2_fma(h, t, h);
}

// ---------------------------------------------------------------- philox ---
// Counter-based generator (Philox4x32, 7 rounds) used for every dropout mask:
// the mask of element i of stream `stream` under `seed` is a pure function of
// (seed, stream, i), so backward kernels regenerate it instead of storing it.
struct Philox4 {
  uint32_t x, y, z, w;
};
__host__ __device__ __forceinline__ Philox4 philox4x32_7(uint64_t seed, uint32_t stream,
                                                         uint64_t counter) {
  uint32_t k0 = static_cast<uint32_t>(seed), k1 = static_cast<uint32_t>(seed >> 32);
  uint32_t c0 = static_cast<uint32_t>(counter), c1 = static_cast<uint32_t>(counter >> 32);
  uint32_t c2 = stream, c3 = 0x9E3779B9u;
#pragma unroll
  for (int r = 0; r < 7; ++r) {
    const uint64_t p0 = static_cast<uint64_t>(0xD2511F53u) * c0, p1 = static_cast<uint64_t>(0xCD9E8D57u) * c2;
    c0 = static_cast<uint32_t>(p1 >> 32) ^ c1 ^ k0;
    c2 = static_cast<uint32_t>(p0 >> 32) ^ c3 ^ k1;
    c1 = static_cast<uint32_t>(p1);
    c3 = static_cast<uint32_t>(p0);
    k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
  }
  return Philox4{c0, c1, c2, c3};
}
// The seed reaches a kernel by value, which a captured CUDA graph would freeze.  Every launcher
// therefore also hands its kernel seed_salt_ptr(): null in ordinary launches (the seed is used as
// it is), or, while a training step is being captured, the address of a device word that the
// graph's first node advances on every replay; kernels key the generator with salted(seed, salt).
extern const unsigned long long* g_seed_salt;       // host variable, defined in embed.cu
inline const unsigned long long* seed_salt_ptr() { return g_seed_salt; }
__device__ __forceinline__ unsigned long long salted(unsigned long long seed,
                                                     const unsigned long long* salt) {
  return salt ? (seed ^ __ldg(salt)) : seed;
}
// A value that is the same for all lanes of a converged warp, known to be: the generator's seven keys per half then
// lie in uniform registers instead of being added up for every draw.
__device__ __forceinline__ uint64_t uniform64(uint64_t v) {
  const uint32_t hi = __shfl_sync(0xffffffffu, static_cast<uint32_t>(v >> 32), 0);
  return (static_cast<uint64_t>(hi) << 32) | __shfl_sync(0xffffffffu, static_cast<uint32_t>(v), 0);
}
// Dropout decisions come in groups of eight consecutive elements: element
// index i uses 16 bits of philox(seed, stream, i / 8).  keep iff bits >= thr16.
__host__ __device__ __forceinline__ uint32_t dropout_thr16(float p) {
  float t = p * 65536.f;
  return t <= 0.f ? 0u : (t >= 65535.f ? 65535u : static_cast<uint32_t>(t + 0.5f));
}
__host__ __device__ __forceinline__ float dropout_scale(uint32_t thr16) {
  return 65536.f / static_cast<float>(65536u - thr16);
}
// Appends a keep bit to `m`: 1 where the upper 16 bits of `x` are at least the threshold.  `wrap` is
// -(thr16 << 16): the addition carries out exactly then, and the carry is shifted in (thr16 > 0).
__host__ __device__ __forceinline__ void push_keep(uint32_t& m, uint32_t x, uint32_t wrap) {
#ifdef __CUDA_ARCH__
  asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %1, %2;\n\taddc.u32 %0, %0, %0;\n\t}" : "+r"(m) : "r"(x), "r"(wrap));
#else
  m = 2 * m + (static_cast<uint64_t>(x) + wrap > 0xffffffffu);
#endif
}
// the eight bits of a group behind those in `m`, the last element first
__host__ __device__ __forceinline__ void push_keep8(uint32_t& m, uint64_t seed, uint32_t stream, uint64_t group, uint32_t wrap) {
  const Philox4 r = philox4x32_7(seed, stream, group);
  push_keep(m, r.w, wrap); push_keep(m, r.w << 16, wrap);
  push_keep(m, r.z, wrap); push_keep(m, r.z << 16, wrap);
  push_keep(m, r.y, wrap); push_keep(m, r.y << 16, wrap);
  push_keep(m, r.x, wrap); push_keep(m, r.x << 16, wrap);
}
// keep-mask bits (bit j set = keep element 8 * group + j); thr16 > 0
__host__ __device__ __forceinline__ uint32_t dropout_keep8(uint64_t seed, uint32_t stream, uint64_t group, uint32_t thr16) {
  uint32_t m = 0;
  push_keep8(m, seed, stream, group, 0u - (thr16 << 16));
  return m;
}
// the same for four groups in a row
__device__ __forceinline__ uint32_t dropout_keep32(uint64_t seed, uint32_t stream, uint64_t group, uint32_t thr16) {
  uint32_t m = 0;
#pragma unroll
  for (int k = 3; k >= 0; --k) push_keep8(m, seed, stream, group + k, 0u - (thr16 << 16));
  return m;
}

// Host helper: encode a 2-D row-major tensor (rows x cols, `ld` elements
// between rows) for TMA with a (box_cols x box_rows) tile and 128B swizzle.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_tiled();
// Returns 0 on success.
int make_tmap_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                 uint32_t box_rows, uint32_t box_cols, int elem_bytes, bool swizzle128);
// Same with an explicit swizzle span in bytes (0, 32, 64 or 128).
int make_tmap_2d_sw(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                    uint32_t box_rows, uint32_t box_cols, int elem_bytes, int swizzle_bytes);

}  // namespace ab
