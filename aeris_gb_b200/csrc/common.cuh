// Shared device-side primitives for the sm_100a kernels: mbarrier, TMA (cp.async.bulk.tensor),
// tcgen05 (TMEM alloc, MMA, commit, ld) and UMMA descriptor construction.
//
// Every wait in this file is bounded: a spin that exceeds its time limit records an error code
// in a global status word and returns false, so the kernel can free its TMEM and return instead
// of hanging the GPU.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef AERIS_WAIT_TIMEOUT_NS
#define AERIS_WAIT_TIMEOUT_NS 2000000000ull  // 2 s per wait, far above any legitimate tile time
#endif

namespace aeris {

// Error codes written to the status word (0 = ok).
enum : int {
  ERR_NONE = 0,
  ERR_TIMEOUT_FULL = 1,
  ERR_TIMEOUT_EMPTY = 2,
  ERR_TIMEOUT_TMEM_FULL = 3,
  ERR_TIMEOUT_TMEM_EMPTY = 4,
  ERR_TIMEOUT_SIGNAL = 5,
  ERR_BOUNDS = 6,
  ERR_TIMEOUT_ATTN = 7,
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool elect_one_sync() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t"
      ".reg .pred P1;\n\t"
      "elect.sync _|P1, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait. Returns false (and records `code`) when the time limit passes. The first try (which suspends the thread in
// hardware for a while) is the whole wait nearly always; the loop with its timer lives out of line, because inlined it
// costs every wait a dozen instructions and branches of which none is needed.
static __device__ __noinline__ bool mbar_wait_slow(uint64_t* bar, uint32_t parity, int* status, int code) {
#pragma unroll 1
  for (int i = 0; i < 128; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (globaltimer_ns() - t0 > AERIS_WAIT_TIMEOUT_NS) {
      if (status) atomicCAS(status, 0, code);
      return false;
    }
    if (status && *reinterpret_cast<volatile int*>(status) != 0) return false;  // someone else gave up
  }
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, status, code);
}
// Waits of a warp that stays together: every lane asks, the votes keep it one, and the loop is in line. Against mbar_wait,
// whose second try is behind a call, a hand-over that has to be waited for takes 103 instead of 287 cycles (two warps that
// hand one back and forth), and a kernel without calls can split its registers between warpgroups. A try that fails suspends
// the warp for 1.3 us (measured), so the limit is about as long as the other waits' 2 s.
constexpr int MBAR_TRIES = 1500000;
__device__ __forceinline__ bool mbar_try_wait_at(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, int* status, int code) {
#pragma unroll 1
  for (int i = 0; i < MBAR_TRIES; ++i)
    if (__all_sync(0xffffffffu, mbar_try_wait_at(bar, parity))) return true;
  if (status) atomicCAS(status, 0, code);
  return false;
}
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, int* status, int code) {
  return mbar_wait_warp(smem_u32(bar), parity, status, code);
}
// Two barriers in one step: a wait that is over costs 110-200 cycles of latency once for both. Each of the two tries may
// suspend the warp, hence half the steps.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, int* status, int code) {
#pragma unroll 1
  for (int i = 0; i < MBAR_TRIES / 2; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
        "and.pred p, p, q;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(b0), "r"(p0), "r"(b1), "r"(p1)
        : "memory");
    if (__all_sync(0xffffffffu, ok != 0)) return true;
  }
  if (status) atomicCAS(status, 0, code);
  return false;
}
// Non-suspending poll (mbarrier.test_wait) with the same time limit: the waiting thread never yields its issue slot,
// which suits single elected threads that wait on barriers signalled from another CTA of the cluster.
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_poll(uint64_t* bar, uint32_t parity, int* status, int code) {
  const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 512; ++i)
      if (mbar_test_wait(bar, parity)) return true;
    if (globaltimer_ns() - t0 > AERIS_WAIT_TIMEOUT_NS) {
      if (status) atomicCAS(status, 0, code);
      return false;
    }
    if (status && *reinterpret_cast<volatile int*>(status) != 0) return false;
  }
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---------------------------------------------------------------- TMA
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 2D tiled load, no multicast. c0 = innermost coordinate (elements), c1 = row.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// Tiled store of a shared-memory tile as a bulk group of its own. What lies outside the tensor is not written.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* smem_src, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];\n\t"
      "cp.async.bulk.commit_group;" ::"l"(reinterpret_cast<uint64_t>(m)),
      "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* smem_src, int c0, int c1) {   // no group yet
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(c0), "r"(c1)
               : "memory");
}

// ---------------------------------------------------------------- tcgen05 / TMEM
// Chained launches. A kernel launched by launch_chained may start while the one before it in the stream still runs, once
// every CTA of that one has passed its chain_point (or left): its launch, its barriers and its TMEM allocation then cost
// nothing. chain_point returns when everything before this grid in the stream has completed and is visible. Two rules keep
// this sound: every thread passes it before it touches global memory, early exits included (the kernel after next waits for
// this one alone), and a kernel passes it after its TMEM allocation (a waiting CTA may hold what an older one would need).
// Kernels that wait for other GPUs are launched without it. us per launch, back to back, plain / chained: two-CTA product
// 256 x 256 x 256 10.3 / 7.6, 14400 x 768 x 768 21.1 / 18.5; a sampler step of seven evaluations of two blocks of width 256
// on 14,400 tokens (155 launches) 2.24 / 1.95 ms. Chained products and attention alone: 2.06.
// The modulation vectors' small products and the loss too: training steps of 209 and 217 launches 3.85 / 3.82, 2.90 / 2.89.
__device__ __forceinline__ void chain_point() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Whether a kernel gave up.
__device__ __forceinline__ bool failed(const int* status) {
  return status && *reinterpret_cast<const volatile int*>(status) != 0;
}
// A kernel may look at the status word before its chain_point (or set it, where its shared memory is misplaced) and leave at
// once: the one exception to the first rule. What it sees there are kernels that have ended, not the one in front, which may
// still be running. Behind chain_point every warp that writes results asks again, and keeps them to itself where the kernel
// in front has given up (what it read of that one is incomplete; scratch for a kernel behind, which asks as well, is
// written). `slot` is the warp's own word of shared memory: nothing is held in registers, and the read's 0.3 us pass while the
// first operands are on their way. A sampler step of seven evaluations of two blocks of width 256 on 14,400 tokens 1,733 ->
// 1,738 us; one decision for the whole CTA behind chain_point is on the way of every kernel (1,755) and spilled registers of
// the attention kernels, a look at `slot` for every row of delta took 3 % of the backward pass. (The two-CTA products do not
// ask.)
__device__ __forceinline__ void note_failure(const int* status, int* slot) {
  if ((threadIdx.x & 31) == 0) *reinterpret_cast<volatile int*>(slot) = failed(status);
}
__device__ __forceinline__ bool noted(const int* slot) { return *reinterpret_cast<const volatile int*>(slot) != 0; }
// The result is the launch's only trace: it has taken the error from the runtime.
template <typename... P, typename... A>
[[nodiscard]] static inline int launch_chained(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                                               A&&... args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Arrive on an mbarrier once every tcgen05 op issued so far by this thread has completed.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]; bf16 inputs, fp32 accumulate.
__device__ __forceinline__ void umma_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Products and commits of a warp that stays together: the lane with `lead` set issues them, and what they are made of can
// live in uniform registers. A loop of two waits, eight products and two commits: 251 cycles, by a single thread 304.
__device__ __forceinline__ void umma_ss_warp(uint32_t lead, uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, e;\n\t"
      "setp.ne.b32 e, %5, 0;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
      : "memory");
}
__device__ __forceinline__ void umma_ts_warp(uint32_t lead, uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, e;\n\t"
      "setp.ne.b32 e, %5, 0;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
      : "memory");
}
// Four steps of 16 at a time: the operands' low words advance by A_STEP and B_STEP (tensor memory: words), `acc` is the
// first step's. Fewer instructions than four calls.
template <int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_ss4_warp(uint32_t lead, uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                              uint32_t acc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, e;\n\t"
      ".reg .b32 a, b;\n\t"
      ".reg .b64 x, y;\n\t"
      "setp.ne.b32 e, %5, 0;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 x, {%1, %6};\n\t"
      "mov.b64 y, {%2, %6};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, p;\n\t"
      "add.u32 a, %1, %7;\n\t"
      "add.u32 b, %2, %8;\n\t"
      "mov.b64 x, {a, %6};\n\t"
      "mov.b64 y, {b, %6};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, 1;\n\t"
      "add.u32 a, a, %7;\n\t"
      "add.u32 b, b, %8;\n\t"
      "mov.b64 x, {a, %6};\n\t"
      "mov.b64 y, {b, %6};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, 1;\n\t"
      "add.u32 a, a, %7;\n\t"
      "add.u32 b, b, %8;\n\t"
      "mov.b64 x, {a, %6};\n\t"
      "mov.b64 y, {b, %6};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, 1;\n\t"
      "}\n" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(acc), "r"(lead), "r"((1024u >> 4) | (1u << 14) | (2u << 29)), "n"(A_STEP),
      "n"(B_STEP)
      : "memory");
}
template <int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_ts4_warp(uint32_t lead, uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc,
                                              uint32_t acc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, e;\n\t"
      ".reg .b32 a, b;\n\t"
      ".reg .b64 y;\n\t"
      "setp.ne.b32 e, %5, 0;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 y, {%2, %6};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], y, %3, p;\n\t"
      "add.u32 a, %1, %7;\n\t"
      "add.u32 b, %2, %8;\n\t"
      "mov.b64 y, {b, %6};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], y, %3, 1;\n\t"
      "add.u32 a, a, %7;\n\t"
      "add.u32 b, b, %8;\n\t"
      "mov.b64 y, {b, %6};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], y, %3, 1;\n\t"
      "add.u32 a, a, %7;\n\t"
      "add.u32 b, b, %8;\n\t"
      "mov.b64 y, {b, %6};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], y, %3, 1;\n\t"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "r"(b_lo), "r"(idesc), "r"(acc), "r"(lead), "r"((1024u >> 4) | (1u << 14) | (2u << 29)), "n"(A_STEP),
      "n"(B_STEP)
      : "memory");
}
__device__ __forceinline__ void tc_commit_warp(uint32_t lead, uint32_t bar) {
  asm volatile(
      "{\n\t"
      ".reg .pred e;\n\t"
      "setp.ne.b32 e, %1, 0;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
      "}\n" ::"r"(bar),
      "r"(lead)
      : "memory");
}
// Registers per thread of the warpgroup that executes this; a kernel's shares may add up to what it was launched with.
template <int N> __device__ __forceinline__ void regs_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N> __device__ __forceinline__ void regs_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

// 32 lanes x 32 columns of fp32: thread i of the warp gets row (lane base + i), 32 consecutive columns.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------- UMMA descriptors
// Shared-memory matrix descriptor, 128-byte swizzle, sm_100 version field set.
//   K-major operand  (rows of 64 bf16 = 128 B, 8-row swizzle atoms): SBO = bytes between 8-row groups (1024
//                     when rows are packed); LBO unused.
//   MN-major operand (k-rows of 64 MN-elements = 128 B): SBO = bytes between groups of 8 k-rows (1024),
//                     LBO = bytes between consecutive 64-element MN chunks.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= static_cast<uint64_t>(1) << 46;  // descriptor version for sm_100
  d |= static_cast<uint64_t>(2) << 61;  // SWIZZLE_128B
  return d;
}
// The same in two halves. The low word (address, leading offset) advances by bytes / 16; the high one is that of every
// 128-byte swizzled tile whose groups of eight rows are 1024 bytes apart.
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr & 0x3FFFF) >> 4) | ((lbo_bytes >> 4) << 16);
}
__device__ __forceinline__ uint64_t smem_desc(uint32_t lo) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"((1024u >> 4) | (1u << 14) | (2u << 29)));
  return d;
}
// Instruction descriptor for kind::f16 with bf16 inputs and fp32 accumulation.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, int a_mn_major, int b_mn_major) {
  return (1u << 4)                              // D format: f32
         | (1u << 7)                            // A format: bf16
         | (1u << 10)                           // B format: bf16
         | (static_cast<uint32_t>(a_mn_major) << 15) | (static_cast<uint32_t>(b_mn_major) << 16) |
         (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}

// Two fp32 lanes per instruction (Blackwell `*.f32x2`): the same arithmetic rate as scalar fp32, half the issue slots.
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// bf16 pair -> fp32 pair (exact): the low element is the word shifted up, the high one the word with its low half cleared.
__device__ __forceinline__ uint64_t f2_from_bf16x2(uint32_t u) {
  return f2_pack(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
__device__ __forceinline__ uint32_t f2_to_bf16x2(uint64_t v) {
  float lo, hi;
  f2_unpack(v, lo, hi);
  return pack_bf16x2(lo, hi);
}

}  // namespace aeris
