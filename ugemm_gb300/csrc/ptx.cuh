// ptx.cuh -- inline-PTX building blocks for sm_103a kernels: mbarriers,
// TMA (cp.async.bulk.tensor), tcgen05 (TMEM alloc, UMMA, commit, ld) and
// bounded waits.  Every wait on an mbarrier gives up after a time limit,
// records an error code in a device flag and lets the kernel wind down, so a
// logic error never leaves a spinning kernel on the GPU.
#pragma once

#include <cuda.h>
#include <cstdint>

namespace ugemm {

// Error codes written to the device error word (first writer wins).
enum DeviceError : int {
  kDevOk = 0,
  kDevTimeoutFull = 1,    // consumer gave up waiting for a TMA stage
  kDevTimeoutEmpty = 2,   // producer gave up waiting for a free stage
  kDevTimeoutAccum = 3,   // epilogue gave up waiting for the accumulator
  kDevBadConfig = 4,
};

// Wall-clock limit of one wait, in nanoseconds.  Real waits last
// microseconds; 2 s only trips on a broken pipeline.
constexpr uint64_t kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void record_error(int* err, int code) {
  if (err) atomicCAS(err, 0, code);
}

__device__ __forceinline__ bool error_raised(const int* err) {
  return err && *reinterpret_cast<const volatile int*>(err) != 0;
}

// Registers handed back by, or granted to, every thread of a warpgroup
// (all four warps execute it).  The warpgroups' shares of a kernel must add
// up to no more than threads x registers at its launch, or the grant waits
// for ever.
template <int kRegs>
__device__ __forceinline__ void setmaxnreg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}
template <int kRegs>
__device__ __forceinline__ void setmaxnreg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Non-blocking test of the same (mbarrier.test_wait never suspends).
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for the phase with the given parity to complete.  Returns false (and
// records `code`) if the wait exceeded kWaitLimitNs or another thread of the
// grid already recorded an error.
// (The limit is a template parameter only so that the failure self-test can
// exercise this same loop with a short limit.)
template <uint64_t kLimitNs = kWaitLimitNs>
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 255u) == 0) {
      if (error_raised(err)) return false;
      if (globaltimer() - t0 > kLimitNs) {
        record_error(err, code);
        return false;
      }
    }
  }
  return true;
}

// -------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// im2col mode on a {channels, W, H, images} tensor: the map's pixels-per-column
// consecutive output pixels from base pixel (w, h, n) on, each read at the
// offset (ow, oh) from its base -- a kernel tap -- with zeros outside the image.
__device__ __forceinline__ void tma_load_im2col(void* dst, const CUtensorMap* map, uint64_t* bar,
                                                int c, int w, int h, int n, int ow, int oh) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c), "r"(w), "r"(h), "r"(n),
      "h"(static_cast<uint16_t>(ow)), "h"(static_cast<uint16_t>(oh))
      : "memory");
}

// ---------------------------------------------------------------- tcgen05
// TMEM allocation: executed by one whole warp; writes the TMEM base address
// to shared memory.  `ncols` is a power of two >= 32.
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

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory matrix descriptor for tcgen05.mma (K-major operand).
//   bits  0-13 start address >> 4
//   bits 16-29 leading-dimension byte offset >> 4 (unused for swizzled K-major;
//              MN-major: distance between blocks of one swizzle width of rows)
//   bits 32-45 stride-dimension byte offset >> 4 (distance between 8-row
//              groups; MN-major: between groups of 8 k)
//   bits 46-48 fixed 0b001
//   bits 61-63 swizzle: 0 none, 2 128B, 4 64B, 6 32B
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t saddr, uint32_t sbo_bytes,
                                                   uint32_t swizzle_code,
                                                   uint32_t lbo_bytes = 16) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes & 0x3FFFFu) >> 4) << 16;
  d |= static_cast<uint64_t>((sbo_bytes & 0x3FFFFu) >> 4) << 32;
  d |= static_cast<uint64_t>(1u) << 46;
  d |= static_cast<uint64_t>(swizzle_code & 7u) << 61;
  return d;
}

// Operands MN-major instead of K-major (16-bit types), added to a descriptor.
constexpr uint32_t kUmmaMnMajor = (1u << 15) | (1u << 16);
// Instruction descriptor, kind::f16 / kind::tf32 with FP32 accumulation,
// both operands K-major.  a_fmt/b_fmt: 0 F16, 1 BF16, 2 TF32.
__host__ __device__ constexpr uint32_t umma_idesc(uint32_t a_fmt, uint32_t b_fmt, uint32_t m,
                                                  uint32_t n) {
  return (1u << 4)              // D format F32
         | (a_fmt << 7) | (b_fmt << 10)
         | ((n >> 3) << 17)     // N / 8
         | ((m >> 4) << 24);    // M / 16
}

// Descriptors come as their two words: the upper one is the same for a whole
// launch, and the lower one is a 32-bit sum.  A converged warp executes the call;
// the lane whose `issue` is set issues the MMA (a predicate, not a branch: in a
// branch of one lane the compiler keeps the operands in vector registers).
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint32_t alo, uint32_t ahi,
                                          uint32_t blo, uint32_t bhi, uint32_t idesc,
                                          uint32_t accumulate, uint32_t issue) {
  asm volatile(
      "{\n"
      ".reg .pred p, i;\n"
      ".reg .b64 a, b;\n"
      "mov.b64 a, {%1, %2};\n"
      "mov.b64 b, {%3, %4};\n"
      "setp.ne.b32 p, %6, 0;\n"
      "setp.ne.b32 i, %7, 0;\n"
      "@i tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate), "r"(issue)
      : "memory");
}

__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint32_t alo, uint32_t ahi,
                                          uint32_t blo, uint32_t bhi, uint32_t idesc,
                                          uint32_t accumulate, uint32_t issue) {
  asm volatile(
      "{\n"
      ".reg .pred p, i;\n"
      ".reg .b64 a, b;\n"
      "mov.b64 a, {%1, %2};\n"
      "mov.b64 b, {%3, %4};\n"
      "setp.ne.b32 p, %6, 0;\n"
      "setp.ne.b32 i, %7, 0;\n"
      "@i tcgen05.mma.cta_group::1.kind::tf32 [%0], a, b, %5, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate), "r"(issue)
      : "memory");
}

// Non-zero in one lane of a converged warp, the same one every time.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok));
  return ok;
}

// Arrive on an mbarrier once all tcgen05 operations issued so far by this
// thread have completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t receives lane (base+t).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
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

// 32 lanes x 16 consecutive 32-bit columns (half the registers of x32).
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

__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace ugemm
