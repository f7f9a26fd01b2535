// tcgen.cuh - the tcgen05 / mbarrier / TMA instructions that the tensor-core kernels are written with.
#pragma once

#include "moe_internal.cuh"

// a number as a type (a pass of a block, a column offset)
template <int V> struct PassC { static constexpr int value = V; };

__device__ __forceinline__ uint32_t tc_s32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned long long tc_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// shared-memory matrix descriptor, K-major, no swizzle: 8x16 B core matrices,
// lbo = bytes between the two 16-byte K chunks of one MMA, sbo = bytes between
// 8-row groups
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3fff) | ((uint64_t)((lbo >> 4) & 0x3fff) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3fff) << 32) | (1ull << 46);
}
// D[tmem_c] (+)= A[tmem_a] * B[db]: A from tensor memory (row = lane, 32-bit column c =
// K values 4c..4c+3), B from shared memory
__device__ __forceinline__ void tc_mma_i8_ta(uint32_t tmem_c, uint32_t tmem_a, uint64_t db, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_c),
      "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_mma_f16(uint32_t tmem_c, uint64_t da, uint64_t db, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_c),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One lane of a converged warp. The products are issued under this predicate and not under
// "lane == 0": the compiler knows it to be one thread, keeps descriptors and addresses in uniform
// registers and issues a product every 10-12 cycles; under a lane comparison every product first
// moved its six operands across, 48 cycles whatever N is (measured: N = 16 50 -> 12, N = 64 50 -> 34,
// N = 128 66 -> 66 cycles a K step).
__device__ __forceinline__ bool tc_elect() {
  uint32_t p;
  asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.u32 %0, 1, 0, P;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   tc_s32(bar))
               : "memory");
}
// (OFF: a constant column offset on top of a warp-uniform address: the address stays in one uniform register)
template <int OFF> __device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t r[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8 + %9];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr), "n"(OFF));
}
template <int OFF> __device__ __forceinline__ void tc_ld4(uint32_t taddr, uint32_t r[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4 + %5];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr), "n"(OFF));
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t r[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t r[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
      "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
      "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tc_mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_s32(bar)), "r"(count));
}
__device__ __forceinline__ void tc_mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_s32(bar)) : "memory");
}
// The arrival that hands a place of a ring back after words were read from it. `used` is made of every load's words
// and goes into the address (times `zero`, which is 0 at run time and unknown to the compiler): the arrival cannot be
// issued before the loads have returned, wherever the arithmetic on them is scheduled. (One lane's words stand for
// the warp's where all lanes read the same address: one load instruction.)
__device__ __forceinline__ void tc_mbar_arrive_used(uint64_t *bar, uint32_t used, uint32_t zero) {
  asm volatile(
      "{\n .reg .b32 a;\n and.b32 a, %1, %2;\n add.u32 a, a, %0;\n mbarrier.arrive.shared::cta.b64 _, [a];\n}\n" ::"r"(tc_s32(bar)),
      "r"(used), "r"(zero)
      : "memory");
}
__device__ __forceinline__ void tc_mbar_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc_s32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool tc_bar_test(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(tc_s32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool tc_bar_sleep(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(tc_s32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// A bounded wait on a phase of an mbarrier. False after the wait limit (or soon after an error is recorded):
// the caller carries on with whatever the accumulators hold and the call reports the error. (All inline: a
// call in the slow path makes the compiler keep the workers' registers out of its way everywhere.)
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, int *err, unsigned long long wait_ns) {
  if (tc_bar_test(bar, parity)) return true;
  unsigned long long t0 = 0;
  for (;;) {
    // (sleeps in hardware for a while: two waiting warps that polled took a fifth of the issue slots)
    if (tc_bar_sleep(bar, parity)) return true;
    const unsigned long long t = tc_now();
    if (t0 == 0) t0 = t;
    if (*(volatile int *)err != 0 || t - t0 > wait_ns) break;
  }
  atomicCAS(err, 0, 7);
  return false;
}
// A copy still in flight lands in whatever the SM's shared memory holds next: before a CTA ends - also when a wait ran
// out and it gives up - its last copies are waited for, with a limit that is not the call's (a copy takes microseconds).
#define TC_LANDED_NS 100000000ull
__device__ __forceinline__ void tc_landed(uint64_t *bar, uint32_t parity) {
  const unsigned long long t0 = tc_now();
  while (!tc_bar_test(bar, parity) && tc_now() - t0 < TC_LANDED_NS) {
  }
}
// Two f32 in one register pair. A product whose rounded value goes into an addition is written as
// fma(a, b, -0) with a -0 that the compiler cannot see (a kernel parameter): it contracts a plain
// mul.rn.f32x2 and the add.rn.f32x2 behind it into one fma, which has other bits than the reference's
// separately rounded steps (adding -0 changes no product, signed zeros included).
__device__ __forceinline__ uint64_t tc_pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void tc_unpack2(uint64_t v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t tc_mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t tc_add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t tc_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// eight bytes at any address as the two aligned words that hold them, put together only where they are used: shifted
// right behind the loads they made the warp wait for memory there (650 of an iteration's 1,900 cycles)
struct TcBytes8 {
  unsigned long long a, b;
  int sh;
  __device__ __forceinline__ void load(const uint8_t *p) {
    const unsigned long long *q = (const unsigned long long *)((uintptr_t)p & ~(uintptr_t)7);
    sh = 8 * (int)((uintptr_t)p & 7);
    a = __ldg(q);
    b = __ldg(q + 1);
  }
  __device__ __forceinline__ unsigned long long get() const { return sh ? (a >> sh) | (b << (64 - sh)) : a; }
};
__device__ __forceinline__ void tc_tma3(uint32_t dst, const CUtensorMap *m, int x, int y, int z, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(m), "r"(x), "r"(y), "r"(z), "r"(tc_s32(bar))
      : "memory");
}
