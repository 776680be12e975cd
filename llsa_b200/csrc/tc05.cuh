// Thin wrappers over the Blackwell tensor-core path: tcgen05.mma with operands in
// shared memory (128-byte swizzled tiles) and accumulators in tensor memory (TMEM),
// mbarrier completion, and TMEM loads for the epilogue.
//
// Shared-memory tile format used everywhere here: rows of 64 bf16 (128 bytes), row r at
// r * 128 bytes from a 1024-byte aligned base, its 16-byte chunk c stored at chunk
// c ^ (r & 7) -- the SWIZZLE_128B canonical layout.  One such tile serves as
//   * a K-major operand  (rows = M or N index, the 64 channels = K), and
//   * an MN-major operand (rows = K index, the 64 channels = the M/N index),
// so the same copy of a key tile feeds both S = Q.K^T and dQ = dS.K, and the same copy of
// a Q / dO tile feeds S and dK = dS^T.Q.
//
// Every wait on an mbarrier is bounded; on expiry the caller records an error status and
// falls through (results are then garbage but the kernel ends and frees its TMEM).
#pragma once
#include "common.cuh"

namespace llsa {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t) __cvta_generic_to_shared(p); }

// ---- TMEM allocation (one full warp executes these) ----
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---- mbarrier ----
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
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
// One look, no suspension
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
// ---- bounded waits of the warp-specialised kernels -------------------------------------------------
// One WaitCtl per CTA (shared memory).  A wait polls at most `limit` times; the first wait that runs out raises
// `abort`, which every other wait of the CTA notices within a thousand polls, so all roles leave their loops, the
// kernel ORs LLSA_DEV_WAIT_EXPIRED into the caller's status word, lets what it still has in flight finish
// (abort_drain), frees its tensor memory and returns normally: the context stays usable and the host can tell.
struct WaitCtl {
  int abort;
  int limit;
};
constexpr int kWaitPolls = 400000;
__device__ __forceinline__ bool bounded_wait(uint64_t* bar, uint32_t parity, volatile WaitCtl* c) {
  if (mbar_test(bar, parity)) return true;            // the first of the `limit` polls: a try_wait may suspend the thread for a while
  const int limit = c->limit;
  for (int i = 1; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 1023) == 1023 && c->abort) return false;
  }
  c->abort = 1;
  return false;
}
// The same by a whole warp in step: lane l waits for bars[l]'s phase (several barriers at the price of one: the test is one instruction
// whatever addresses its lanes bring), and the answer is the same in every lane, which keeps the control flow around it uniform.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile WaitCtl* c) {
  if (__all_sync(0xffffffffu, mbar_test(bar, parity))) return true;
  const int limit = c->limit;
  for (int i = 1; i < limit; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((i & 1023) == 1023 && __any_sync(0xffffffffu, c->abort != 0)) return false;
  }
  c->abort = 1;
  return false;
}
// After an abort: a fixed, bounded pause (about 60 microseconds) in which bulk copies and tensor-core instructions
// this CTA has already issued complete, before its shared and tensor memory are given back.
__device__ __forceinline__ void abort_drain() {
  for (int i = 0; i < 64; ++i) __nanosleep(1000);
}

// ---- register split of a warp-specialised kernel: a warpgroup (all of it, once) gives back registers or takes more than the LAUNCH it was
// launched with.  All the warpgroups' shares together stay within threads x LAUNCH, or the takers wait for good; an increase to fewer
// registers than a warp has, or a decrease to more, is an illegal instruction.
template <int N, int LAUNCH>
__device__ __forceinline__ void regs_set() {
  static_assert(N % 8 == 0 && N >= 24 && N <= 256, "what setmaxnreg takes");
  if constexpr (N < LAUNCH) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
  else if constexpr (N > LAUNCH) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

// ---- fences ----
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- descriptors ----
// Shared-memory matrix descriptor, SWIZZLE_128B (layout type 2), descriptor version 1 (sm_100).
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t) ((saddr >> 4) & 0x3FFF);
  d |= (uint64_t) ((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t) ((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t) 1 << 46;
  d |= (uint64_t) 2 << 61;
  return d;
}
// Instruction descriptor: bf16 x bf16 -> fp32, dense; a_mn / b_mn = 1 for an MN-major operand.
__host__ __device__ constexpr uint32_t instr_desc(int M, int N, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) a_mn << 15) | ((uint32_t) b_mn << 16) | ((uint32_t) (N >> 3) << 17) |
         ((uint32_t) (M >> 4) << 24);
}

// ---- issue by a warp in step: every lane executes the statement, elect.sync picks the lane that issues.  tcgen05.mma takes its
// descriptors from uniform registers and is issued once per executing thread; where the compiler sees an elected thread in uniform control
// flow the descriptors stay there, where it sees `if (lane == 0)` every instruction costs some 98 cycles of moves, whatever its size, and
// issuing, not the tensor pipe, is the pace of a kernel whose products have N = 64.
// One statement issues four k-steps, 16 elements of K each.
// A, B in shared memory; AS / BS: descriptor units (16 bytes) per k-step, 2 for a K-major operand (32 bytes inside the swizzled row), 128
// for an MN-major one (16 rows).  D (+)= A . B, K = 64; `accumulate` is for the first k-step
template <int AS = 2, int BS = 2>
__device__ __forceinline__ void umma_ss_k64(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                            uint32_t accumulate = 0) {
  asm volatile(
      "{\n\t.reg .pred f, t, e;\n\t.reg .b32 al, bl;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 f, %7, 0; setp.eq.b32 t, %6, 0;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "add.u32 al, %1, 0; add.u32 bl, %3, 0;\n\t"
      "mov.b64 da, {al, %2}; mov.b64 db, {bl, %4};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, {%6, %6, %6, %6}, f;\n\t"
      "add.u32 al, %1, %8; add.u32 bl, %3, %9;\n\t"
      "mov.b64 da, {al, %2}; mov.b64 db, {bl, %4};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, %10; add.u32 bl, %3, %11;\n\t"
      "mov.b64 da, {al, %2}; mov.b64 db, {bl, %4};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, %12; add.u32 bl, %3, %13;\n\t"
      "mov.b64 da, {al, %2}; mov.b64 db, {bl, %4};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, {%6, %6, %6, %6}, t;\n\t"
      "}"
      :
      : "r"(tmem_d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(0u), "r"(accumulate), "n"(AS), "n"(BS), "n"(2 * AS),
        "n"(2 * BS), "n"(3 * AS), "n"(3 * BS)
      : "memory");
}
// A in tensor memory (two K values per column), B in shared memory and MN-major (16 rows of 128 bytes per k-step): D (+)= A . B, K = 32, 64
// or 128; `accumulate` is for the first k-step
__device__ __forceinline__ void umma_ts_k32(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, t, e;\n\t.reg .b32 al, bl;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 p, %5, 0; setp.eq.b32 t, %6, 0;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "add.u32 al, %1, 0; add.u32 bl, %2, 0;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, p;\n\t"
      "add.u32 al, %1, 8; add.u32 bl, %2, 128;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "}"
      :
      : "r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void umma_ts_k64(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, t, e;\n\t.reg .b32 al, bl;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 p, %5, 0; setp.eq.b32 t, %6, 0;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "add.u32 al, %1, 0; add.u32 bl, %2, 0;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, p;\n\t"
      "add.u32 al, %1, 8; add.u32 bl, %2, 128;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, 16; add.u32 bl, %2, 256;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, 24; add.u32 bl, %2, 384;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "}"
      :
      : "r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void umma_ts_k128(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, t, e;\n\t.reg .b32 al, bl;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 p, %5, 0; setp.eq.b32 t, %6, 0;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "add.u32 al, %1, 0; add.u32 bl, %2, 0;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, p;\n\t"
      "add.u32 al, %1, 8; add.u32 bl, %2, 128;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, 16; add.u32 bl, %2, 256;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, 24; add.u32 bl, %2, 384;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, 32; add.u32 bl, %2, 512;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, 40; add.u32 bl, %2, 640;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, 48; add.u32 bl, %2, 768;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "add.u32 al, %1, 56; add.u32 bl, %2, 896;\n\t"
      "mov.b64 db, {bl, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [al], db, %4, {%6, %6, %6, %6}, t;\n\t"
      "}"
      :
      : "r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void umma_commit_w(uint64_t* bar) {
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
               "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
// ---- TMEM -> registers: lane (32 * (warp % 4) + lane id) gets 32 consecutive fp32 columns ----
// Asynchronous: the registers may be read only after tmem_ld_wait(v) (which ties them to the wait).
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, float (&v)[32]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait(float (&v)[32]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                 "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                 "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}
// 16 consecutive columns: half the registers of tmem_ld32 in flight
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// registers -> TMEM: lane (32 * (warp % 4) + lane id) writes 16 consecutive 32-bit columns
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 128-bit store to shared memory at (addr ^ XOR_BYTES): with addr = the swizzled start of a 128-byte row, XOR_BYTES = 16 * chunk
// walks the row's chunks in swizzled order from ONE register (the address arithmetic stays inside the statement, so the
// compiler cannot hoist eight precomputed addresses out of a loop and spill them).
template <int XOR_BYTES>
__device__ __forceinline__ void sts128_xor(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("{\n\t.reg .b32 t;\n\txor.b32 t, %0, %1;\n\tst.shared.v4.b32 [t], {%2, %3, %4, %5};\n\t}"
               :
               : "r"(addr), "n"(XOR_BYTES), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}

// ---- swizzled tile addressing (elements) ----
__device__ __forceinline__ int swz(int r, int chunk) { return r * 64 + ((chunk ^ (r & 7)) << 3); }

}  // namespace tc
}  // namespace llsa
