// Inline-PTX wrappers for sm_100a: mbarrier, TMA tiled copies, tcgen05 (alloc, mma,
// commit, ld/st), proxy fences, and the UMMA descriptor encodings.  Every wait is
// bounded: when its limit runs out it raises the CTA-wide abort flag and returns, and the
// end of the kernel records its code in the caller's status word, so a broken pipeline ends
// instead of hanging the GPU.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace evo {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// The primitives on 32-bit shared-window addresses (smem_u32 of the barrier, computed once): no
// generic-pointer arithmetic or address-space conversion per call.
__device__ __forceinline__ void mbar_init_s(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_s(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_s(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bounded wait on an mbarrier (32-bit shared-window addresses; about one second at B200 clocks).  `abort_flag_s`
// is a word of shared memory that belongs to the CTA: once any wait has run out it holds that wait's code, all
// later waits fall through, and the end of the kernel reports it (end_of_cta).  The retries carry a
// suspend-time hint: the hardware parks the thread until the phase completes, so a waiting warp does not
// compete for issue slots with the warps that do the arithmetic.  All of it is one short sequence on purpose: a
// kernel has some thirty waits, and the code of its loops has to fit the instruction caches.
constexpr uint32_t kWaitLimitCycles = 2000000000u;
__device__ __forceinline__ void mbar_wait_s(uint32_t bar, uint32_t parity, uint32_t abort_flag_s, int code) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .u32 t0, t1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%0], %1;\n\t"
      "@p bra EVO_W_DONE;\n\t"
      "mov.u32 t0, %%clock;\n"
      "EVO_W_AGAIN:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%0], %1, 1000000;\n\t"
      "@p bra EVO_W_DONE;\n\t"
      "ld.volatile.shared.u32 t1, [%2];\n\t"
      "setp.ne.u32 p, t1, 0;\n\t"
      "@p bra EVO_W_DONE;\n\t"
      "mov.u32 t1, %%clock;\n\t"
      "sub.u32 t1, t1, t0;\n\t"
      "setp.lt.u32 p, t1, %4;\n\t"
      "@p bra EVO_W_AGAIN;\n\t"
      "st.volatile.shared.u32 [%2], %3;\n"
      "EVO_W_DONE:\n\t}"
      ::"r"(bar), "r"(parity), "r"(abort_flag_s), "r"(code), "n"(kWaitLimitCycles)
      : "memory");
}
// What every thread of a CTA does at the end if a wait has run out: the status word gets the code of that wait,
// and copies that may still be in flight get time to land before the CTA retires.
static __device__ __noinline__ void report_abort(int code, int* status) {
  if (threadIdx.x == 0 && status) atomicCAS(status, 0, code);
  const long long t0 = clock64();
  while (clock64() - t0 < 200000) {}
}

// Generic-proxy writes to shared memory -> visible to the async proxy (TMA, tcgen05.mma).
__device__ __forceinline__ void fence_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---------------------------------------------------------------- TMA (tiled, no multicast)
__device__ __forceinline__ void tma_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Wait until the bulk groups of this thread have finished READING their shared-memory source.
__device__ __forceinline__ void tma_wait_group_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_wait_group_read1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }  // (all but the last)
// Wait until the bulk groups of this thread have completed entirely.
__device__ __forceinline__ void tma_wait_group0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---------------------------------------------------------------- tcgen05: TMEM management
// Whole-warp instructions (.sync.aligned): call with all 32 lanes converged.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot_in_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_in_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// The end of a CTA, for all of its threads; what it still owns (tensor memory) is freed after this.  The flag is
// looked at behind the barrier, when every warp is through with its waits: the thread that reports belongs to a warp
// that may be done long before the last of them, and a wait that ran out after that would go unreported.
__device__ __forceinline__ void end_of_cta(volatile int* abort_flag, int* status) {
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) report_abort(*abort_flag, status);
}

// ---------------------------------------------------------------- tcgen05: MMA
// One lane of a converged warp.  Every operand of a tcgen05.mma lives in a uniform register: in a branch that one
// lane takes (lane == 0) the compiler has to move each of them there, and the waits of that branch are slow too.
// With the whole warp walking the issue loop on warp-uniform values and only the instruction itself under this
// predicate, a hand-over of four MMAs with A in tensor memory, two with A in shared memory, three commits and
// the wait for them took 376 cycles next to 16 busy warps, against 830 from a single-lane branch.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e;
}
// The MMAs of a converged warp, issued by its elected lane.
__device__ __forceinline__ void mma_ss_e(uint32_t elected, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}
__device__ __forceinline__ void mma_ts_e(uint32_t elected, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}

// Instruction descriptor for kind::f16 (bf16 or fp16 operands, fp32 accumulate).
//   [4,6) D format: 1 = f32      [7,10) A format: 0 = f16, 1 = bf16     [10,13) B format
//   [15] A major: 0 = K, 1 = MN  [16] B major                            [17,23) N>>3   [24,29) M>>4
__host__ __device__ constexpr uint32_t make_idesc(bool bf16, bool a_mn_major, bool b_mn_major, int M, int N) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

// Shared-memory matrix descriptor.
//   [0,14) start address >> 4   [16,30) leading byte offset >> 4   [32,46) stride byte offset >> 4
//   [46,48) version = 1 (Blackwell)   [61,64) swizzle: 0 none, 2 = 128B, 4 = 64B, 6 = 32B
// Swizzled K-major tiles: rows of `swizzle` bytes, 8-row atoms, SBO = 8 * swizzle (next 8 rows).
// Swizzled MN-major tiles: SBO = next 8 K-rows, LBO = next `swizzle`-byte block along M/N.
constexpr uint32_t SWZ_128B = 2, SWZ_64B = 4, SWZ_32B = 6;
// The same encoding without the start address, usable in constant expressions, and the
// assembly of a descriptor from a precomputed low word ((address >> 4) | leading-offset field)
// and high word.
__host__ __device__ constexpr uint64_t make_sdesc_const(uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t swz) {
  return (static_cast<uint64_t>(lbo_bytes >> 4) << 16) | (static_cast<uint64_t>(sbo_bytes >> 4) << 32) | (1ull << 46) |
         (static_cast<uint64_t>(swz) << 61);
}
__device__ __forceinline__ uint64_t pack_desc(uint32_t lo, uint32_t hi) {
  return static_cast<uint64_t>(lo) | (static_cast<uint64_t>(hi) << 32);
}
__host__ __device__ constexpr uint32_t swizzle_code_for_row_bytes(int row_bytes) {
  return row_bytes == 128 ? SWZ_128B : (row_bytes == 64 ? SWZ_64B : SWZ_32B);
}

// ---------------------------------------------------------------- tcgen05: TMEM <-> registers
// 32x32b shape: lane l of the warp reads TMEM lane (base_lane + l), N consecutive 32-bit columns.
// A warp may only touch the 32 TMEM lanes of its own quarter: lanes 32*(warp_id % 4) ...
#define EVO_R4(r, i) "=r"(r[i]), "=r"(r[i + 1]), "=r"(r[i + 2]), "=r"(r[i + 3])
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : EVO_R4(r, 0), EVO_R4(r, 4), EVO_R4(r, 8), EVO_R4(r, 12), EVO_R4(r, 16), EVO_R4(r, 20), EVO_R4(r, 24),
        EVO_R4(r, 28)
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : EVO_R4(r, 0), EVO_R4(r, 4), EVO_R4(r, 8), EVO_R4(r, 12)
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : EVO_R4(r, 0), EVO_R4(r, 4)
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : EVO_R4(r, 0) : "r"(taddr) : "memory");
}
#undef EVO_R4
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[N]) {
  static_assert(N == 4 || N == 8 || N == 16 || N == 32, "unsupported TMEM load width");
  if constexpr (N == 32) tmem_ld32(taddr, r);
  else if constexpr (N == 16) tmem_ld16(taddr, r);
  else if constexpr (N == 8) tmem_ld8(taddr, r);
  else tmem_ld4(taddr, r);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

#define EVO_I4(r, i) "r"(r[i]), "r"(r[i + 1]), "r"(r[i + 2]), "r"(r[i + 3])
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
      ::EVO_I4(r, 0), EVO_I4(r, 4), EVO_I4(r, 8), EVO_I4(r, 12), EVO_I4(r, 16), EVO_I4(r, 20), EVO_I4(r, 24),
      EVO_I4(r, 28), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      ::EVO_I4(r, 0), EVO_I4(r, 4), EVO_I4(r, 8), EVO_I4(r, 12), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
               ::EVO_I4(r, 0), EVO_I4(r, 4), "r"(taddr)
               : "memory");
}
#undef EVO_I4

// ---------------------------------------------------------------- predicated global loads
// A load whose value is needed much later must not be followed by a select on its result: the
// select would wait for the load where it stands.  These write the destination only when `pred`
// holds and leave `dflt` in it otherwise; the address is not touched when `pred` is false.
__device__ __forceinline__ uint32_t ldg_u32_if(const void* p, bool pred) {
  uint32_t v = 0u;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q ld.global.u32 %0, [%1];\n\t}"
               : "+r"(v) : "l"(p), "r"((int)pred));
  return v;
}
__device__ __forceinline__ uint32_t ldg_u16_if(const void* p, bool pred) {
  uint32_t v = 0u;
  asm volatile("{\n\t.reg .pred q;\n\t.reg .b16 h;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b16 h, 0;\n\t"
               "@q ld.global.u16 h, [%1];\n\t@q cvt.u32.u16 %0, h;\n\t}"
               : "+r"(v) : "l"(p), "r"((int)pred));
  return v;
}
__device__ __forceinline__ uint32_t ldg_u8_if(const void* p, bool pred) {
  uint32_t v = 0u;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q ld.global.u8 %0, [%1];\n\t}"
               : "+r"(v) : "l"(p), "r"((int)pred));
  return v;
}

// Adds four floats to global memory (sixteen-byte aligned).
__device__ __forceinline__ void red_add_v4(float* p, float x, float y, float z, float w) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
// Adds a float to global memory where pred holds.
__device__ __forceinline__ void red_add_if(float* p, float x, bool pred) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q red.global.add.f32 [%0], %1;\n\t}" ::"l"(p), "f"(x), "r"((int)pred) : "memory");
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ---------------------------------------------------------------- shared-memory access by 32-bit address
// A load through a generic pointer that happens to point into shared memory is a generic load: it
// pays the address-space check and 64-bit address arithmetic, and the hardware tracks it like a
// global load.  These take the 32-bit shared-window address (smem_u32) and stay LDS / STS.
__device__ __forceinline__ float lds_f32(uint32_t saddr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(saddr));
  return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t saddr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(saddr));
  return v;
}
__device__ __forceinline__ uint4 lds_v4(uint32_t saddr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr));
  return v;
}
__device__ __forceinline__ uint16_t lds_u16(uint32_t saddr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(saddr));
  return v;
}
__device__ __forceinline__ float4 lds_v4f(uint32_t saddr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(saddr));
  return v;
}
__device__ __forceinline__ float2 lds_v2f(uint32_t saddr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(saddr));
  return v;
}
__device__ __forceinline__ void sts_u32(uint32_t saddr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(saddr), "r"(v) : "memory");
}
__device__ __forceinline__ void sts_f32(uint32_t saddr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(saddr), "f"(v) : "memory");
}
__device__ __forceinline__ void sts_v4(uint32_t saddr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// ---------------------------------------------------------------- small math / sync helpers
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1 / (1 + e^-x) to a few units in the last place of fp32, for results that are rounded to 16 bits: an
// exponential and a reciprocal, without the division's correction steps.
__device__ __forceinline__ float sigmoid16(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(1.f + ex2(x * -1.4426950408889634f)));
  return y;
}
// Packed fp32x2 arithmetic (sm_100): one instruction works on two floats held in a 64-bit
// register pair; halves the issue slots of the element-wise softmax math.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2_make(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ F2 f2_from_bits(uint32_t lo, uint32_t hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void f2_get(F2 a, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Move registers between the warps of a CTA (whole-warp instructions).  The requests of all
// warps must sum to at most the launch-time pool, or `inc` blocks for ever.
template <int N> __device__ __forceinline__ void setmaxnreg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N> __device__ __forceinline__ void setmaxnreg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// Programmatic dependent launch: wait until the kernels before this one on the stream have completed (and
// their writes are visible); let the next one be scheduled.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }


// ---------------------------------------------------------------- leader-predicated commit
// For a warp that runs with all 32 lanes converged and predicates only the instruction that must be
// issued by a single thread (`leader` is non-zero in exactly one lane).
__device__ __forceinline__ void mma_commit_if_s(uint32_t leader, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(bar), "r"(leader)
      : "memory");
}
// ---------------------------------------------------------------- TMA on 32-bit shared-window addresses
__device__ __forceinline__ void tma_load_5d_s(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2,
                                              int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_s(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2,
                                              int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_s(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// Tiled store shared -> global.
__device__ __forceinline__ void tma_store_5d_s(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3, int c4) {
  asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
               ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
               : "memory");
}
// Tiled reduction shared -> global: global[tile] += shared[tile] (type and tile from the map).
__device__ __forceinline__ void tma_reduce_add_4d_s(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
      ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_reduce_add_3d_s(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
      ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

}  // namespace ptx
}  // namespace evo
