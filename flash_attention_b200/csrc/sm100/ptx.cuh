// Thin inline-PTX wrappers for the Blackwell (sm_100a) features the tensor-core kernels use:
// mbarrier with bounded waits, TMA tiled loads, TMEM allocation, tcgen05.mma / ld / st / commit,
// shared-memory matrix descriptors and the instruction descriptor.  No CUTLASS dependency.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace fa {
namespace ptx {

// Every wait in the tensor-core kernels is bounded: a wait that has not completed after `limit` SM
// cycles (kWaitCycles unless a caller says otherwise) gives up, records `code` in the CTA's abort
// flag and in the device status word, and the kernel winds down (all other waits then fail fast),
// so a protocol bug shows up as an error code, not as a hang.
constexpr long long kWaitCycles = 3000000000ll;  // ~1.5 s at 2 GHz

// Where a kernel reports a wait that gave up: one word in device memory (the library's status
// word, shared by all its kernels) and, when the host has one, its mirror in mapped host memory,
// which the entry points read without synchronising.  Passed to every kernel by value.
struct StatusRef {
  int* dev;
  int* host;  // may be null
};

// Shared-memory block of every kernel that waits: [tmem address][abort flag][StatusRef], 24 bytes,
// 8-byte aligned.  Kernels hold a pointer to the abort flag; the StatusRef sits right behind it.
constexpr int kAbortBlockBytes = 24;
__device__ __forceinline__ void abort_publish(volatile int* abort_flag, int code) {
  int* dev = *reinterpret_cast<int* volatile*>(const_cast<int*>(abort_flag) + 1);
  int* host = *reinterpret_cast<int* volatile*>(const_cast<int*>(abort_flag) + 3);
  if (dev != nullptr && atomicCAS(dev, 0, code) == 0 && host != nullptr) {
    *reinterpret_cast<volatile int*>(host) = code;
    __threadfence_system();
  }
}
// One thread, before the CTA's first barrier: a failed earlier launch makes every later CTA bail
// out at its first wait (the status word is sticky until the host clears it).
__device__ __forceinline__ void abort_init(volatile int* abort_flag, const StatusRef& s) {
  *reinterpret_cast<int* volatile*>(const_cast<int*>(abort_flag) + 1) = s.dev;
  *reinterpret_cast<int* volatile*>(const_cast<int*>(abort_flag) + 3) = s.host;
  *abort_flag = s.dev ? *reinterpret_cast<volatile int*>(s.dev) : 0;
}
__device__ __forceinline__ void abort_raise(volatile int* abort_flag, int code) {
  *abort_flag = code;
  abort_publish(abort_flag, code);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// try_wait that lets the hardware park the thread for up to `ns` nanoseconds while the phase is
// incomplete (it is woken when the phase completes), instead of returning at once to a spin loop
// that competes for issue slots with the warps doing useful work on the same scheduler.
__device__ __forceinline__ bool mbar_try_wait_parked(uint32_t bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}
// Non-blocking test of a phase.  For a lone thread the round trip to the barrier is ~100+ cycles;
// the MMA issuer tests the barrier of its NEXT group before it issues the current group's MMAs and
// consumes the answer afterwards (mbar_wait_probed), so the tensor pipe is not left idle meanwhile.
// A phase that has been seen complete stays complete until its barrier completes another phase,
// which in these kernels needs further work of the testing thread itself.
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
// Returns false (and records `code`) when the wait gave up or the kernel is already aborting.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int code, volatile int* abort_flag,
                                          int mode = 0, long long limit = kWaitCycles) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  uint32_t polls = 0;
  while (true) {
    if (mode == 1) {
      if (mbar_try_wait_parked(bar, parity, 2000)) return true;
    } else if (mode == 2) {
      __nanosleep(40);
    } else if (mode == 3) {
      // a warp that waits for long stretches (an epilogue or bookkeeping role) must not compete for issue
      // slots with the warps that do the arithmetic on the same scheduler
      __nanosleep(400);
    }
    if (mbar_try_wait(bar, parity)) return true;
    if ((++polls & 63u) == 0) {
      if (*abort_flag) return false;
      if (clock64() - t0 > limit) {
        abort_raise(abort_flag, code);
        return false;
      }
    }
  }
}

// For a warp that must stay converged (an MMA-issuing warp): every lane waits, and all lanes get the
// same answer even if a wait gave up for some lanes just as the phase completed for others.
__device__ __forceinline__ bool mbar_wait_w(uint32_t bar, uint32_t parity, int code, volatile int* abort_flag) {
  const bool ok = mbar_wait(bar, parity, code, abort_flag);
  return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ bool mbar_wait_probed(uint32_t hit, uint32_t bar, uint32_t parity, int code,
                                                 volatile int* abort_flag) {
  if (hit) return true;
  return mbar_wait(bar, parity, code, abort_flag);
}

// ---- TMA -------------------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 4-D tiled load into this CTA's own shared memory only.  c0 is the innermost (contiguous) coordinate and must keep
// c0 * sizeof(element) a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2,
                                            int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// Bulk fp32 add-reduction of `bytes` contiguous bytes from shared to global memory (both 16-byte
// aligned, bytes a multiple of 16).  The reduction is performed at the memory side in whole lines.
__device__ __forceinline__ void bulk_reduce_add_f32(float* gdst, uint32_t ssrc, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(gdst), "r"(ssrc),
               "r"(bytes)
               : "memory");
}
// Closes the bulk group of this thread and waits until its shared-memory source has been read.
__device__ __forceinline__ void bulk_commit_wait_read() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
// Waits until the bulk groups of this thread have completed entirely (writes performed).
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---- TMEM ------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
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
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// arrive on an mbarrier once all tcgen05.mma issued so far by this thread have completed
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// The same three instructions for an issuing WARP that stays converged: every lane executes the
// surrounding control flow (so that addresses and descriptors are warp-uniform values, which the
// compiler keeps in uniform registers instead of moving them there one by one for a lone thread),
// and one elected lane issues.  elect.sync picks the same lane every time for a full mask, which
// tcgen05.commit relies on (it tracks the MMAs of the thread that executes it).
__device__ __forceinline__ void mma_ss_w(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_ts_w(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit_w(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(bar)
      : "memory");
}

// 32 lanes x 32 columns of 32 bits: thread i of the warp gets lane (warp%4)*32 + i.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
      "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
      "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// ---- descriptors -----------------------------------------------------------------------------
// Shared-memory matrix descriptor for a 128-byte-swizzled tile whose rows are 128 bytes
// (64 16-bit elements) and whose 8-row groups are 1024 bytes apart.
//   K-major operand  (rows = M or N index, 64 K-elements per row): SBO = 1024, LBO unused.
//   MN-major operand (rows = K index, 64 MN-elements per row): SBO = 1024 (8 K-rows),
//                    LBO = byte distance between consecutive 64-element MN chunks.
// bits: [0,14) addr>>4, [16,30) LBO>>4, [32,46) SBO>>4, [46,48) version=1, [61,64) layout (2 = 128B swizzle)
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Instruction descriptor for kind::f16 with fp32 accumulation.
// ab_format: 0 = fp16, 1 = bf16; *_mn_major: 1 when the operand is MN-major in shared memory.
__host__ __device__ constexpr uint32_t make_idesc(int M, int N, int ab_format, int a_mn_major, int b_mn_major) {
  return (1u << 4)                           // D format: F32
         | ((uint32_t)ab_format << 7)        // A format
         | ((uint32_t)ab_format << 10)       // B format
         | ((uint32_t)a_mn_major << 15)      // A major
         | ((uint32_t)b_mn_major << 16)      // B major
         | ((uint32_t)(N >> 3) << 17)        // N / 8
         | ((uint32_t)(M >> 4) << 24);       // M / 16
}

// Head dims between the kernels' own (64, 128, 256): the products take the 16-column k-steps and the result columns that hold
// data, and the loads the 64-column chunks that do; what a tile holds behind them is not read.
// 8 x 2048 tokens, full, forward / backward in us with the padding and without: 32 heads of 32 420 / 1000 -> 409 / 944, 25 of 80
// 372 / 1153 -> 356 / 1026, 21 of 96 333 / 1022 -> 324 / 932, 12 of 160 448 / 1425 -> 382 / 1267, 10 of 192 369 / 1199 -> 333 / 1132.
// f(integral_constant) is called with the number of k-steps, a constant, because the issuing warp is often what a product waits
// for: with a test per MMA of a count read from the parameters head dims 64 and 128 took 1 to 4 % longer, 256 (backward) 20 %.
// TRIM is an instance of the kernel of its own for the same reason (all in one: 128 1.4 %, 256 9 % longer).
template <int DH, bool TRIM, typename F>
__device__ __forceinline__ void with_head_steps(int head_dim, F&& f) {
  if constexpr (!TRIM) {
    f(std::integral_constant<int, DH / 16>{});
  } else {  // (head_trims: at most three quarters of DH)
    constexpr int kLess = DH == 64 ? 2 : DH == 128 ? 5 : 10, kMore = DH / 16 * 3 / 4;
    if (head_dim <= kLess * 16)
      f(std::integral_constant<int, kLess>{});
    else
      f(std::integral_constant<int, kMore>{});
  }
}
// chunks of a tile of DH columns (a tile of up to 128 columns is always loaded whole: its last chunk holds data)
template <int DH, bool TRIM>
__device__ __forceinline__ int head_chunks(int head_dim) {
  return TRIM && DH > 128 ? (head_dim + 63) / 64 : DH / 64;
}

// whether with_head_steps has a smaller count than DH / 16 for this head dim
template <int DH>
constexpr bool head_trims(int head_dim) {
  return head_dim <= DH * 3 / 4;
}

// ---- packed fp32 pairs (sm_100 has two-wide fp32 FMA/ADD and a three-input max) ------------------
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pack2u(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

template <int N>
__device__ __forceinline__ void setmaxnreg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
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

}  // namespace ptx
}  // namespace fa
