// Thin inline-PTX wrappers for the sm_100a features the attention kernels use:
// mbarrier, TMA (cp.async.bulk.tensor), tcgen05 (alloc / mma / commit / ld / st / fences).
// Every wait is bounded: on expiry it raises the CTA-wide abort flag so that all roles
// drain and the kernel returns with an error status instead of hanging the GPU.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

namespace fsa {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ----------------------------------------------------------------------------------------------
// mbarrier
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok;
}

// Upper bound of any wait, in SM clock cycles (about two seconds). Far above any legitimate wait
// (a whole CTA lives for well under a second) and still ends a broken pipeline in bounded time.
#ifndef FSA_WAIT_CYCLES
#define FSA_WAIT_CYCLES (4000000000ll)
#endif

// Bounded wait. Returns false when the wait expired or another role already aborted.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t i = 0;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63u) == 63u) {
      if (*abort_flag) return false;
      if (clock64() - t0 > FSA_WAIT_CYCLES) break;
    }
  }
  *abort_flag = 1;
  return false;
}

// The same for a converged warp, with a result that the compiler knows to be the same in all lanes. It waits until every lane has
// seen the phase: a vote orders no memory, so a lane has acquired only what its own test saw. The phase stays until all have,
// since the next one needs this warp.
__device__ __forceinline__ bool mbar_wait_uniform(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const long long t0 = clock64();
  for (uint32_t i = 0;; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((i & 63u) == 63u) {
      if (__any_sync(0xffffffffu, *abort_flag)) return false;
      if (__any_sync(0xffffffffu, clock64() - t0 > FSA_WAIT_CYCLES)) break;
    }
  }
  *abort_flag = 1;
  return false;
}

// ----------------------------------------------------------------------------------------------
// Proxy / tcgen05 fences
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Named barrier over a subset of the CTA (id 1..15; id 0 is __syncthreads).
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// ----------------------------------------------------------------------------------------------
// TMA tiled loads (no multicast anywhere: each CTA fetches its own tiles)
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// ----------------------------------------------------------------------------------------------
// tcgen05: tensor memory management
// ----------------------------------------------------------------------------------------------
// One full warp allocates `ncols` (power of two, >= 32) TMEM columns; the base address lands in smem.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ----------------------------------------------------------------------------------------------
// tcgen05: descriptors
// ----------------------------------------------------------------------------------------------
// Shared-memory matrix descriptor for a tile stored as rows of 128 bytes with the 128-byte
// swizzle (what a TMA box of 64 16-bit elements x R rows with SWIZZLE_128B produces; R a
// multiple of 8, tile base 1024-byte aligned).
//   * used K-major   (rows = M/N index, the 64 elements of a row = K): SBO = 1024 (next 8 rows)
//   * used MN-major  (rows = K index, the 64 elements of a row = M/N): SBO = 1024 (next 8 K rows),
//     LBO = byte distance to the next 64-wide M/N slab
// Fields: [0,14) start>>4, [16,30) LBO>>4, [32,46) SBO>>4, [46,48) version=1, [61,64) layout=2.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}

// Instruction descriptor for kind::f16 (A/B both fp16 or both bf16, fp32 accumulate).
// a_mn / b_mn: 1 when that operand is MN-major in shared memory.
__host__ __device__ constexpr uint32_t umma_idesc_f16(int M, int N, bool is_bf16, bool a_mn, bool b_mn) {
  return (1u << 4)                                  // D = f32
         | ((is_bf16 ? 1u : 0u) << 7)               // A format
         | ((is_bf16 ? 1u : 0u) << 10)              // B format
         | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}
// Instruction descriptor for kind::f8f6f4 with e4m3 (0) / e5m2 (1) operands, fp32 accumulate.
__host__ __device__ constexpr uint32_t umma_idesc_f8(int M, int N, int a_fmt, int b_fmt, bool a_mn, bool b_mn) {
  return (1u << 4) | (static_cast<uint32_t>(a_fmt) << 7) | (static_cast<uint32_t>(b_fmt) << 10) |
         ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}

// ----------------------------------------------------------------------------------------------
// tcgen05: MMA issue (one thread), completion tracking
// ----------------------------------------------------------------------------------------------
// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem, 8-bit, four values per 32-bit column] * B[smem]
__device__ __forceinline__ void umma_f8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_f8_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 1 in one lane of a converged warp, 0 in the others.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t r;
  asm volatile(
      "{\n\t"
      ".reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, e;\n\t"
      "}\n"
      : "=r"(r));
  return r;
}
// Leader-predicated forms: the whole warp runs the (warp-uniform) address arithmetic and the instruction
// carries the single-lane predicate, instead of a divergent branch around a block of MMAs. `lead` has to come from
// elect_one(): with "lane == 0" in its place the issue of a 128 x 128 x 16 MMA takes 68 to 80 cycles, the more the busier the
// other warps of the scheduler are, with the elected lane 64, as long as the MMA itself
// (148 CTAs, 2000 steps of 40 MMAs and five commits each, ten warps beside the issuer copying, loading or calculating).
#define FSA_UMMA_LEAD(NAME, KIND, AFMT, ATYPE, ACONS)                                                        \
  __device__ __forceinline__ void NAME(uint32_t lead, uint32_t d_tmem, ATYPE a, uint64_t bdesc, uint32_t idesc, \
                                       uint32_t accumulate) {                                                \
    asm volatile(                                                                                            \
        "{\n\t"                                                                                              \
        ".reg .pred p, e;\n\t"                                                                               \
        "setp.ne.b32 p, %4, 0;\n\t"                                                                          \
        "setp.ne.b32 e, %5, 0;\n\t"                                                                          \
        "@e tcgen05.mma.cta_group::1.kind::" KIND " [%0], " AFMT ", %2, %3, p;\n\t"                          \
        "}\n" ::"r"(d_tmem),                                                                                 \
        ACONS(a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)                                         \
        : "memory");                                                                                         \
  }
FSA_UMMA_LEAD(umma_ss_lead, "f16", "%1", uint64_t, "l")
FSA_UMMA_LEAD(umma_ts_lead, "f16", "[%1]", uint32_t, "r")
FSA_UMMA_LEAD(umma_f8_ss_lead, "f8f6f4", "%1", uint64_t, "l")
FSA_UMMA_LEAD(umma_f8_ts_lead, "f8f6f4", "[%1]", uint32_t, "r")
#undef FSA_UMMA_LEAD
__device__ __forceinline__ void umma_commit_lead(uint32_t lead, uint64_t* bar) {
  asm volatile(
      "{\n\t"
      ".reg .pred e;\n\t"
      "setp.ne.b32 e, %1, 0;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
      "}\n" ::"r"(smem_u32(bar)),
      "r"(lead)
      : "memory");
}
// Shared-memory descriptor of a 128-byte-swizzled operand with stride-byte-offset 1024 as (low word, constant
// high word): advancing inside a tile is an add on the low word (the address field holds addr >> 4, 14 bits,
// enough for every shared-memory address).
constexpr uint32_t UMMA_DESC_HI_SW128 = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr >> 4) & 0x3FFFu) | ((lbo_bytes >> 4) << 16);
}
__device__ __forceinline__ uint64_t umma_desc_at(uint32_t lo, uint32_t byte_off) {
  return (static_cast<uint64_t>(UMMA_DESC_HI_SW128) << 32) | static_cast<uint64_t>(lo + (byte_off >> 4));
}
// mbarrier arrives once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// ----------------------------------------------------------------------------------------------
// tcgen05: TMEM <-> registers. Shape 32x32b: lane i of the warp owns TMEM lane (base + i);
// register j is column (base + j). A warp can only touch lanes [32*(warp_id%4), +32).
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
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
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
      "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
      "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ----------------------------------------------------------------------------------------------
// Small math helpers
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// logsigmoid(x) = min(x, 0) - log1p(exp(-|x|)) with one special-function op (the exponential): log1p(u)
// on u in (0, 1] is a degree-5 polynomial u * q(u), absolute error < 4.1e-5 - far below the rounding of the
// 16-bit probabilities the gate ends up in. (flash_sparse_attn/ops/triton/activations.py:245-262)
__device__ __forceinline__ float log_sigmoid_fast(float x) {
  float u;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(u) : "f"(-fabsf(x) * 1.4426950408889634f));
  float q = fmaf(u, 0.0415511145f, -0.157838377f);
  q = fmaf(q, u, 0.3065611f);
  q = fmaf(q, u, -0.497030843f);
  q = fmaf(q, u, 0.999944993f);
  return fminf(x, 0.f) - u * q;
}
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Bits [a, a + n) of a word, a and n clamped to it: a in 0..32, n >= 0.
__device__ __forceinline__ uint32_t bit_range(int a, int n) {
  uint32_t r;
  asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(n));
  return r;
}
// The part of the half-open interval [lo, lo + len) that falls on columns [base, base + 32), as bits.
__device__ __forceinline__ uint32_t interval_bits(int lo, unsigned len, int base) {
  const int a = max(lo - base, 0), b = min(lo + (int)len - base, 32);
  return bit_range(a, max(b - a, 0));
}

// 3-input maximum and packed two-wide fp32 arithmetic (one instruction for two lanes of data).
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ uint64_t f2_pack(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t r) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(r));
  return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t rd;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(f2_pack(a.x, a.y)), "l"(f2_pack(b.x, b.y)), "l"(f2_pack(c.x, c.y)));
  return f2_unpack(rd);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  uint64_t rd;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(f2_pack(a.x, a.y)), "l"(f2_pack(b.x, b.y)));
  return f2_unpack(rd);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  uint64_t rd;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(f2_pack(a.x, a.y)), "l"(f2_pack(b.x, b.y)));
  return f2_unpack(rd);
}

// logsigmoid(x) for two values, x given as y = x * log2(e): the arithmetic of log_sigmoid_fast, packed. The polynomial carries the
// minus sign (a packed operation cannot negate an operand). The forward adds it to the scores in a rounding of its own where the backward
// takes add_log_sigmoid2: they differ by an ulp of the logit, and both are off by 4.1e-5 at most and 4.9e-6 in the root mean square, which
// is the polynomial (two million points of |x| <= 20, scores of deviation 1 to 30).
__device__ __forceinline__ float2 log_sigmoid2(float2 y) {
  const float2 u = make_float2(ex2_approx(-fabsf(y.x)), ex2_approx(-fabsf(y.y)));
  float2 q = fma2(u, make_float2(-0.0415511145f, -0.0415511145f), make_float2(0.157838377f, 0.157838377f));
  q = fma2(q, u, make_float2(-0.3065611f, -0.3065611f));
  q = fma2(q, u, make_float2(0.497030843f, 0.497030843f));
  q = fma2(q, u, make_float2(-0.999944993f, -0.999944993f));
  return fma2(make_float2(fminf(y.x, 0.f), fminf(y.y, 0.f)), make_float2(0.6931471806f, 0.6931471806f), mul2(q, u));
}
// s + logsigmoid(x)
__device__ __forceinline__ float2 add_log_sigmoid2(float2 s, float2 y) {
  const float2 u = make_float2(ex2_approx(-fabsf(y.x)), ex2_approx(-fabsf(y.y)));
  float2 q = fma2(u, make_float2(-0.0415511145f, -0.0415511145f), make_float2(0.157838377f, 0.157838377f));
  q = fma2(q, u, make_float2(-0.3065611f, -0.3065611f));
  q = fma2(q, u, make_float2(0.497030843f, 0.497030843f));
  q = fma2(q, u, make_float2(-0.999944993f, -0.999944993f));
  s = fma2(make_float2(fminf(y.x, 0.f), fminf(y.y, 0.f)), make_float2(0.6931471806f, 0.6931471806f), s);
  return fma2(u, q, s);
}

// sigmoid(-x) = 1 / (1 + 2^y) for two values, y = x * log2(e): one reciprocal for both. 2^y is capped at 2^62, so that the
// product of the two denominators stays finite; a sigmoid below 2^-62 counts as 2^-62.
__device__ __forceinline__ float2 sigmoid_neg2(float2 y) {
  const float2 d = add2(make_float2(ex2_approx(fminf(y.x, 62.f)), ex2_approx(fminf(y.y, 62.f))), make_float2(1.f, 1.f));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d.x * d.y));
  return mul2(make_float2(r, r), make_float2(d.y, d.x));
}

template <typename T>
__device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Four fp32 values rounded (nearest even, clamped to the largest finite value) to FP8 and packed in
// memory order v0, v1, v2, v3.
template <typename T>
__device__ __forceinline__ uint32_t pack4_fp8(float v0, float v1, float v2, float v3);
template <>
__device__ __forceinline__ uint32_t pack4_fp8<__nv_fp8_e5m2>(float v0, float v1, float v2, float v3) {
  uint16_t lo, hi;
  asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(v1), "f"(v0));
  asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(v3), "f"(v2));
  return uint32_t(lo) | (uint32_t(hi) << 16);
}
template <>
__device__ __forceinline__ uint32_t pack4_fp8<__nv_fp8_e4m3>(float v0, float v1, float v2, float v3) {
  uint16_t lo, hi;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(v1), "f"(v0));
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(v3), "f"(v2));
  return uint32_t(lo) | (uint32_t(hi) << 16);
}

// Conversion that clamps to the largest finite value (matters for fp16 only), and the packed product
// rounded once to the 16-bit type.
template <typename T>
__device__ __forceinline__ uint32_t pack2_sat(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack2_sat<__nv_bfloat16>(float lo, float hi) {
  return pack2<__nv_bfloat16>(lo, hi);
}
template <>
__device__ __forceinline__ uint32_t pack2_sat<__half>(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
template <typename T>
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b);
template <>
__device__ __forceinline__ uint32_t hmul2<__nv_bfloat16>(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <>
__device__ __forceinline__ uint32_t hmul2<__half>(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// Byte offset of 16-byte chunk `chunk` (0..7) of row `row` inside a [rows x 128 B] tile with the
// 128-byte swizzle (tile base 1024-byte aligned).
__device__ __forceinline__ uint32_t sw128_offset(uint32_t row, uint32_t chunk) {
  return row * 128u + ((chunk ^ (row & 7u)) << 4);
}

}  // namespace fsa
