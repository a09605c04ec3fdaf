// Inline-PTX building blocks of the tcgen05 kernels (k_tc_gemm.cu,
// k_chol_tc.cu): mbarriers, TMA tile loads, UMMA shared-memory and
// instruction descriptors, tcgen05.mma / commit / ld.
#pragma once
#include <cuda.h>
#include <cstdint>

namespace uhm_gpu {

constexpr uint32_t TC_DRAIN_LIMIT = 1u << 22;   // waits for a CTA's own copies in flight

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.b32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// bounded wait with an explicit limit: false (and the error word set to
// code) when the barrier does not complete, or at once when another role of
// the CTA has raised the abort flag
__device__ __forceinline__ bool mbar_wait_lim(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                              int* err, int code, uint32_t lim) {
  for (uint32_t i = 0; i < lim; ++i) {
    if (mbar_try(bar, parity)) return true;
    if (*abort_flag) return false;
    if (i > 64) __nanosleep(64);
  }
  *abort_flag = 1;
  if (err) atomicExch(err, code);
  return false;
}

// wait with a fixed limit that the settable one does not shorten: used only
// to let the CTA's own TMA copies and MMAs land before it frees its memory
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < TC_DRAIN_LIMIT; ++i) {
    if (mbar_try(bar, parity)) return;
    __nanosleep(64);
  }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// UMMA shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row
// groups 1024 bytes apart (SBO), descriptor version 1 (bits 46-47)
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;            // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;  // stride byte offset
  d |= (uint64_t)1 << 46;            // version
  d |= (uint64_t)2 << 61;            // SWIZZLE_128B
  return d;
}

// the same with 64-byte swizzle (rows of 32 BF16): 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;            // SWIZZLE_64B
  return d;
}

// instruction descriptor, kind::f16: D = F32, A = B = BF16, K-major both, M = N = 128
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// one lane of the (converged) warp
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.b32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e;
}

// the low word of a K-major shared-memory descriptor at saddr (sdesc_sw128's
// high word is SDESC_SW128_HI); 32 bytes further along a row is + 2
__device__ __forceinline__ uint32_t sdesc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | 1u << 16; }
constexpr uint32_t SDESC_SW128_HI = (1024u >> 4) | 1u << 14 | 2u << 29;

// umma_bf16 by the elected lane of a converged warp, descriptors by their low
// words: the whole warp runs the issue loop, so that its addresses and barriers
// stay in uniform registers, which the instruction takes its operands from.
// From one thread's branch every operand is moved there first: the sliced update
// took 170 clocks per 128 x 128 x 16 MMA that way, 118 so (a kernel whose MMAs
// wait for HBM, k_tc_chol or k_tc_syrk, gains nothing).
__device__ __forceinline__ void umma_bf16_w(uint32_t elected, uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t hi,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, e;\n .reg .b64 da, db;\n setp.ne.b32 e, %0, 0;\n setp.ne.b32 p, %6, 0;\n"
      " mov.b64 da, {%2, %4};\n mov.b64 db, {%3, %4};\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %5, p;\n}\n" ::"r"(elected),
      "r"(tmem_d), "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "r"(accumulate));
}
// the same, accumulating, in a row of MMAs with one A operand: the first one keeps
// A in the tensor core's collector buffer, the others take it from there
enum { UMMA_A_FILL, UMMA_A_USE, UMMA_A_LAST };
template <int OP>
__device__ __forceinline__ void umma_bf16_wa(uint32_t elected, uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t hi,
                                             uint32_t idesc) {
#define UMMA_WA(op)                                                                                          \
  asm volatile("{\n .reg .pred p, e;\n .reg .b64 da, db;\n setp.ne.b32 e, %0, 0;\n setp.eq.b32 p, %0, %0;\n"  \
               " mov.b64 da, {%2, %4};\n mov.b64 db, {%3, %4};\n"                                            \
               " @e tcgen05.mma.cta_group::1.kind::f16.collector::a::" op " [%1], da, db, %5, p;\n}\n"       \
               ::"r"(elected), "r"(tmem_d), "r"(alo), "r"(blo), "r"(hi), "r"(idesc))
  if constexpr (OP == UMMA_A_FILL) UMMA_WA("fill");
  else if constexpr (OP == UMMA_A_USE) UMMA_WA("use");
  else UMMA_WA("lastuse");
#undef UMMA_WA
}
__device__ __forceinline__ void umma_commit_w(uint32_t elected, uint32_t bar) {
  asm volatile(
      "{\n .reg .pred e;\n setp.ne.b32 e, %0, 0;\n"
      " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];\n}\n" ::"r"(elected),
      "r"(bar)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

#define TC_LD32(taddr, v)                                                                        \
  asm volatile(                                                                                  \
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14," \
      "%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"              \
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),      \
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),   \
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),            \
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),            \
        "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])             \
      : "r"(taddr))

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

}  // namespace uhm_gpu
