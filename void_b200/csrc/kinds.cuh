// Operand kinds of the tensor-memory kernels and their matrix instructions.
#pragma once
#include <stdint.h>

#include "../../include/void_b200.h"
#include "ptx.cuh"

namespace vb {

// Bytes per element of the operands of a kind: the 8-bit kinds, fp16 / bf16, fp32 read as TF32.  A tile
// takes kTileBytes * ES bytes, a 128-column panel kPanelBytes * ES (stored as ES blocks of 32 k-rows x
// 128 bytes, one swizzle atom wide each), and one (tile, panel) product takes ES MMAs of 32 bytes of k.
template <int KIND>
struct Elem {
  static constexpr int ES = (KIND == VOID_KIND_TF32) ? 4 : ((KIND == VOID_KIND_F16 || KIND == VOID_KIND_BF16) ? 2 : 1);
};
// D[tmem] (+)= A[smem desc] * B[smem desc], issued by the one lane of a converged warp whose `leader` is true, as a predicated
// instruction: a branch around every product costs the warp more than the issue.  fp32 4096^2, 90 %, N = 512 (four products per tile
// and panel) 12.4 -> 11.6 us; one product per tile and panel: within 0.5 %.
template <int KIND>
__device__ __forceinline__ void issue_mma(bool leader, uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
#define VB_MMA(NAME)                                                                                                   \
  asm volatile(                                                                                                        \
      "{\n .reg .pred p, q;\n setp.ne.b32 q, %5, 0;\n setp.ne.b32 p, %4, 0;\n"                                        \
      " @q tcgen05.mma.cta_group::1." NAME " [%0], %1, %2, %3, p;\n}\n"                                                \
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"((uint32_t)leader) : "memory")
  if constexpr (KIND == VOID_KIND_I8) VB_MMA("kind::i8");
  else if constexpr (KIND == VOID_KIND_F8E4M3) VB_MMA("kind::f8f6f4");
  else if constexpr (KIND == VOID_KIND_TF32) VB_MMA("kind::tf32");
  else VB_MMA("kind::f16");
#undef VB_MMA
}

// The same with the descriptors in halves (their upper halves do not change from one instruction to the next).
template <int KIND>
__device__ __forceinline__ void mma_halves(bool leader, uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                           uint32_t idesc, uint32_t acc) {
#define VB_MMA(NAME)                                                                                                   \
  asm volatile(                                                                                                        \
      "{\n .reg .pred p, q;\n .reg .b64 a, b;\n mov.b64 a, {%1, %2};\n mov.b64 b, {%3, %4};\n setp.ne.b32 p, %6, 0;\n" \
      " setp.ne.b32 q, %7, 0;\n @q tcgen05.mma.cta_group::1." NAME " [%0], a, b, %5, p;\n}\n"                          \
      ::"r"(d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc), "r"((uint32_t)leader) : "memory")
  if constexpr (KIND == VOID_KIND_I8) VB_MMA("kind::i8");
  else if constexpr (KIND == VOID_KIND_F8E4M3) VB_MMA("kind::f8f6f4");
  else if constexpr (KIND == VOID_KIND_TF32) VB_MMA("kind::tf32");
  else VB_MMA("kind::f16");
#undef VB_MMA
}

}  // namespace vb
