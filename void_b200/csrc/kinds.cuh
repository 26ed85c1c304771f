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
template <int KIND>
__device__ __forceinline__ void issue_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if (KIND == VOID_KIND_I8) mma_i8(d, a, b, idesc, acc);
  else if (KIND == VOID_KIND_F8E4M3) mma_f8(d, a, b, idesc, acc);
  else if (KIND == VOID_KIND_TF32) mma_tf32(d, a, b, idesc, acc);
  else mma_f16(d, a, b, idesc, acc);
}

}  // namespace vb
