// Epilogue of the tensor-memory product kernels: raw accumulators of one output column n and a few tile rows m to finished
// values of C (dequantise, bias, activation, conversion), stored directly, through a staging tile, or transposed.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "../../include/void_b200.h"
#include "ptx.cuh"

namespace vb {

constexpr int kTile = 32;
constexpr int kTileBytes = 1024;
constexpr int kPanelN = 128;
constexpr int kPanelBytes = kTile * kPanelN;  // 4096

// 1 / (1 + 2^w) with the hardware's exponential and reciprocal (a few ulp together; far inside the path's 1e-3 bar).
__device__ __forceinline__ float sigmoid_exp2(float w) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(w));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  return r;
}
constexpr double kLog2e = 1.4426950408889634074;
// GELU in the tanh form written with a sigmoid, void/fusion.py:38-43: x * 0.5 * (1 + (2 sigmoid(2u) - 1)) = x * sigmoid(2u),
// 2u = 1.5957691216 (x + 0.044715 x^3); the factor log2(e) of the exponential is in the constants.
constexpr float kGelu1 = (float)(-1.5957691216 * kLog2e), kGelu3 = (float)(-1.5957691216 * 0.044715 * kLog2e);
constexpr float kSilu = (float)-kLog2e;
// One value, for the kernels whose epilogue is no loop over registers.
__device__ __forceinline__ float activate(float x, int act) {
  if (act == VOID_ACT_NONE) return x;
  if (act == VOID_ACT_RELU) return fmaxf(x, 0.0f);
  return x * sigmoid_exp2(x * (act == VOID_ACT_GELU ? fmaf(x * x, kGelu3, kGelu1) : kSilu));
}
// The same for PAIRS pairs of values, the choice made once.
__device__ __forceinline__ f32x2 times_sigmoid(f32x2 x, f32x2 w) {
  float a, b;
  unpair(w, a, b);
  return mul2(x, pair(sigmoid_exp2(a), sigmoid_exp2(b)));
}
template <int PAIRS>
__device__ __forceinline__ void activate(f32x2 (&x)[PAIRS], int act) {
  if (act == VOID_ACT_NONE) return;
  if (act == VOID_ACT_GELU) {
#pragma unroll
    for (int k = 0; k < PAIRS; ++k)
      x[k] = times_sigmoid(x[k], mul2(x[k], fma2(mul2(x[k], x[k]), pair(kGelu3, kGelu3), pair(kGelu1, kGelu1))));
  } else if (act == VOID_ACT_RELU) {
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) {
      float a, b;
      unpair(x[k], a, b);
      x[k] = pair(fmaxf(a, 0.0f), fmaxf(b, 0.0f));
    }
  } else {
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) x[k] = times_sigmoid(x[k], mul2(x[k], pair(kSilu, kSilu)));
  }
}
// What an epilogue thread needs to know about C, read from the kernel parameters once.
struct OutDesc {
  void* out;
  long long ldc;
  void* acc_out;
  const float* row_bias;  // [M] added per output row before the activation (linear-layer bias), or null
  int M, N, dtype, act;
};
// Raw accumulators of one output column, matrix rows r0 .. r0 + 2 PAIRS - 1, to finished values: dequantise (floating tiles have
// no row scale), bias, activation.
template <int KIND>
__device__ __forceinline__ f32x2 dequantise(uint32_t a, uint32_t b, f32x2 row_scale, f32x2 cs, f32x2 bias) {
  if (KIND == VOID_KIND_I8) return fma2(mul2(pair(__int2float_rn((int)a), __int2float_rn((int)b)), row_scale), cs, bias);
  const f32x2 x = pair(__uint_as_float(a), __uint_as_float(b));
  return fma2(KIND == VOID_KIND_F8E4M3 ? mul2(x, row_scale) : x, cs, bias);
}
// ACT: whether there may be a row bias or an activation.
template <int PAIRS>
__device__ __forceinline__ void row_bias_activation(const OutDesc& o, int r0, f32x2 (&x)[PAIRS]) {
  if (o.row_bias != nullptr) {
    const int rows = o.M - r0;  // rows left below r0
#pragma unroll
    for (int k = 0; k < PAIRS; ++k)
      x[k] = add2(x[k], pair(2 * k < rows ? o.row_bias[r0 + 2 * k] : 0.0f, 2 * k + 1 < rows ? o.row_bias[r0 + 2 * k + 1] : 0.0f));
  }
  activate<PAIRS>(x, o.act);
}
template <int KIND, int PAIRS, bool ACT>
__device__ __forceinline__ void finished(const OutDesc& o, int r0, const uint32_t* r, float row_scale, float cs, float bias,
                                         float (&v)[2 * PAIRS]) {
  const f32x2 rs2 = pair(row_scale, row_scale), cs2 = pair(cs, cs), bias2 = pair(bias, bias);
  f32x2 x[PAIRS];
#pragma unroll
  for (int k = 0; k < PAIRS; ++k) x[k] = dequantise<KIND>(r[2 * k], r[2 * k + 1], rs2, cs2, bias2);
  if (ACT) row_bias_activation<PAIRS>(o, r0, x);
#pragma unroll
  for (int k = 0; k < PAIRS; ++k) unpair(x[k], v[2 * k], v[2 * k + 1]);
}
// Store eight values of output column n, matrix rows row*32 + m0 .. + 7, after row bias and activation.
__device__ __forceinline__ void store8(const OutDesc& o, int row, int n, int m0, float (&v)[8]) {
  const int r0 = row * kTile + m0;
  const int rows = o.M - r0;
  f32x2 x[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) x[k] = pair(v[2 * k], v[2 * k + 1]);
  row_bias_activation<4>(o, r0, x);
#pragma unroll
  for (int k = 0; k < 4; ++k) unpair(x[k], v[2 * k], v[2 * k + 1]);
  if (o.dtype == VOID_OUT_F16) {
    __half* dst = reinterpret_cast<__half*>(o.out) + (size_t)r0 * o.ldc + n;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < rows) dst[(size_t)k * o.ldc] = __float2half_rn(v[k]);
  } else if (o.dtype == VOID_OUT_BF16) {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(o.out) + (size_t)r0 * o.ldc + n;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < rows) dst[(size_t)k * o.ldc] = __float2bfloat16_rn(v[k]);
  } else {
    float* dst = reinterpret_cast<float*>(o.out) + (size_t)r0 * o.ldc + n;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < rows) dst[(size_t)k * o.ldc] = v[k];
  }
}

// Epilogue of eight raw accumulators of one output column: dequantise, bias, activation, store.
template <int KIND>
__device__ __forceinline__ void finish8(const OutDesc& o, int row, int n, int m0, const uint32_t (&r)[8],
                                        float row_scale, float cs, float bias) {
  if (n >= o.N) return;
  if (o.acc_out != nullptr) {
    uint32_t* a = reinterpret_cast<uint32_t*>(o.acc_out) + ((size_t)row * kTile + m0) * o.N + n;
#pragma unroll
    for (int k = 0; k < 8; ++k) a[(size_t)k * o.N] = r[k];
  }
  const f32x2 rs2 = pair(row_scale, row_scale), cs2 = pair(cs, cs), bias2 = pair(bias, bias);
  float v[8];
#pragma unroll
  for (int k = 0; k < 4; ++k) unpair(dequantise<KIND>(r[2 * k], r[2 * k + 1], rs2, cs2, bias2), v[2 * k], v[2 * k + 1]);
  store8(o, row, n, m0, v);
}

// Fast epilogue of sixteen raw accumulators of output column n (tile rows m0 .. m0 + 15) straight to C
// (no raw-accumulator dump, no split row), stores specialised per output type.
template <int KIND, bool ACT = true>
__device__ __forceinline__ void finish16(const OutDesc& o, int row, int n, int m0, const uint32_t* r,
                                         float row_scale, float cs, float bias) {
  if (n >= o.N) return;
  const int r0 = row * kTile + m0;
  const int rows = o.M - r0;
  float v[16];
  finished<KIND, 8, ACT>(o, r0, r, row_scale, cs, bias, v);
  const size_t first = (size_t)r0 * o.ldc + n;
  if (o.dtype == VOID_OUT_F16) {
    __half* dst = reinterpret_cast<__half*>(o.out) + first;
#pragma unroll
    for (int k = 0; k < 16; ++k, dst += o.ldc)
      if (k < rows) *dst = __float2half_rn(v[k]);
  } else if (o.dtype == VOID_OUT_BF16) {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(o.out) + first;
#pragma unroll
    for (int k = 0; k < 16; ++k, dst += o.ldc)
      if (k < rows) *dst = __float2bfloat16_rn(v[k]);
  } else {
    float* dst = reinterpret_cast<float*>(o.out) + first;
#pragma unroll
    for (int k = 0; k < 16; ++k, dst += o.ldc)
      if (k < rows) *dst = v[k];
  }
}

// A warp's 32 columns of a tile row of raw accumulators, as fragments (tmem_ld_fragments: lanes are columns), to finished
// 16-bit values in a part of shared memory, rows of 64 bytes whose 16-byte pieces lie as the copy engine's 64-byte swizzle
// has them (piece ^ row / 2 % 4; a part starts on 512 bytes).  cs and bias: those of the lane's own column.
// What bounds an epilogue is the number of its instructions, the sixteen epilogue warps of an SM being in theirs together; a
// thread that owns a column puts 32 halves into shared memory one by one; pairs of rows and matrix stores take a third of it.
// Instructions of a launch and its time, before and now: INT8 16384^2 power-law rows, N = 256, GELU 7.0 M 17.8 us, 5.4 M 14.2;
// bf16 4096 -> 16384, 2048 columns, GELU 57 M 95 us, 41 M 75; INT8 4096^2, 90 %, N = 512 2.67 M, 2.40 M.
template <bool F16>
__device__ __forceinline__ uint32_t half2_bits(f32x2 x) {
  float a, b;
  uint32_t d;
  unpair(x, a, b);
  if (F16) asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
  else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
  return d;
}
template <int KIND, bool ACT>
__device__ __forceinline__ void finish_fragments(const OutDesc& o, int r0, const uint32_t (&lo)[16], const uint32_t (&hi)[16],
                                                 float row_scale, float cs, float bias, bool biased, uint32_t part, int lane) {
  const f32x2 rs2 = pair(row_scale, row_scale);
  f32x2 x[16];   // [group of rows][columns t / 4 + 8 q]
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float c = __shfl_sync(0xffffffffu, cs, 8 * q + (lane >> 2));
    const float b = biased ? __shfl_sync(0xffffffffu, bias, 8 * q + (lane >> 2)) : 0.0f;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int k = 4 * g + 2 * (q & 1);
      x[4 * g + q] = dequantise<KIND>(q < 2 ? lo[k] : hi[k], q < 2 ? lo[k + 1] : hi[k + 1], rs2, pair(c, c), pair(b, b));
    }
  }
  if (ACT && o.row_bias != nullptr) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int r = r0 + 8 * g + 2 * (lane & 3);
      const f32x2 rb = pair(r < o.M ? o.row_bias[r] : 0.0f, r + 1 < o.M ? o.row_bias[r + 1] : 0.0f);
#pragma unroll
      for (int q = 0; q < 4; ++q) x[4 * g + q] = add2(x[4 * g + q], rb);
    }
  }
  if (ACT) activate<16>(x, o.act);
  const uint32_t at = part + (uint32_t)(lane & 7) * 64u + (uint32_t)(((lane >> 3) ^ ((lane >> 1) & 3)) << 4);
  if (o.dtype == VOID_OUT_F16) {
#pragma unroll
    for (int g = 0; g < 4; ++g)
      stmatrix_x4_trans(at + (uint32_t)g * 512u, half2_bits<true>(x[4 * g]), half2_bits<true>(x[4 * g + 1]), half2_bits<true>(x[4 * g + 2]),
                        half2_bits<true>(x[4 * g + 3]));
  } else {
#pragma unroll
    for (int g = 0; g < 4; ++g)
      stmatrix_x4_trans(at + (uint32_t)g * 512u, half2_bits<false>(x[4 * g]), half2_bits<false>(x[4 * g + 1]),
                        half2_bits<false>(x[4 * g + 2]), half2_bits<false>(x[4 * g + 3]));
  }
}

// Transposed output (C stored as [N, M], m contiguous): the thread owns output row n and sixteen consecutive
// columns m0 .. m0 + 15 of it, so the values leave in 16-byte stores.  bias_n is the bias of this n, the
// per-m bias (o.row_bias) is the same for every thread of the warp.
template <int KIND, bool ACT = true>
__device__ __forceinline__ void finish16_tr(const OutDesc& o, int row, int n, int m0, const uint32_t* r,
                                            float row_scale, float cs, float bias_n) {
  if (n >= o.N) return;
  const int c0 = row * kTile + m0;   // first output column (a row index of A)
  const int cols = o.M - c0;         // columns left
  if (cols <= 0) return;
  float v[16];
  finished<KIND, 8, ACT>(o, c0, r, row_scale, cs, bias_n, v);
  const size_t first = (size_t)n * o.ldc + c0;
  if (o.dtype == VOID_OUT_F32) {
    float* dst = reinterpret_cast<float*>(o.out) + first;
    if (cols >= 16 && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
#pragma unroll
      for (int k = 0; k < 16; k += 4) *reinterpret_cast<float4*>(dst + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (k < cols) dst[k] = v[k];
    }
  } else {
    uint32_t h[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (o.dtype == VOID_OUT_F16) {
        const __half2 t = __floats2half2_rn(v[2 * k], v[2 * k + 1]);
        h[k] = *reinterpret_cast<const uint32_t*>(&t);
      } else {
        const __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
        h[k] = *reinterpret_cast<const uint32_t*>(&t);
      }
    }
    uint16_t* dst = reinterpret_cast<uint16_t*>(o.out) + first;
    if (cols >= 16 && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint4*>(dst + 8) = make_uint4(h[4], h[5], h[6], h[7]);
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (k < cols) dst[k] = (uint16_t)(h[k >> 1] >> ((k & 1) * 16));
    }
  }
}

}  // namespace vb
