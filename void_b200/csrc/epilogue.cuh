// Epilogue of the tensor-memory product kernels: raw accumulators of one output column n and a few tile rows m to finished
// values of C (dequantise, bias, activation, conversion), stored directly, through a staging tile, or transposed.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "../../include/void_b200.h"

namespace vb {

constexpr int kTile = 32;
constexpr int kTileBytes = 1024;
constexpr int kPanelN = 128;
constexpr int kPanelBytes = kTile * kPanelN;  // 4096

// GELU in the tanh form written with a sigmoid, void/fusion.py:38-43.  exp and the reciprocal use
// the hardware approximations (a few ulp; far inside the path's 1e-3 bar): with the full-precision
// versions this epilogue, run by two warps per scheduler, cost more than the product itself.
__device__ __forceinline__ float fast_sigmoid(float x) { return __fdividef(1.0f, 1.0f + __expf(-x)); }
__device__ __forceinline__ float gelu_tanh_sigmoid(float x) {
  // x * 0.5 * (1 + (2 sigmoid(2u) - 1)) = x * sigmoid(2u),  2u = 1.5957691216 (x + 0.044715 x^3)
  const float two_u = 1.5957691216f * x * fmaf(0.044715f * x, x, 1.0f);
  return x * fast_sigmoid(two_u);
}
// One value, for the kernels whose epilogue is no loop over registers.
__device__ __forceinline__ float activate(float x, int act) {
  if (act == VOID_ACT_RELU) return fmaxf(x, 0.0f);
  if (act == VOID_ACT_GELU) return gelu_tanh_sigmoid(x);
  if (act == VOID_ACT_SILU) return x * fast_sigmoid(x);
  return x;
}
// What an epilogue thread needs to know about C, read from the kernel parameters once.
struct OutDesc {
  void* out;
  long long ldc;
  void* acc_out;
  const float* row_bias;  // [M] added per output row before the activation (linear-layer bias), or null
  int M, N, dtype, act;
};
// Store eight finished values of output column n: matrix rows row*32 + m0 .. + 7.
__device__ __forceinline__ void store8(const OutDesc& o, int row, int n, int m0, float (&v)[8]) {
  const int r0 = row * kTile + m0;
  const int rows = o.M - r0;  // rows left below r0
  if (o.row_bias != nullptr) {
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < rows) v[k] += __ldg(o.row_bias + r0 + k);
  }
  switch (o.act) {
    case VOID_ACT_RELU:
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = fmaxf(v[k], 0.0f);
      break;
    case VOID_ACT_GELU:
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = gelu_tanh_sigmoid(v[k]);
      break;
    case VOID_ACT_SILU:
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = v[k] * fast_sigmoid(v[k]);
      break;
    default:
      break;
  }
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
  float v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float x = (KIND == VOID_KIND_I8) ? __int2float_rn((int)r[k]) : __uint_as_float(r[k]);
    v[k] = (x * row_scale) * cs + bias;
  }
  store8(o, row, n, m0, v);
}

// Fast epilogue of sixteen raw accumulators of output column n (tile rows m0 .. m0 + 15) straight to C
// (no raw-accumulator dump, no split row), stores specialised per output type.
template <int KIND>
__device__ __forceinline__ void finish16(const OutDesc& o, int row, int n, int m0, const uint32_t* r,
                                         float row_scale, float cs, float bias) {
  if (n >= o.N) return;
  float v[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float x = (KIND == VOID_KIND_I8) ? __int2float_rn((int)r[k]) : __uint_as_float(r[k]);
    v[k] = (x * row_scale) * cs + bias;
  }
  const int r0 = row * kTile + m0;
  const int rows = o.M - r0;
  if (o.row_bias != nullptr) {
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k < rows) v[k] += __ldg(o.row_bias + r0 + k);
  }
  if (o.act != VOID_ACT_NONE) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      if (o.act == VOID_ACT_GELU) v[k] = gelu_tanh_sigmoid(v[k]);
      else if (o.act == VOID_ACT_RELU) v[k] = fmaxf(v[k], 0.0f);
      else v[k] = v[k] * fast_sigmoid(v[k]);
    }
  }
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

// Sixteen finished 16-bit values of output column n into a staging tile [32 m][PITCH n] in shared memory
// (stage_col points at element [0][n - n0]); same arithmetic as finish16.
template <int KIND, int PITCH>
__device__ __forceinline__ void finish16_stage(const OutDesc& o, int row, int n, int m0, const uint32_t* r,
                                               float row_scale, float cs, float bias, uint16_t* stage_col) {
  float v[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float x = (KIND == VOID_KIND_I8) ? __int2float_rn((int)r[k]) : __uint_as_float(r[k]);
    v[k] = (x * row_scale) * cs + bias;
  }
  const int r0 = row * kTile + m0;
  const int rows = o.M - r0;
  if (o.row_bias != nullptr) {
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k < rows) v[k] += __ldg(o.row_bias + r0 + k);
  }
  if (o.act != VOID_ACT_NONE) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      if (o.act == VOID_ACT_GELU) v[k] = gelu_tanh_sigmoid(v[k]);
      else if (o.act == VOID_ACT_RELU) v[k] = fmaxf(v[k], 0.0f);
      else v[k] = v[k] * fast_sigmoid(v[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    uint16_t h;
    if (o.dtype == VOID_OUT_F16) h = __half_as_ushort(__float2half_rn(v[k]));
    else h = __bfloat16_as_ushort(__float2bfloat16_rn(v[k]));
    stage_col[(m0 + k) * PITCH] = h;
  }
}

// Transposed output (C stored as [N, M], m contiguous): the thread owns output row n and sixteen consecutive
// columns m0 .. m0 + 15 of it, so the values leave in 16-byte stores.  bias_n is the bias of this n, the
// per-m bias (o.row_bias) is the same for every thread of the warp.
template <int KIND>
__device__ __forceinline__ void finish16_tr(const OutDesc& o, int row, int n, int m0, const uint32_t* r,
                                            float row_scale, float cs, float bias_n) {
  if (n >= o.N) return;
  const int c0 = row * kTile + m0;   // first output column (a row index of A)
  const int cols = o.M - c0;         // columns left
  if (cols <= 0) return;
  float v[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float x = (KIND == VOID_KIND_I8) ? __int2float_rn((int)r[k]) : __uint_as_float(r[k]);
    v[k] = (x * row_scale) * cs + bias_n;
  }
  if (o.row_bias != nullptr) {
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k < cols) v[k] += __ldg(o.row_bias + c0 + k);
  }
  if (o.act != VOID_ACT_NONE) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      if (o.act == VOID_ACT_GELU) v[k] = gelu_tanh_sigmoid(v[k]);
      else if (o.act == VOID_ACT_RELU) v[k] = fmaxf(v[k], 0.0f);
      else v[k] = v[k] * fast_sigmoid(v[k]);
    }
  }
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
