// Products with few columns (one token, a handful of activations):  C = act(dequant(A . B) + bias), N small.
//
// The tensor-memory kernels of pipeline.cuh multiply 128 columns of B whatever N is and stream a tile row through one CTA's
// ring, a stage's round trip (1.2 us) at a time: 15 us for a decode step whose bytes take 2.  Here a CTA takes one tile
// row and up to 32 columns, its warps share the row's tiles, every warp keeps its sums in registers (mma.sync,
// D[32 x 8 NG] += tile[32 x 32] . B[32 x 8 NG]) and the warps' sums meet in shared memory once, before the epilogue.
// The time is a chain of four memory latencies (row range, block columns, B, store) plus A's bytes.
//
// A is the packed store of pipeline.cuh, read straight into fragments: which k a lane holds in which register is free as long
// as A and B agree, so lane (g, t) = (lane / 4, lane % 4) takes the t-th contiguous piece of row g's 32 k:
//   8-bit   8 k   (8 bytes: one mma.m16n8k32 per 16 rows)
//   16-bit  8 k   (16 bytes: two mma.m16n8k16)
//   32-bit  4 + 4 k (two 16-byte pieces: four mma.m16n8k8, TF32)
// and every load of a warp covers whole 128-byte lines.  B stored [N, K] (TR) is read the same way; B stored [K, N] is read
// NG columns per lane and k-row and turned in registers (byte permutes), column n = NG * j + i being column j of the
// i-th mma, so no shared memory and no transposed copy is needed.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/void_b200.h"
#include "epilogue.cuh"
#include "kinds.cuh"
#include "launch.cuh"
#include "ptx.cuh"
#include "skinny.cuh"

namespace vb {

namespace {

template <int KIND>
struct AccType { using T = float; };
template <>
struct AccType<VOID_KIND_I8> { using T = int; };

// one mma of 32 bytes of k: D (4 accumulators) += A (16 rows) . B (8 columns)
template <int KIND, typename T>
__device__ __forceinline__ void mma32(T (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (KIND == VOID_KIND_I8)
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else if constexpr (KIND == VOID_KIND_F8E4M3)
    asm("mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else if constexpr (KIND == VOID_KIND_F16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else if constexpr (KIND == VOID_KIND_BF16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Words of a lane per 32 k of one row: 2 (8-bit), 4 (16-bit), 8 (32-bit), in the order the mma's take them:
// mma i uses words [2 i] and [2 i + 1] as its two k halves.
template <int ES>
__device__ __forceinline__ void order_words(uint32_t (&w)[2 * ES]) {
  if constexpr (ES == 4) {   // pieces of k = 4 t + i and 16 + 4 t + i: mma i takes one element of each
    const uint32_t v[8] = {w[0], w[4], w[1], w[5], w[2], w[6], w[3], w[7]};
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = v[i];
  }
}
// A: row group rg (8 rows) of a packed tile
template <int ES>
__device__ __forceinline__ void load_a(const uint8_t* tile, int rg, int g, int t, uint32_t (&w)[2 * ES]) {
  const uint8_t* p = tile + rg * (256 * ES);
  if constexpr (ES == 1) {
    const uint2 v = *reinterpret_cast<const uint2*>(p + (t >> 1) * 128 + g * 16 + (t & 1) * 8);
    w[0] = v.x; w[1] = v.y;
  } else {
#pragma unroll
    for (int h = 0; h < ES / 2; ++h) {
      const uint4 v = *reinterpret_cast<const uint4*>(p + (h * 4 + t) * 128 + g * 16);
      w[4 * h] = v.x; w[4 * h + 1] = v.y; w[4 * h + 2] = v.z; w[4 * h + 3] = v.w;
    }
    order_words<ES>(w);
  }
}
// B stored [N, K]: 32 k of row n, starting at element k0; elements at k >= K are zero
template <int ES>
__device__ __forceinline__ void load_b_tr(const uint8_t* row, int k0, int K, int t, bool ok, uint32_t (&w)[2 * ES]) {
#pragma unroll
  for (int i = 0; i < 2 * ES; ++i) w[i] = 0u;
  if (!ok || k0 < 0) return;
  if (k0 + 32 <= K) {
    if constexpr (ES == 1) {
      const uint2 v = *reinterpret_cast<const uint2*>(row + k0 + 8 * t);
      w[0] = v.x; w[1] = v.y;
    } else {
#pragma unroll
      for (int h = 0; h < ES / 2; ++h) {
        const uint4 v = *reinterpret_cast<const uint4*>(row + (size_t)k0 * ES + (h * 4 + t) * 16);
        w[4 * h] = v.x; w[4 * h + 1] = v.y; w[4 * h + 2] = v.z; w[4 * h + 3] = v.w;
      }
    }
  } else {   // the last columns of a K that is no multiple of 32
#pragma unroll
    for (int i = 0; i < 2 * ES; ++i) {
      const int piece = (ES == 1) ? 8 * t + 4 * i : ((i >> 2) * 4 + t) * 16 + (i & 3) * 4;   // byte offset of the word
#pragma unroll
      for (int e = 0; e < 4 / ES; ++e) {
        const int k = k0 + piece / ES + e;
        if (k < K) {
          const uint8_t* p = row + (size_t)k * ES;
          const uint32_t v = ES == 1 ? *p : (ES == 2 ? *reinterpret_cast<const uint16_t*>(p) : *reinterpret_cast<const uint32_t*>(p));
          w[i] |= v << (8 * ES * e);
        }
      }
    }
  }
  order_words<ES>(w);
}
// B stored [K, N]: columns n .. n + NG - 1 of the lane's k's, turned into the words of NG mma columns
template <int ES, int NG>
__device__ __forceinline__ void load_b(const uint8_t* b, long long ldb, int k0, int K, int n, int N, int t, uint32_t (&w)[NG][2 * ES]) {
  constexpr int RB = NG * ES;            // bytes of a k-row a lane reads
  constexpr int RW = (RB + 3) / 4;       // words
  uint32_t r[8][RW];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = k0 + (ES == 4 ? (i >> 2) * 16 + 4 * t + (i & 3) : 8 * t + i);
#pragma unroll
    for (int j = 0; j < RW; ++j) r[i][j] = 0u;
    if ((unsigned)k < (unsigned)K && n < N) {
      const uint8_t* p = b + (long long)k * ldb + (size_t)n * ES;
      if (n + NG <= N) {
        if constexpr (RB == 16) { const uint4 v = *reinterpret_cast<const uint4*>(p); r[i][0] = v.x; r[i][1] = v.y; r[i][2] = v.z; r[i][3] = v.w; }
        else if constexpr (RB == 8) { const uint2 v = *reinterpret_cast<const uint2*>(p); r[i][0] = v.x; r[i][1] = v.y; }
        else if constexpr (RB == 4) r[i][0] = *reinterpret_cast<const uint32_t*>(p);
        else if constexpr (RB == 2) r[i][0] = *reinterpret_cast<const uint16_t*>(p);
        else r[i][0] = *p;
      } else {
#pragma unroll
        for (int e = 0; e < NG; ++e)
          if (n + e < N) {
            const uint8_t* q = p + e * ES;
            const uint32_t v = ES == 1 ? *q : (ES == 2 ? *reinterpret_cast<const uint16_t*>(q) : *reinterpret_cast<const uint32_t*>(q));
            r[i][e * ES / 4] |= v << (8 * ((e * ES) & 3));
          }
      }
    }
  }
  if constexpr (ES == 4) {
#pragma unroll
    for (int c = 0; c < NG; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) { w[c][2 * i] = r[i][c]; w[c][2 * i + 1] = r[4 + i][c]; }
  } else if constexpr (ES == 2) {
#pragma unroll
    for (int c = 0; c < NG; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) w[c][i] = __byte_perm(r[2 * i][c / 2], r[2 * i + 1][c / 2], (c & 1) ? 0x7632 : 0x5410);
  } else {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t lo0 = __byte_perm(r[4 * i][0], r[4 * i + 1][0], 0x5140), lo1 = __byte_perm(r[4 * i + 2][0], r[4 * i + 3][0], 0x5140);
      w[0][i] = __byte_perm(lo0, lo1, 0x5410);
      if constexpr (NG > 1) w[1][i] = __byte_perm(lo0, lo1, 0x7632);
      if constexpr (NG > 2) {
        const uint32_t hi0 = __byte_perm(r[4 * i][0], r[4 * i + 1][0], 0x7362), hi1 = __byte_perm(r[4 * i + 2][0], r[4 * i + 3][0], 0x7362);
        w[2][i] = __byte_perm(hi0, hi1, 0x5410);
        w[3][i] = __byte_perm(hi0, hi1, 0x7632);
      }
    }
  }
}

// ACT: whether there may be an activation or a row bias (the kernel without is 0.2 us faster).
template <int KIND, bool TR, int NG, bool ACT>
__global__ void __launch_bounds__(512) skinny_kernel(const __grid_constant__ SkinnyParams p) {
  constexpr int ES = Elem<KIND>::ES, NB = 8 * NG;
  using T = typename AccType<KIND>::T;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  T* red = reinterpret_cast<T*>(smem_raw);   // [warps][32][NB + 1]
  constexpr int PITCH = NB + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int row = blockIdx.x, n0 = blockIdx.y * NB;
  if (!p.a_stable) grid_dependency_wait();
  const int t0 = p.row_ptr[row], t1 = p.row_ptr[row + 1];
  T d[2][NG][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < NG; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) d[h][i][e] = T(0);
  const int terms = KIND == VOID_KIND_F8E4M3 ? p.terms : 1;
  const uint8_t* b = p.b;
  int cols = 0;    // block columns of this warp's next 32 tiles, one per lane
  if (t0 + warp + lane * warps < t1) cols = p.tile_cols[t0 + warp + lane * warps];
  if (p.a_stable) grid_dependency_wait();
  int seen = 0;
#pragma unroll 2
  for (int tile = t0 + warp; tile < t1; tile += warps, ++seen) {
    if (seen == 32) {
      seen = 0;
      cols = 0;
      if (tile + lane * warps < t1) cols = p.tile_cols[tile + lane * warps];
    }
    const int k0 = __shfl_sync(0xffffffffu, cols, seen) * 32;
    uint32_t bw[NG][2 * ES];
    if constexpr (TR) {
#pragma unroll
      for (int i = 0; i < NG; ++i) {
        const int n = n0 + 8 * i + g;
        load_b_tr<ES>(b + (long long)n * p.ldb, k0, p.K, t, n < p.N, bw[i]);
      }
    } else {
      load_b<ES, NG>(b, p.ldb, k0, p.K, n0 + NG * g, p.N, t, bw);
    }
    const uint8_t* a = p.tiles + (size_t)tile * (size_t)(1024 * ES * terms);
    for (int v = 0; v < terms; ++v, a += 1024 * ES) {
      uint32_t aw[4][2 * ES];
#pragma unroll
      for (int rg = 0; rg < 4; ++rg) load_a<ES>(a, rg, g, t, aw[rg]);
#pragma unroll
      for (int i = 0; i < NG; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int q = 0; q < ES; ++q)
            mma32<KIND>(d[h][i], aw[2 * h][2 * q], aw[2 * h + 1][2 * q], aw[2 * h][2 * q + 1], aw[2 * h + 1][2 * q + 1],
                        bw[i][2 * q], bw[i][2 * q + 1]);
    }
  }
  struct Output { int m, c, n, r; bool in; float cs, bias, row_bias; };
  auto output = [&](int o) {
    Output x;
    x.m = TR ? (o & 31) : o / NB;
    x.c = TR ? (o >> 5) : o % NB;
    x.n = n0 + x.c;
    x.r = row * 32 + x.m;
    x.in = x.n < p.N && x.r < p.M;
    x.cs = p.b_scale;
    x.bias = x.row_bias = 0.0f;
    if (x.in) {
      if (p.col_scale != nullptr) x.cs *= p.col_scale[x.n];
      if (p.bias != nullptr) x.bias = p.bias[x.n];
      if (ACT && p.row_bias != nullptr) x.row_bias = p.row_bias[x.r];
    }
    return x;
  };
  // (biases are on their way while the warps' sums are put together; a column scale alone is better read with them)
  Output x;
  if (ACT) x = output(threadIdx.x);
  // (late: a product that starts beside this one's first CTAs takes the places of those still to come; fp16 8192 x 2048,
  // N = 8 4.7 -> 3.9 us, 2048 x 8192 6.4 -> 4.8)
  grid_launch_dependents();
  // this warp's sums, [m][column]: d[h][i] holds rows 16 h + g (+ 8) and columns j = 2 t (+ 1) of mma i
  T* mine = red + warp * (32 * PITCH);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < NG; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = 16 * h + g + 8 * (e >> 1), j = 2 * t + (e & 1);
        mine[m * PITCH + (TR ? 8 * i + j : NG * j + i)] = d[h][i][e];
      }
  __syncthreads();
  const float rs = p.row_scale != nullptr && t1 > t0 ? p.row_scale[row] : 1.0f;
  for (int o = threadIdx.x; o < 32 * NB; o += blockDim.x) {
    if (!ACT || o >= (int)blockDim.x) x = output(o);
    if (!x.in) continue;
    T s = T(0);
    for (int w = 0; w < warps; ++w) s += red[(w * 32 + x.m) * PITCH + x.c];
    float v = KIND == VOID_KIND_I8 ? __int2float_rn((int)s) : (float)s;
    v = (v * rs) * x.cs + x.bias;
    if constexpr (ACT) v = activate(v + x.row_bias, p.act);
    const long long at = TR ? (long long)x.n * p.ldc + x.r : (long long)x.r * p.ldc + x.n;
    if (p.out_dtype == VOID_OUT_F16) reinterpret_cast<__half*>(p.out)[at] = __float2half_rn(v);
    else if (p.out_dtype == VOID_OUT_BF16) reinterpret_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(v);
    else reinterpret_cast<float*>(p.out)[at] = v;
  }
}

template <int KIND, bool TR, int NG, bool ACT>
cudaError_t launch(const SkinnyParams& p, int nbr, int warps, cudaStream_t st) {
  auto kernel = skinny_kernel<KIND, TR, NG, ACT>;
  const int smem = warps * 32 * (8 * NG + 1) * 4;
  if (smem > 48 * 1024 && ensure_smem((const void*)kernel, smem)) return cudaErrorInvalidValue;
  return launch_pdl(kernel, dim3((unsigned)nbr, (unsigned)((p.N + 8 * NG - 1) / (8 * NG))), 32 * warps, smem, st, p);
}
template <int KIND, bool TR, int NG>
cudaError_t launch(const SkinnyParams& p, int nbr, int warps, cudaStream_t st) {
  return p.act != VOID_ACT_NONE || p.row_bias != nullptr ? launch<KIND, TR, NG, true>(p, nbr, warps, st) : launch<KIND, TR, NG, false>(p, nbr, warps, st);
}
template <int KIND, bool TR>
cudaError_t launch_columns(const SkinnyParams& p, int nbr, int warps, cudaStream_t st) {
  if (p.N <= 8) return launch<KIND, TR, 1>(p, nbr, warps, st);
  if (p.N <= 16) return launch<KIND, TR, 2>(p, nbr, warps, st);
  return launch<KIND, TR, 4>(p, nbr, warps, st);
}

}  // namespace

cudaError_t skinny_launch(const SkinnyParams& p, int kind, bool transposed, int nbr, long long nnz, cudaStream_t st) {
  // enough warps that a warp has a few tiles of its row, so that their loads are in flight together
  const long long avg = nbr > 0 ? nnz / nbr : 0;
  const int warps = avg >= 24 ? 16 : (avg >= 6 ? 8 : 4);
  switch (kind) {
    case VOID_KIND_I8: return transposed ? launch_columns<VOID_KIND_I8, true>(p, nbr, warps, st) : launch_columns<VOID_KIND_I8, false>(p, nbr, warps, st);
    case VOID_KIND_F8E4M3: return transposed ? cudaErrorInvalidValue : launch_columns<VOID_KIND_F8E4M3, false>(p, nbr, warps, st);
    case VOID_KIND_F16: return transposed ? launch_columns<VOID_KIND_F16, true>(p, nbr, warps, st) : launch_columns<VOID_KIND_F16, false>(p, nbr, warps, st);
    case VOID_KIND_BF16: return transposed ? launch_columns<VOID_KIND_BF16, true>(p, nbr, warps, st) : launch_columns<VOID_KIND_BF16, false>(p, nbr, warps, st);
    default: return transposed ? launch_columns<VOID_KIND_TF32, true>(p, nbr, warps, st) : launch_columns<VOID_KIND_TF32, false>(p, nbr, warps, st);
  }
}

}  // namespace vb
