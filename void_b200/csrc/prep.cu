// Preparation kernels of the SpMM path: tile index (row_ptr / block_indices), packing of the
// Morton-ordered tiles into tile-row-major core-matrix order, the INT8 / FP8-E4M3 quantisers
// for A tiles and for the columns of B, and the Stream-K worker table.  All of them are
// bandwidth-bound elementwise or gather kernels; none waits on another CTA.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <atomic>

#include "../../include/void_b200.h"
#include "epilogue.cuh"
#include "launch.cuh"

namespace vb {

static inline cudaStream_t as_stream(void_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

// Exclusive prefix sum of n int32 values by ONE block of 1024 threads; out[n] = total.
// in and out may alias.
__device__ void block_exclusive_scan(const int32_t* in, int32_t* out, int n) {
  __shared__ int32_t part[1024];
  const int tid = threadIdx.x;
  const int per = (n + 1023) / 1024;
  const int lo = tid * per < n ? tid * per : n;
  const int hi = (lo + per) < n ? (lo + per) : n;
  int32_t s = 0;
  for (int i = lo; i < hi; ++i) s += in[i];
  part[tid] = s;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    const int32_t v = (tid >= off) ? part[tid - off] : 0;
    __syncthreads();
    part[tid] += v;
    __syncthreads();
  }
  int32_t run = part[tid] - s;  // exclusive prefix of this thread's chunk
  for (int i = lo; i < hi; ++i) {
    const int32_t v = in[i];
    out[i] = run;
    run += v;
  }
  if (tid == 1023) out[n] = part[1023];
  __syncthreads();
}

// ------------------------------------------------------------------------------ tile index
// Coordinates outside the block grid are skipped here and in rank_tiles_kernel: the caller sees them (and
// repeated coordinates, which set one bit twice) as row_ptr[nbr] < nnz.
__global__ void mark_tiles_kernel(const int32_t* __restrict__ brow, const int32_t* __restrict__ bcol, int64_t nnz,
                                  int nbr, int nbc, int wpr, uint32_t* __restrict__ bitmap,
                                  int32_t* __restrict__ block_indices) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nnz) return;
  block_indices[i] = 0;   // every entry is a valid position even when the list is rejected afterwards
  const int r = brow[i], c = bcol[i];
  if ((unsigned)r >= (unsigned)nbr || (unsigned)c >= (unsigned)nbc) return;
  atomicOr(bitmap + (size_t)r * wpr + (c >> 5), 1u << (c & 31));
}

__global__ void count_rows_kernel(const uint32_t* __restrict__ bitmap, int nbr, int wpr, int32_t* __restrict__ counts) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= nbr) return;
  int c = 0;
  for (int w = lane; w < wpr; w += 32) c += __popc(bitmap[(size_t)warp * wpr + w]);
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (lane == 0) counts[warp] = c;
}

__global__ void __launch_bounds__(1024) scan_rows_kernel(const int32_t* counts, int32_t* row_ptr, int nbr) {
  block_exclusive_scan(counts, row_ptr, nbr);
}

// both in one launch, for bitmaps one block reads in a couple of microseconds
constexpr int kOneBlockBitmap = 32768;   // words
__global__ void __launch_bounds__(1024) count_scan_rows_kernel(const uint32_t* __restrict__ bitmap, int nbr, int wpr,
                                                               int32_t* __restrict__ counts, int32_t* __restrict__ row_ptr) {
  const int per = (nbr + 1023) / 1024;
  for (int r = threadIdx.x * per; r < (int)(threadIdx.x + 1) * per && r < nbr; ++r) {
    int c = 0;
    for (int w = 0; w < wpr; ++w) c += __popc(bitmap[(size_t)r * wpr + w]);
    counts[r] = c;
  }
  __syncthreads();
  block_exclusive_scan(counts, row_ptr, nbr);
}

__global__ void rank_tiles_kernel(const int32_t* __restrict__ brow, const int32_t* __restrict__ bcol, int64_t nnz,
                                  int nbr, int nbc, int wpr, const uint32_t* __restrict__ bitmap,
                                  const int32_t* __restrict__ row_ptr, int32_t* __restrict__ block_indices) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nnz) return;
  const int r = brow[i], c = bcol[i];
  if ((unsigned)r >= (unsigned)nbr || (unsigned)c >= (unsigned)nbc) return;
  const uint32_t* row = bitmap + (size_t)r * wpr;
  int rank = 0;
  for (int w = 0; w < (c >> 5); ++w) rank += __popc(row[w]);
  rank += __popc(row[c >> 5] & ((1u << (c & 31)) - 1u));
  block_indices[row_ptr[r] + rank] = (int32_t)i;
}

// All of the above by one block, the bitmap in shared memory beside the number of tiles ahead of each of its words (16 bits), for
// the lists that most matrices have.  A tile's place is one word's sum and one word's bits, however wide the grid; rows lie an odd
// number of words apart, so that neighbouring ones start on different banks.  (Adding up a row's words for every tile took 58 us for
// 8000 tiles of a 363 x 1024 grid, now 8.1, and 353 for 16384 of 93 x 4096.)
// Bound by one SM's two passes over the list, about 0.4 us per thousand tiles, so longer lists go to the kernels above, which
// spread over the device.  us for the index, this kernel and those: 128 x 128 grid, 3277 tiles 4.2 10.4, 8000 5.2 10.5; 256 x 256,
// 8192 6.1 7.8, 16384 9.4 8.0; 512 x 512, 8192 7.3 10.3, 16384 11.5 10.3; 1000 x 333, 8192 7.7 8.8, 16384 11.8 9.1; 363 x 1024,
// 8192 8.1 16.0; 960 x 512, 8192 8.5 12.3.  Where the bitmap is small those are slow with 16384 as well: 128 x 128 8.4 11.2, 64 x 512
// 8.6 12.4, but 160 x 256 (1440 words) 9.1 8.4.
constexpr int kOneBlockTiles = 8192, kOneBlockWords = 16384;                // words: those of the bitmap, rows padded
constexpr int kOneBlockManyTiles = 16384, kOneBlockFewWords = 1100;
constexpr int kOneBlockOrder = 256;   // tile rows one block puts in order, a quarter of its threads: 128 rows 0.9 us, 256 1.3
static bool one_block_index(int64_t nnz, int64_t words) {
  return words <= kOneBlockWords && nnz <= (words <= kOneBlockFewWords ? kOneBlockManyTiles : kOneBlockTiles);
}
constexpr int one_block_pitch(int wpr) { return wpr | 1; }
constexpr int one_block_smem(int words) { return words * 4 + (words + 2) / 2 * 4; }
__global__ void __launch_bounds__(1024) tile_index_kernel(const int32_t* brow, const int32_t* bcol, int nnz,
                                                          int nbr, int nbc, int pitch, int32_t* row_ptr,
                                                          int32_t* block_indices, int32_t* row_order) {
  extern __shared__ uint32_t bits[];   // [nbr][pitch], then the tiles ahead of every word and of the end
  __shared__ int32_t warp_sum[32];
  __shared__ __align__(16) uint32_t key[kOneBlockOrder];
  const int words = nbr * pitch;
  uint16_t* ahead = reinterpret_cast<uint16_t*>(bits + words);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int i = tid; i < words; i += 1024) bits[i] = 0u;
  grid_dependency_wait();
  __syncthreads();
#pragma unroll 4
  for (int i = tid; i < nnz; i += 1024) {
    const int r = brow[i], c = bcol[i];
    block_indices[i] = 0;   // every entry is a valid position even when the list is rejected afterwards
    if ((unsigned)r < (unsigned)nbr && (unsigned)c < (unsigned)nbc) atomicOr(bits + r * pitch + (c >> 5), 1u << (c & 31));
  }
  __syncthreads();
  const int per = (words + 1023) / 1024 | 1, lo = tid * per < words ? tid * per : words, hi = lo + per < words ? lo + per : words;
  int sum = 0;
  for (int w = lo; w < hi; ++w) sum += __popc(bits[w]);
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int v = warp_sum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    warp_sum[lane] = v;
  }
  __syncthreads();
  int run = (wid ? warp_sum[wid - 1] : 0) + incl - sum;
  for (int w = lo; w < hi; ++w) {
    ahead[w] = (uint16_t)run;
    run += __popc(bits[w]);
  }
  if (tid == 1023) ahead[words] = (uint16_t)run;
  __syncthreads();
  for (int r = tid; r <= nbr; r += 1024) row_ptr[r] = ahead[r * pitch];
  if (row_order != nullptr) {   // as row_order_kernel: a row comes after all rows with a larger key, four threads count them
    if (tid < kOneBlockOrder) key[tid] = tid < nbr ? (uint32_t)(ahead[(tid + 1) * pitch] - ahead[tid * pitch]) * kOneBlockOrder + (kOneBlockOrder - 1 - tid) : 0u;
    __syncthreads();
    const int r = tid >> 2;
    const uint32_t mine = key[r];
    int before = 0;
    for (int i = tid & 3; i < (nbr + 3) / 4; i += 4) {
      const uint4 k = reinterpret_cast<const uint4*>(key)[i];
      before += (k.x > mine ? 1 : 0) + (k.y > mine ? 1 : 0) + (k.z > mine ? 1 : 0) + (k.w > mine ? 1 : 0);
    }
    before += __shfl_xor_sync(0xffffffffu, before, 1);
    before += __shfl_xor_sync(0xffffffffu, before, 2);
    if ((tid & 3) == 0 && r < nbr) row_order[before] = r;
  }
#pragma unroll 4
  for (int i = tid; i < nnz; i += 1024) {
    const int r = brow[i], c = bcol[i];
    if ((unsigned)r >= (unsigned)nbr || (unsigned)c >= (unsigned)nbc) continue;
    const int w = r * pitch + (c >> 5);
    block_indices[ahead[w] + __popc(bits[w] & ((1u << (c & 31)) - 1u))] = i;
  }
}

// ------------------------------------------------------------------------------ pack
// One thread per 16-byte chunk of the packed tile.  Packed chunk q of a tile holds bytes
// [c16*16, c16*16+16) of tile row r with  q = (r/8)*16 + c16*8 + (r%8): four groups of eight
// rows, each group stored as two 8x16-byte core matrices (k bytes 0..15, then 16..31).
// The first thread of a tile also gathers its block column and scale.
struct TileMeta {
  const int32_t* block_cols;
  const float* scales;     // null: 1
  int64_t n_scales;        // 1 (one scale for all tiles) or one per tile
  int32_t* tile_cols;      // null: not wanted
  float* tile_scales;      // null: not wanted
};
__device__ __forceinline__ float tile_scale(const TileMeta& m, int64_t src) {
  return m.scales == nullptr ? 1.0f : m.scales[m.n_scales == 1 ? 0 : src];
}
__device__ __forceinline__ void put_meta(const TileMeta& m, int64_t packed, int64_t src) {
  if (m.tile_cols != nullptr) m.tile_cols[packed] = m.block_cols[src];
  if (m.tile_scales != nullptr) m.tile_scales[packed] = tile_scale(m, src);
}
// Row scales, a warp per tile row, by the blocks behind those that pack: the mean of the row's tile scales, added one by one
// in row order like the reference's loop.
struct RowScales {
  const int32_t* row_ptr;
  float* row_scale;        // null: not wanted
  int nbr;
  unsigned pack_blocks;
};
__device__ __forceinline__ void mean_scale(const RowScales& rows, const TileMeta& meta, const int32_t* block_indices) {
  const int r = (int)(((blockIdx.x - rows.pack_blocks) * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (r >= rows.nbr) return;
  const int t0 = rows.row_ptr[r], t1 = rows.row_ptr[r + 1];
  float s = 0.0f;
  for (int t = t0; t < t1; t += 32) {
    const float x = t + lane < t1 ? tile_scale(meta, block_indices[t + lane]) : 0.0f;
    const int n = t1 - t < 32 ? t1 - t : 32;
    for (int k = 0; k < n; ++k) s = __fadd_rn(s, __shfl_sync(0xffffffffu, x, k));
  }
  if (lane == 0) rows.row_scale[r] = t1 > t0 ? __fdiv_rn(s, (float)(t1 - t0)) : 0.0f;
}
// The kernels of a store's set-up (quantised tiles, index, packing, row order) let the next one start when they are through; a
// product packed inside a stream capture follows them without a host's wait in between.
__global__ void __launch_bounds__(256) pack_tiles_kernel(const uint4* values, const int32_t* block_indices, int64_t nnz, uint4* packed,
                                                         TileMeta meta, RowScales rows) {
  grid_dependency_wait();
  if (blockIdx.x >= rows.pack_blocks) {
    mean_scale(rows, meta, block_indices);
    return;
  }
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nnz * 64) return;
  const int64_t j = g >> 6;
  const int q = (int)(g & 63);
  const int r = (q >> 4) * 8 + (q & 7);
  const int c16 = (q >> 3) & 1;
  const int64_t src_tile = block_indices[j];
  packed[g] = values[src_tile * 64 + r * 2 + c16];
  if (q == 0) put_meta(meta, j, src_tile);
}

// The same for elements of ES bytes: a tile row holds KC = 2*ES 16-byte chunks, a packed tile
// 64*ES of them in the order [row / 8][chunk][row % 8].
template <int ES>
__global__ void pack_tiles_fp_kernel(const uint4* __restrict__ values, const int32_t* __restrict__ block_indices,
                                     int64_t nnz, uint4* __restrict__ packed, TileMeta meta) {
  constexpr int KC = 2 * ES, PER_TILE = 64 * ES;
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nnz * PER_TILE) return;
  const int64_t j = g / PER_TILE;
  const int q = (int)(g - j * PER_TILE);
  const int r = (q / (8 * KC)) * 8 + (q & 7);
  const int kc = (q >> 3) % KC;
  const int64_t src_tile = block_indices[j];
  uint4 v = values[src_tile * PER_TILE + r * KC + kc];
  if (ES == 4) {
    // The tensor cores read an fp32 operand as TF32 by dropping its low 13 mantissa bits.  Rounding the
    // tiles to the nearest TF32 value here, once, halves the error of that and removes its bias.
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(v.x) : "f"(__uint_as_float(v.x)));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(v.y) : "f"(__uint_as_float(v.y)));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(v.z) : "f"(__uint_as_float(v.z)));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(v.w) : "f"(__uint_as_float(v.w)));
  }
  packed[g] = v;
  if (q == 0) put_meta(meta, j, src_tile);
}

// The packed form of the TRANSPOSED tiles (A^T for the gradient of the dense operand): chunk kc of row r' holds
// T[kc * E + i][r'], i < E = 16 / ES.  A warp takes one chunk column of a tile: every load reads one row of the tile and
// every eight lanes write 128 contiguous bytes.  No transposed copy of the tiles is made first.
template <int ES>
__global__ void pack_tiles_fp_t_kernel(const void* __restrict__ values, const int32_t* __restrict__ block_indices,
                                       int64_t nnz, uint4* __restrict__ packed) {
  constexpr int KC = 2 * ES, E = 16 / ES;
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int r = threadIdx.x & 31;
  const int64_t j = w / KC;
  const int kc = (int)(w - j * KC);
  if (j >= nnz) return;
  const int64_t src = (int64_t)block_indices[j] * 1024 + kc * E * 32 + r;
  uint32_t o[4];
  if constexpr (ES == 4) {
    const float* v = reinterpret_cast<const float*>(values) + src;
#pragma unroll
    for (int i = 0; i < 4; ++i) asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(o[i]) : "f"(v[i * 32]));
  } else {
    const uint16_t* v = reinterpret_cast<const uint16_t*>(values) + src;
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = (uint32_t)v[(2 * i) * 32] | (uint32_t)v[(2 * i + 1) * 32] << 16;
  }
  packed[j * (64 * ES) + ((r >> 3) * KC + kc) * 8 + (r & 7)] = make_uint4(o[0], o[1], o[2], o[3]);
}

// FP8 tiles with their scales folded in, for the row-accumulate kernel: the tensor cores cannot scale a
// product per tile, so each element a * s_tile / R_row (R_row = the largest tile scale of the tile row) is
// written as a sum of `terms` E4M3 numbers - the nearest E4M3 value, then the nearest E4M3 value of what is
// left, and once more for three terms - and every term is multiplied by the same panel of B.  Two terms carry
// 8 significant bits (relative error below 2^-8 per element, unbiased), three carry 12; the differences
// x - hi and (x - hi) - mid are exact in fp32.  The epilogue multiplies the row's sums by R_row.
// One thread per 16-byte chunk of a packed tile, same chunk order as pack_tiles_kernel; term k of packed
// tile j lies at chunk (j * terms + k) * 64.
__device__ __forceinline__ float e4m3_to_float(uint8_t v) {
  return __half2float(__half(__nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)v, __NV_E4M3)));
}
template <int TERMS>
__global__ void pack_tiles_f8_split_kernel(const uint4* __restrict__ values, const float* __restrict__ scales,
                                           int64_t n_scales, const int32_t* __restrict__ block_rows,
                                           const int32_t* __restrict__ block_indices,
                                           const float* __restrict__ row_scale, int64_t nnz, int nbr,
                                           uint4* __restrict__ packed) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nnz * 64) return;
  const int64_t j = g >> 6;
  const int q = (int)(g & 63);
  const int r = (q >> 4) * 8 + (q & 7);
  const int c16 = (q >> 3) & 1;
  const int64_t src = block_indices[j];
  const uint4 v = values[src * 64 + r * 2 + c16];
  const float s = (scales == nullptr) ? 1.0f : (n_scales == 1 ? scales[0] : scales[src]);
  const int row = block_rows[src];
  const float R = (unsigned)row < (unsigned)nbr ? row_scale[row] : 0.0f;   // (the list is checked after it is packed)
  const float ratio = (R > 0.0f) ? __fdiv_rn(s, R) : 0.0f;
  const uint32_t in[4] = {v.x, v.y, v.z, v.w};
  uint32_t out[TERMS][4];
#pragma unroll
  for (int w = 0; w < 4; ++w) {
#pragma unroll
    for (int k = 0; k < TERMS; ++k) out[k][w] = 0u;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float x = __fmul_rn(e4m3_to_float((uint8_t)(in[w] >> (8 * e))), ratio);
#pragma unroll
      for (int k = 0; k < TERMS; ++k) {
        const uint8_t t = (uint8_t)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
        out[k][w] |= (uint32_t)t << (8 * e);
        x = __fsub_rn(x, e4m3_to_float(t));
      }
    }
  }
#pragma unroll
  for (int k = 0; k < TERMS; ++k) packed[(j * TERMS + k) * 64 + q] = make_uint4(out[k][0], out[k][1], out[k][2], out[k][3]);
}

// Sum of the per-rank partial tiles of the tile rows this GPU owns, then the INT8 epilogue.  One block per
// (owned tile row, 128-column panel), one thread per column n: the slots hold int32 tiles [32 m][128 n], so a
// warp reads 128 contiguous bytes per m.  contrib[row] has bit r set when rank r stored a tile for the row
// (a rank without tiles in the row stores nothing and its slot is not read).
__global__ void __launch_bounds__(128) reduce_slots_kernel(const int32_t* __restrict__ slots, const uint8_t* __restrict__ contrib,
                                                           int n_ranks, int rows_owned, int row0, int n_panels,
                                                           int np, const float* __restrict__ row_scale,
                                                           const float* __restrict__ col_scale, float b_scale,
                                                           const float* __restrict__ bias, int act, void* out,
                                                           long long ldc, int out_dtype, int M, int N) {
  const int item = blockIdx.x;                 // local row * n_panels + panel
  const int lr = item / n_panels, pan = item - lr * n_panels;
  if (lr >= rows_owned) return;
  const int n = pan * 128 + threadIdx.x;
  const unsigned mask = contrib[lr];
  int acc[32];
#pragma unroll
  for (int m = 0; m < 32; ++m) acc[m] = 0;
  for (int r = 0; r < n_ranks; ++r) {
    if (!((mask >> r) & 1u)) continue;
    // slots are laid out as the SpMM kernel writes them: [row][chunk of np panels][rank][panel of the chunk]
    const int n_chunks = (n_panels + np - 1) / np;
    const int32_t* t = slots + ((((size_t)lr * n_chunks + pan / np) * n_ranks + r) * np + pan % np) * 4096 + threadIdx.x;
#pragma unroll
    for (int m = 0; m < 32; ++m) acc[m] += __ldcs(t + m * 128);
  }
  if (n >= N) return;
  const int grow = row0 + lr;                  // global tile row
  const float rs = row_scale[grow];
  const float cs = (col_scale != nullptr ? col_scale[n] : 1.0f) * b_scale;
  const float bi = bias != nullptr ? bias[n] : 0.0f;
#pragma unroll
  for (int m = 0; m < 32; ++m) {
    const long long gm = (long long)grow * 32 + m;
    if (gm >= M) break;
    const float v = activate((__int2float_rn(acc[m]) * rs) * cs + bi, act);
    const size_t o = (size_t)(lr * 32 + m) * ldc + n;
    if (out_dtype == VOID_OUT_F16) reinterpret_cast<__half*>(out)[o] = __float2half_rn(v);
    else if (out_dtype == VOID_OUT_BF16) reinterpret_cast<__nv_bfloat16*>(out)[o] = __float2bfloat16_rn(v);
    else reinterpret_cast<float*>(out)[o] = v;
  }
}

// largest tile scale of every tile row (0 for an empty row)
__global__ void row_max_scale_kernel(const int32_t* __restrict__ row_ptr, const float* __restrict__ tile_scales, int nbr,
                                     float* __restrict__ row_scale) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nbr) return;
  float m = 0.0f;
  for (int t = row_ptr[r]; t < row_ptr[r + 1]; ++t) m = fmaxf(m, tile_scales[t]);
  row_scale[r] = m;
}

__global__ void gather_tile_meta_kernel(const int32_t* __restrict__ bcol, const float* __restrict__ scales,
                                        int64_t n_scales, const int32_t* __restrict__ block_indices, int64_t nnz,
                                        int32_t* __restrict__ tile_cols, float* __restrict__ tile_scales) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nnz) return;
  const int64_t src = block_indices[j];
  tile_cols[j] = bcol[src];
  if (tile_scales != nullptr) tile_scales[j] = (scales == nullptr) ? 1.0f : (n_scales == 1 ? scales[0] : scales[src]);
}

// Tile rows by falling tile count, ties in their own order: a row's place is the number of rows that come before it.  One
// warp per row counts them, which for the few thousand rows of a matrix takes less than a sort's launches.
__global__ void row_order_kernel(const int32_t* row_ptr, int nbr, int32_t* order) {
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  grid_dependency_wait();
  if (r >= nbr) return;
  const int mine = row_ptr[r + 1] - row_ptr[r];
  int before = 0;
#pragma unroll 4
  for (int i = lane; i < nbr; i += 32) {
    const int c = row_ptr[i + 1] - row_ptr[i];
    before += (c > mine || (c == mine && i < r)) ? 1 : 0;
  }
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0) order[before] = r;
}

// ------------------------------------------------------------------------------ quantisers
__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ int8_t quant_i8(float x, float scale) {
  float q = rintf(__fdiv_rn(x, scale));
  q = fminf(fmaxf(q, -128.0f), 127.0f);
  return (int8_t)(int)q;
}
// Four values at once, without a division for almost every one.  y = x * (1 / scale) is off the quotient by less than
// 2.4e-5 (|y| <= 128: half an ulp each of the reciprocal, of y and of the quotient), so both round to the same integer
// unless y lies within 3e-5 of a half integer: only then (about one element in 16000) the four are divided.  Rounding is
// the addition of 1.5 * 2^23, which leaves the integer in the low byte of the sum.  Clamping first gives the clamp of the
// rounded value; NaN ends at -128 in both forms.
__device__ __noinline__ uint32_t quant_i8x4_div(float x0, float x1, float x2, float x3, float s0, float s1, float s2, float s3) {
  return (uint32_t)(uint8_t)quant_i8(x0, s0) | (uint32_t)(uint8_t)quant_i8(x1, s1) << 8 |
         (uint32_t)(uint8_t)quant_i8(x2, s2) << 16 | (uint32_t)(uint8_t)quant_i8(x3, s3) << 24;
}
__device__ __forceinline__ uint32_t quant_i8x4(const float4 x, const float4 scale, const float4 inv) {
  constexpr float kRound = 12582912.0f;
  float t[4], d = 0.0f;
  const float xs[4] = {x.x, x.y, x.z, x.w}, is[4] = {inv.x, inv.y, inv.z, inv.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float y = fminf(fmaxf(__fmul_rn(xs[e], is[e]), -128.0f), 127.0f);
    t[e] = __fadd_rn(y, kRound);
    d = fmaxf(d, fabsf(__fsub_rn(y, __fsub_rn(t[e], kRound))));
  }
  if (d > 0.5f - 3e-5f) return quant_i8x4_div(x.x, x.y, x.z, x.w, scale.x, scale.y, scale.z, scale.w);
  const uint32_t lo = __byte_perm(__float_as_uint(t[0]), __float_as_uint(t[1]), 0x0040);
  const uint32_t hi = __byte_perm(__float_as_uint(t[2]), __float_as_uint(t[3]), 0x0040);
  return __byte_perm(lo, hi, 0x5410);
}
__device__ __forceinline__ uint8_t quant_e4m3(float x, float scale_inv) {
  float s = __fmul_rn(x, scale_inv);
  s = fminf(fmaxf(s, -448.0f), 448.0f);
  return (uint8_t)__nv_cvt_float_to_fp8(s, __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ uint32_t quant_e4m3x4(const float4 x, const float4 inv) {
  const float2 a = make_float2(fminf(fmaxf(__fmul_rn(x.x, inv.x), -448.0f), 448.0f), fminf(fmaxf(__fmul_rn(x.y, inv.y), -448.0f), 448.0f));
  const float2 b = make_float2(fminf(fmaxf(__fmul_rn(x.z, inv.z), -448.0f), 448.0f), fminf(fmaxf(__fmul_rn(x.w, inv.w), -448.0f), 448.0f));
  return (uint32_t)__nv_cvt_float2_to_fp8x2(a, __NV_SATFINITE, __NV_E4M3) |
         (uint32_t)__nv_cvt_float2_to_fp8x2(b, __NV_SATFINITE, __NV_E4M3) << 16;
}

// What a quantised tensor carries beside its tiles: zero points (all zero) and its own copy of the tile coordinates.
// Written by the quantiser's warps, so that the tensor costs one launch.
struct StoreExtras {
  int8_t* zero_points;
  const int32_t* rows_in;
  const int32_t* cols_in;
  int32_t* rows_out;
  int32_t* cols_out;
};
template <typename T>
__device__ __forceinline__ float4 load4(const T* p);
template <>
__device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <>
__device__ __forceinline__ float4 load4<__half>(const __half* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
template <>
__device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                     __uint_as_float(u.y & 0xffff0000u));
}
// One warp per tile: 1024 values, 32 per lane, read once and in their own type.
template <int KIND, typename T>
__global__ void __launch_bounds__(256) quant_tiles_kernel(const T* values, int64_t nnz, uint8_t* q, float* scale_out, float* scale_inv_out,
                                                          float* amax_out, StoreExtras x) {
  const int64_t tile = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  grid_dependency_wait();
  if (tile >= nnz) return;
  const T* src = values + tile * 1024;
  float4 v[8];
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = load4<T>(src + (i * 32 + lane) * 4);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w))));
  amax = warp_max(amax);
  const float scale = KIND == VOID_KIND_I8 ? fmaxf(__fdiv_rn(amax, 128.0f), 1e-8f) : fmaxf(__fdiv_rn(amax, 448.0f), 1e-12f);
  const float inv = __fdiv_rn(1.0f, scale);
  if (lane == 0) {
    scale_out[tile] = scale;
    if (scale_inv_out != nullptr) scale_inv_out[tile] = inv;
    if (amax_out != nullptr) amax_out[tile] = amax;
    if (x.zero_points != nullptr) x.zero_points[tile] = 0;
    if (x.rows_out != nullptr) x.rows_out[tile] = x.rows_in[tile];
    if (x.cols_out != nullptr) x.cols_out[tile] = x.cols_in[tile];
  }
  uint32_t* dst = reinterpret_cast<uint32_t*>(q) + tile * 256;
  const float4 sc = make_float4(scale, scale, scale, scale), si = make_float4(inv, inv, inv, inv);
#pragma unroll
  for (int i = 0; i < 8; ++i) dst[i * 32 + lane] = KIND == VOID_KIND_I8 ? quant_i8x4(v[i], sc, si) : quant_e4m3x4(v[i], si);
}

// column absmax of a row-major [K, N] matrix: block = 128 columns x a slab of k rows
constexpr int kColBlock = 128;
constexpr int kRowSlab = 64;
__global__ void col_amax_kernel(const float* __restrict__ b, int64_t ldb, int K, int N, float* __restrict__ amax) {
  const int n = blockIdx.x * kColBlock + threadIdx.x;
  if (n >= N) return;
  const int k0 = blockIdx.y * kRowSlab;
  const int k1 = (k0 + kRowSlab) < K ? (k0 + kRowSlab) : K;
  float m = 0.0f;
  for (int k = k0; k < k1; ++k) m = fmaxf(m, fabsf(b[(size_t)k * ldb + n]));
  // non-negative floats order like their bit patterns
  atomicMax(reinterpret_cast<int*>(amax) + n, __float_as_int(m));
}
__global__ void col_scale_kernel(float* __restrict__ scale, float* __restrict__ scale_inv, int N, int kind) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const float amax = scale[n];
  float s;
  if (kind == VOID_KIND_I8) s = fmaxf(__fdiv_rn(amax, 128.0f), 1e-8f);
  else s = fmaxf(__fdiv_rn(amax, 448.0f), 1e-12f);
  scale[n] = s;
  if (scale_inv != nullptr) scale_inv[n] = __fdiv_rn(1.0f, s);
}
__global__ void quant_cols_kernel(const float* __restrict__ b, int64_t ldb, int K, int N, int kind,
                                  uint8_t* __restrict__ q, int64_t ldq, const float* __restrict__ scale,
                                  int scale_stride) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y;
  if (n >= ldq) return;
  uint8_t o = 0;
  if (n < N) {
    const float x = b[(size_t)k * ldb + n];
    const float s = scale[(size_t)n * scale_stride];
    if (kind == VOID_KIND_I8) o = (uint8_t)quant_i8(x, s);
    else o = quant_e4m3(x, __fdiv_rn(1.0f, s));
  }
  q[(size_t)k * ldq + n] = o;
}
// four columns per thread (float4 in, 4 bytes out), kColRows rows with their loads in flight together and one reciprocal
// per column; VEC needs N, ldb multiples of 4 and aligned rows, else the floats are loaded one by one (16384 x 1001, both
// passes: INT8 66 us with a thread per element, 35 so).
// ldq is a multiple of 4.
constexpr int kColRows = 8;
template <bool VEC>
__global__ void __launch_bounds__(128) quant_cols4_kernel(const float* __restrict__ b, int64_t ldb, int K, int N, int kind,
                                                          uint8_t* __restrict__ q, int64_t ldq,
                                                          const float* __restrict__ scale, int scale_stride) {
  const int n = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (n >= ldq) return;
  const int k0 = blockIdx.y * kColRows;
  const bool in = n < N;
  float4 x[kColRows];
#pragma unroll
  for (int i = 0; i < kColRows; ++i) {
    x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!in || k0 + i >= K) continue;
    const float* src = b + (size_t)(k0 + i) * ldb + n;
    if (VEC) {
      x[i] = *reinterpret_cast<const float4*>(src);
    } else {
      x[i].x = src[0];
      if (n + 1 < N) x[i].y = src[1];
      if (n + 2 < N) x[i].z = src[2];
      if (n + 3 < N) x[i].w = src[3];
    }
  }
  float4 s = make_float4(1.f, 1.f, 1.f, 1.f);
  if (in) {
    if (!scale_stride) {
      s.x = s.y = s.z = s.w = scale[0];
    } else if (VEC) {
      s = *reinterpret_cast<const float4*>(scale + n);
    } else {
      s.x = scale[n];
      if (n + 1 < N) s.y = scale[n + 1];
      if (n + 2 < N) s.z = scale[n + 2];
      if (n + 3 < N) s.w = scale[n + 3];
    }
  }
  const float4 inv = make_float4(__fdiv_rn(1.0f, s.x), __fdiv_rn(1.0f, s.y), __fdiv_rn(1.0f, s.z), __fdiv_rn(1.0f, s.w));
#pragma unroll
  for (int i = 0; i < kColRows; ++i)
    if (k0 + i < K)
      *reinterpret_cast<uint32_t*>(q + (size_t)(k0 + i) * ldq + n) =
          kind == VOID_KIND_I8 ? quant_i8x4(x[i], s, inv) : quant_e4m3x4(x[i], inv);
}
// Column scales and quantised columns in one launch: a cluster of eight CTAs owns 16 columns, every CTA an eighth of the
// rows, which it keeps in shared memory between the maximum and the quantisation, so B crosses from memory once.  Every
// thread comes back to the words it copied itself (no barrier around the copies); the CTAs exchange their column maxima
// through distributed shared memory.  VEC: four columns per thread.  Bound by the latency of that chain (copy, maximum,
// two cluster barriers, quantise).  Measured against the four launches of the form below (INT8, graph of launches):
// 512 x 128 2.8 us against 10.2, 4096 x 512 6.7 against 12.3, 8192 x 512 7.9 against 14.1.  32 columns per cluster:
// 4096 x 64 4.8 against 3.9, 8192 x 512 13.2 against 7.9 (one CTA per SM).
constexpr int kFusedThreads = 256, kFusedCtas = 8, kFusedCols = 16;
constexpr int kFusedSmem = 64 * 1024, kFusedMaxSmem = 208 * 1024;   // several CTAs per SM, one CTA per SM
template <int KIND, bool VEC>
__global__ void __launch_bounds__(kFusedThreads) quant_cols_fused_kernel(const float* b, int64_t ldb, int K, int N, uint8_t* q, int64_t ldq,
                                                                         float* scale_out, float* scale_inv_out, int early) {
  namespace cg = cooperative_groups;
  constexpr int W = kFusedCols;
  constexpr int E = VEC ? 4 : 1;                        // columns a thread owns
  constexpr int TPR = W / E;                            // threads per row
  constexpr int ROWS = kFusedThreads / TPR;             // rows per pass
  constexpr int WARPS = kFusedThreads / 32;
  extern __shared__ __align__(16) float slab[];         // [rows of this CTA][W]
  __shared__ float part[WARPS][W];
  __shared__ float cta_max[W];
  __shared__ __align__(16) float s_scale[W], s_inv[W];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int n0 = (int)(blockIdx.x / kFusedCtas) * W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int col = (tid % TPR) * E, r0 = tid / TPR;
  const int n = n0 + col;
  const int per = (K + kFusedCtas - 1) / kFusedCtas;
  const int k0 = rank * per;
  const int rows = (K - k0) < per ? ((K - k0) > 0 ? K - k0 : 0) : per;
  const uint32_t bytes = n < N ? 4u * E : 0u;           // (N is a multiple of 4 in the vector form); 0: zero fill
  grid_dependency_wait();

  const float* src = b + (size_t)k0 * ldb + (n < N ? n : 0);
  for (int r = r0; r < rows; r += ROWS) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(slab + r * W + col);
    if constexpr (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src + (size_t)r * ldb), "r"(bytes) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src + (size_t)r * ldb), "r"(bytes) : "memory");
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (early) grid_launch_dependents();
  float m[E];
#pragma unroll
  for (int e = 0; e < E; ++e) m[e] = 0.0f;
#pragma unroll 4
  for (int r = r0; r < rows; r += ROWS) {
    if constexpr (VEC) {
      const float4 x = *reinterpret_cast<const float4*>(slab + r * W + col);
      m[0] = fmaxf(m[0], fabsf(x.x)); m[1] = fmaxf(m[1], fabsf(x.y));
      m[2] = fmaxf(m[2], fabsf(x.z)); m[3] = fmaxf(m[3], fabsf(x.w));
    } else {
      m[0] = fmaxf(m[0], fabsf(slab[r * W + col]));
    }
  }
  // lanes of a warp that share columns, then the warps, then the CTAs of the cluster
#pragma unroll
  for (int o = TPR; o < 32; o <<= 1)
#pragma unroll
    for (int e = 0; e < E; ++e) m[e] = fmaxf(m[e], __shfl_xor_sync(0xffffffffu, m[e], o));
  if (lane < TPR)
#pragma unroll
    for (int e = 0; e < E; ++e) part[warp][col + e] = m[e];
  __syncthreads();
  if (tid < W) {
    float x = 0.0f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) x = fmaxf(x, part[w][tid]);
    cta_max[tid] = x;
  }
  cluster.sync();
  if (tid < W) {
    float x = 0.0f;
#pragma unroll
    for (int c = 0; c < kFusedCtas; ++c) x = fmaxf(x, *cluster.map_shared_rank(cta_max + tid, c));
    const float s = (KIND == VOID_KIND_I8) ? fmaxf(__fdiv_rn(x, 128.0f), 1e-8f) : fmaxf(__fdiv_rn(x, 448.0f), 1e-12f);
    const float inv = __fdiv_rn(1.0f, s);
    s_scale[tid] = s;
    s_inv[tid] = inv;
    if (rank == 0 && n0 + tid < N) {
      scale_out[n0 + tid] = s;
      if (scale_inv_out != nullptr) scale_inv_out[n0 + tid] = inv;
    }
  }
  // No CTA leaves while another still reads its maxima, so the second meeting of the cluster is waited for at the end.
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  __syncthreads();   // the scales for this CTA
  if (!early) grid_launch_dependents();
  const int mine = n < ldq ? rows : 0;
  uint8_t* dst = q + (size_t)k0 * ldq + n;
  if constexpr (VEC) {
    const float4 sc = *reinterpret_cast<const float4*>(s_scale + col), si = *reinterpret_cast<const float4*>(s_inv + col);
#pragma unroll 4
    for (int r = r0; r < mine; r += ROWS) {
      const float4 x = *reinterpret_cast<const float4*>(slab + r * W + col);
      *reinterpret_cast<uint32_t*>(dst + (size_t)r * ldq) = KIND == VOID_KIND_I8 ? quant_i8x4(x, sc, si) : quant_e4m3x4(x, si);
    }
  } else {
    const float sc = s_scale[col], si = s_inv[col];
    const float4 sc4 = make_float4(sc, sc, sc, sc), si4 = make_float4(si, si, si, si);
    int r = r0;
    for (; r + 3 * ROWS < mine; r += 4 * ROWS) {   // (four rows at once: the form that divides only where rounding hangs on it)
      const float4 x = make_float4(slab[r * W + col], slab[(r + ROWS) * W + col], slab[(r + 2 * ROWS) * W + col], slab[(r + 3 * ROWS) * W + col]);
      const uint32_t o = KIND == VOID_KIND_I8 ? quant_i8x4(x, sc4, si4) : quant_e4m3x4(x, si4);
#pragma unroll
      for (int k = 0; k < 4; ++k) dst[(size_t)(r + k * ROWS) * ldq] = (uint8_t)(o >> (8 * k));
    }
    for (; r < mine; r += ROWS) {
      const float x = slab[r * W + col];
      dst[(size_t)r * ldq] = KIND == VOID_KIND_I8 ? (uint8_t)quant_i8(x, sc) : quant_e4m3(x, si);
    }
  }
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// absmax of a whole row-major [K, N] matrix into amax[0] (zero before the launch)
__global__ void tensor_amax_kernel(const float* __restrict__ b, int64_t ldb, int K, int N, float* __restrict__ amax) {
  const int n = blockIdx.x * kColBlock + threadIdx.x;
  const int k0 = blockIdx.y * kRowSlab;
  const int k1 = (k0 + kRowSlab) < K ? (k0 + kRowSlab) : K;
  float m = 0.0f;
  if (n < N)
    for (int k = k0; k < k1; ++k) m = fmaxf(m, fabsf(b[(size_t)k * ldb + n]));
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(amax), __float_as_int(m));
}

// Column sums of a row-major [rows, cols] matrix (the bias gradient), fp32 accumulation in a fixed order: a cluster owns 32
// columns, its CTAs share the rows and add their partial sums in rank order through distributed shared memory.  Bound by
// reading the matrix once: 512 x 4096 fp32 (8 MB) in 3.7 us against 10.4 us for the two-pass library reduction.
constexpr int kSumCols = 32, kSumThreads = 256;
template <typename T> __device__ __forceinline__ float as_float(T v);
template <> __device__ __forceinline__ float as_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float as_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float as_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T, bool VEC>
__global__ void __launch_bounds__(kSumThreads) column_sum_kernel(const T* in, int64_t ld, int rows, int cols, T* out) {
  namespace cg = cooperative_groups;
  constexpr int E = VEC ? 4 : 1, TPR = kSumCols / E, ROWS = kSumThreads / TPR, WARPS = kSumThreads / 32;
  __shared__ float part[WARPS][kSumCols];
  __shared__ float cta_sum[kSumCols];
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int col = (tid % TPR) * E, c0 = (int)(blockIdx.x / ctas) * kSumCols + col;
  const int per = (rows + ctas - 1) / ctas, r_end = (rank + 1) * per < rows ? (rank + 1) * per : rows;
  grid_dependency_wait();
  grid_launch_dependents();
  float s[E];
#pragma unroll
  for (int e = 0; e < E; ++e) s[e] = 0.0f;
  if (c0 < cols) {
#pragma unroll 8
    for (int r = rank * per + tid / TPR; r < r_end; r += ROWS) {
      const T* src = in + (size_t)r * ld + c0;
      if constexpr (VEC) {
        T v[4];
        if constexpr (sizeof(T) == 4) *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(src);
        else *reinterpret_cast<uint2*>(v) = *reinterpret_cast<const uint2*>(src);
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] += as_float<T>(v[e]);
      } else {
        s[0] += as_float<T>(*src);
      }
    }
  }
#pragma unroll
  for (int o = TPR; o < 32; o <<= 1)
#pragma unroll
    for (int e = 0; e < E; ++e) s[e] += __shfl_xor_sync(0xffffffffu, s[e], o);
  if (lane < TPR)
#pragma unroll
    for (int e = 0; e < E; ++e) part[warp][col + e] = s[e];
  __syncthreads();
  if (warp == 0) {
    float x = 0.0f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) x += part[w][lane];
    cta_sum[lane] = x;
  }
  cluster.sync();
  if (rank == 0 && warp == 0) {
    float x = 0.0f;
    for (int c = 0; c < ctas; ++c) x += *cluster.map_shared_rank(cta_sum + lane, c);
    const int c = (int)(blockIdx.x / ctas) * kSumCols + lane;
    if (c < cols) out[c] = T(x);
  }
  cluster.sync();   // no CTA leaves while rank 0 still reads its sums
}
template <typename T>
static bool launch_column_sum(const void* in, int64_t ld, int rows, int cols, void* out, cudaStream_t st) {
  // enough CTAs along the rows that a thread adds few of them, never more than one per 32 rows
  int ctas = 1;
  while (ctas < 8 && ctas * 32 < rows) ctas *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((cols + kSumCols - 1) / kSumCols) * (unsigned)ctas);
  cfg.blockDim = dim3(kSumThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const bool vec = cols % 4 == 0 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(in) & (4 * sizeof(T) - 1)) == 0;
  const T* src = reinterpret_cast<const T*>(in);
  T* dst = reinterpret_cast<T*>(out);
  return (vec ? cudaLaunchKernelEx(&cfg, column_sum_kernel<T, true>, src, ld, rows, cols, dst)
              : cudaLaunchKernelEx(&cfg, column_sum_kernel<T, false>, src, ld, rows, cols, dst)) == cudaSuccess;
}

// Rows copied to a pitch of whole 16-byte pieces (what the copy engine reads); one thread per piece of the result.  The
// padding is written as zeros.
// The product that follows may start only when every block is about to write its result.  Started with the first loads, a
// persistent product settles on the SMs unevenly beside the blocks still running and stays so: INT8 columns quantised and
// multiplied, 16384 x 4096, N = 2048: 75.7 us, started late 59.7 (15.3 + 42.6 alone).  Where all blocks run at once there is nothing
// to settle beside, and it may start with them: bf16 GELU 3001 x 5003, N = 333 (821 blocks) 11.7 -> 10.5 us, 4096 x 1111, N = 777
// 12.9 -> 11.5; started early behind 4032 blocks 47.1 -> 47.4 (fp16 8192^2, 90 %, N = 1001).
template <typename T>
__global__ void __launch_bounds__(256) copy_rows_kernel(const T* in, int64_t ld_in, uint4* out, int64_t pieces, int64_t rows, int cols, int early) {
  constexpr int E = 16 / (int)sizeof(T);
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  grid_dependency_wait();
  if (early) grid_launch_dependents();
  if (i >= rows * pieces) return;
  const int64_t r = i / pieces;
  const int c0 = (int)(i - r * pieces) * E;
  const T* src = in + r * ld_in + c0;
  union { uint4 v; T e[E]; } o;
#pragma unroll
  for (int k = 0; k < E; ++k) o.e[k] = c0 + k < cols ? src[k] : T(0);
  if (!early) grid_launch_dependents();
  out[i] = o.v;
}

// Transposed copy in tiles of 128 bytes by 128 / E elements.  Whole 16-byte pieces in and out: a warp reads four 128-byte
// rows, and eight of its lanes write one 128-byte row of the result, each collecting its piece from a column of shared
// memory (rows of 33 words).  Bound by memory: 2048 x 4096 bf16 (17 MB each way) 7.9 us.
template <typename T>
__global__ void __launch_bounds__(256) transpose_kernel(const T* in, int64_t ld_in, T* out, int64_t ld_out, int rows, int cols, int whole) {
  constexpr int S = 128 / (int)sizeof(T), V = 16 / (int)sizeof(T), C = 4 / (int)sizeof(T);
  __shared__ uint32_t tile[S][33];
  const int r0 = blockIdx.y * S, c0 = blockIdx.x * S;
  grid_dependency_wait();
#pragma unroll
  for (int i = threadIdx.x; i < S * 8; i += 256) {
    const int r = i >> 3, c = i & 7;
    union { uint4 v; uint32_t w[4]; T e[V]; } x;
    x.v = make_uint4(0u, 0u, 0u, 0u);
    if (r0 + r < rows) {
      const T* src = in + (int64_t)(r0 + r) * ld_in + c0 + c * V;
      if (whole && c0 + (c + 1) * V <= cols) {
        x.v = *reinterpret_cast<const uint4*>(src);
      } else {
#pragma unroll
        for (int k = 0; k < V; ++k)
          if (c0 + c * V + k < cols) x.e[k] = src[k];
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) tile[r][c * 4 + k] = x.w[k];
  }
  __syncthreads();
  const int word = threadIdx.x >> 3, first = (threadIdx.x & 7) * V;   // C columns of the tile, V rows of it
  if (r0 + first >= ld_out) return;
  grid_launch_dependents();
  uint32_t w[V], o[C][4];
#pragma unroll
  for (int k = 0; k < V; ++k) w[k] = tile[first + k][word];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (C == 1) {
      o[0][j] = w[j];
    } else if (C == 2) {
      o[0][j] = __byte_perm(w[2 * j], w[2 * j + 1], 0x5410);
      o[C - 1][j] = __byte_perm(w[2 * j], w[2 * j + 1], 0x7632);
    } else {
      const uint32_t a = w[(4 * j) % V], b = w[(4 * j + 1) % V], c = w[(4 * j + 2) % V], d = w[(4 * j + 3) % V];
      const uint32_t ab = __byte_perm(a, b, 0x5140), cd = __byte_perm(c, d, 0x5140);
      const uint32_t AB = __byte_perm(a, b, 0x7362), CD = __byte_perm(c, d, 0x7362);
      o[0][j] = __byte_perm(ab, cd, 0x5410);
      o[1 % C][j] = __byte_perm(ab, cd, 0x7632);
      o[2 % C][j] = __byte_perm(AB, CD, 0x5410);
      o[3 % C][j] = __byte_perm(AB, CD, 0x7632);
    }
  }
#pragma unroll
  for (int q = 0; q < C; ++q) {
    const int c = c0 + word * C + q;
    if (c < cols) *reinterpret_cast<uint4*>(out + (int64_t)c * ld_out + r0 + first) = make_uint4(o[q][0], o[q][1], o[q][2], o[q][3]);
  }
}

// ------------------------------------------------------------------------------ Stream-K table
__global__ void __launch_bounds__(1024) streamk_offsets_kernel(const int32_t* __restrict__ row_ptr, int nbr,
                                                               int target, int32_t* __restrict__ woff,
                                                               int32_t* __restrict__ n_workers_out) {
  // woff[r] = number of chunks of row r, then scanned in place
  for (int r = threadIdx.x; r < nbr; r += blockDim.x) {
    const int cnt = row_ptr[r + 1] - row_ptr[r];
    woff[r] = (cnt + target - 1) / target;
  }
  __syncthreads();
  block_exclusive_scan(woff, woff, nbr);
  if (threadIdx.x == 0) *n_workers_out = woff[nbr];
}
__global__ void streamk_fill_kernel(const int32_t* __restrict__ row_ptr, int nbr, int target,
                                    const int32_t* __restrict__ woff, int32_t* __restrict__ w_rows,
                                    int32_t* __restrict__ w_start, int32_t* __restrict__ w_end,
                                    uint8_t* __restrict__ w_atomic) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nbr) return;
  const int rs = row_ptr[r], re = row_ptr[r + 1];
  const int chunks = woff[r + 1] - woff[r];
  int w = woff[r];
  for (int pos = rs; pos < re; pos += target, ++w) {
    const int e = (pos + target) < re ? (pos + target) : re;
    w_rows[w] = r;
    w_start[w] = pos;
    w_end[w] = e;
    w_atomic[w] = chunks > 1 ? 1 : 0;
  }
}

// Clusters of the column quantiser that run at once when its shared memory lets one and two CTAs share an SM.  A cluster
// stays inside one group of SMs, and the groups differ from device to device, so the driver is asked, once per device.
struct ClusterRoom { int one_per_sm = 0, two_per_sm = 0; };
template <int KIND, bool VEC>
static ClusterRoom cluster_room() {
  static std::atomic<uint32_t> rooms[64];   // 1 + (two_per_sm << 16 | one_per_sm); 0: not asked yet
  int dev = 0;
  ClusterRoom r;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return r;
  uint32_t packed = rooms[dev].load(std::memory_order_relaxed);
  if (packed == 0) {
    auto kernel = quant_cols_fused_kernel<KIND, VEC>;
    if (ensure_smem((const void*)kernel, kFusedMaxSmem)) return r;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kFusedCtas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kFusedCtas);
    cfg.blockDim = dim3(kFusedThreads);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int room[2] = {0, 0};
    for (int ctas = 1; ctas <= 2; ++ctas) {
      cfg.dynamicSmemBytes = (size_t)(kFusedMaxSmem / ctas);
      if (cudaOccupancyMaxActiveClusters(&room[ctas - 1], kernel, &cfg) != cudaSuccess) return r;
    }
    packed = 1u + ((uint32_t)room[1] << 16 | (uint32_t)room[0]);
    rooms[dev].store(packed, std::memory_order_relaxed);   // (threads that ask at once store the same)
  }
  r.one_per_sm = (int)((packed - 1u) & 0xffffu);
  r.two_per_sm = (int)((packed - 1u) >> 16);
  return r;
}
template <int KIND, bool VEC>
static bool launch_quant_cols_fused(const float* b, int64_t ldb, int K, int N, void* q, int64_t ldq, float* scale,
                                    float* scale_inv, cudaStream_t st) {
  auto kernel = quant_cols_fused_kernel<KIND, VEC>;
  const unsigned clusters = (unsigned)((ldq + kFusedCols - 1) / kFusedCols), ctas = clusters * kFusedCtas;
  int smem = (K + kFusedCtas - 1) / kFusedCtas * kFusedCols * 4;
  if (smem > 48 * 1024 && ensure_smem((const void*)kernel, kFusedMaxSmem)) return false;
  // The launch may start beside the end of the kernel before it, whose SMs come free one after the other: a grid that needs
  // two CTAs per SM would fill the first ones with as many as fit and leave others idle.  It asks for the shared memory that
  // keeps it to two, while all its clusters then still run at once: from more than fit one CTA per SM (15 here, 240 columns) to
  // fewer than fit two (33).  Columns quantised and multiplied in turn, without and with it, us: INT8 4096^2, 90 %, N = 256
  // 10.9 / 10.3, 384 12.8 / 11.4, 496 15.7 / 13.9, 512 14.4 / 12.6; FP8 2048 x 4096 256 13.0 / 10.6, 384 11.7 / 11.4, 512 13.7 / 12.4; FP8
  // 4096^2 384 13.7 / 12.4, but 512 15.3 / 16.3.  Where the last cluster has just room, N = 528: INT8 16.0 / 15.0, FP8 2048 x 4096
  // 13.0 / 15.7; where it waits for the first to end, N = 560: 16.8 / 19.3 and 13.2 / 16.3.  From 48 KB a CTA on there is nothing to
  // gain (8192^2: 38.8 / 39.4).
  // The kernel behind it may start with the first maxima where all clusters run at once, two CTAs per SM at most: its own CTAs
  // then only wait for the places.  With more, they would take the places of clusters still to come and settle unevenly (INT8
  // 16384 x 4096, N = 2048 55 us late, 62 early).  us with their products, late and early: FP8 4096^2, 80 %, N = 512 16.9 16.0,
  // 4096 x 2048, N = 128 10.7 8.96, INT8 4096^2, 90 %, N = 512 10.7 10.5, 512^2, N = 128 6.59 6.49; slabs of 64 KB (8192^2, N = 512) 21.8
  // 21.9, as they were.
  int early = 0;
  if (smem <= 48 * 1024) {
    const ClusterRoom room = cluster_room<KIND, VEC>();
    early = (int)clusters <= room.two_per_sm ? 1 : 0;
    if ((int)clusters > room.one_per_sm && (int)clusters < room.two_per_sm) smem = kFusedMaxSmem / 2;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kFusedThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kFusedCtas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, b, ldb, K, N, reinterpret_cast<uint8_t*>(q), ldq, scale, scale_inv, early) == cudaSuccess;
}
// The one-launch form; false: not taken.  It is the faster one while three of its CTAs fit an SM (64 KB of rows each, K up
// to 8192), and beyond that only where one CTA per SM holds everything at once (16384 x 256: 13.8 us against 15.7, but
// 16384 x 2048: 77 against 54, since the phases of a lone CTA do not overlap).
static bool quant_cols_fused(const float* b, int64_t ldb, int K, int N, int kind, void* q, int64_t ldq, float* scale,
                             float* scale_inv, cudaStream_t st) {
  const int64_t smem = (int64_t)((K + kFusedCtas - 1) / kFusedCtas) * kFusedCols * 4;
  const int64_t ctas = (ldq + kFusedCols - 1) / kFusedCols * kFusedCtas;
  if (smem > kFusedMaxSmem || (smem > kFusedSmem && ctas > 144)) return false;
  const bool vec = (N % 4 == 0) && (ldb % 4 == 0) && (ldq % 4 == 0) && ((reinterpret_cast<uintptr_t>(b) & 15u) == 0) &&
                   ((reinterpret_cast<uintptr_t>(q) & 3u) == 0);
  if (kind == VOID_KIND_I8)
    return vec ? launch_quant_cols_fused<VOID_KIND_I8, true>(b, ldb, K, N, q, ldq, scale, scale_inv, st)
               : launch_quant_cols_fused<VOID_KIND_I8, false>(b, ldb, K, N, q, ldq, scale, scale_inv, st);
  return vec ? launch_quant_cols_fused<VOID_KIND_F8E4M3, true>(b, ldb, K, N, q, ldq, scale, scale_inv, st)
             : launch_quant_cols_fused<VOID_KIND_F8E4M3, false>(b, ldb, K, N, q, ldq, scale, scale_inv, st);
}

}  // namespace vb

using namespace vb;

extern "C" {

const char* void_strerror(int status) {
  switch (status) {
    case VOID_OK: return "ok";
    case VOID_ERR_BAD_ARG: return "bad argument (null pointer, negative size or unknown enum value)";
    case VOID_ERR_ALIGN: return "pointer or leading dimension breaks an alignment rule";
    case VOID_ERR_SHAPE: return "unsupported shape";
    case VOID_ERR_ARCH: return "current device is not an sm_100 (B200) GPU";
    case VOID_ERR_CUDA: return "a CUDA runtime or driver call failed";
    case VOID_ERR_WORKSPACE: return "workspace too small";
    case VOID_ERR_DEVICE_TIMEOUT: return "a bounded device-side wait gave up";
    case VOID_ERR_TOO_LARGE: return "size beyond a documented maximum";
    case VOID_ERR_TENSOR_MAP: return "the driver refused the copy-engine (TMA) descriptor of B";
    default: return "unknown status";
  }
}

int void_b200_abi_version(void) { return VOID_B200_ABI_VERSION; }

size_t void_tile_index_ws_bytes(int32_t nbr, int32_t nbc) {
  if (nbr <= 0 || nbc <= 0) return 16;
  const size_t wpr = ((size_t)nbc + 31) / 32;
  return (size_t)nbr * wpr * 4 + (size_t)nbr * 4 + 16;
}

// row_order: null, or written as void_row_order writes it where that costs no launch (*ordered is set then)
static int build_tile_index(const int32_t* block_rows, const int32_t* block_cols, int64_t nnz, int32_t nbr, int32_t nbc,
                            int32_t* row_ptr, int32_t* block_indices, int32_t* row_order, bool* ordered, void* ws, size_t ws_bytes,
                            void_stream_t stream) {
  if (nnz < 0 || nbr < 0 || nbc < 0 || row_ptr == nullptr) return VOID_ERR_BAD_ARG;
  cudaStream_t st = as_stream(stream);
  if (nbr == 0) return cudaMemsetAsync(row_ptr, 0, 4, st) == cudaSuccess ? VOID_OK : VOID_ERR_CUDA;
  if (nnz > 0 && (block_rows == nullptr || block_cols == nullptr || block_indices == nullptr)) return VOID_ERR_BAD_ARG;
  if (nnz > 0x7fffffffLL) return VOID_ERR_TOO_LARGE;
  if (ws == nullptr || ws_bytes < void_tile_index_ws_bytes(nbr, nbc)) return VOID_ERR_WORKSPACE;
  const int wpr = (nbc + 31) / 32;
  const int pitch = one_block_pitch(wpr);
  if (one_block_index(nnz, (int64_t)nbr * pitch)) {
    const int smem = one_block_smem(nbr * pitch);
    if (smem > 48 * 1024 && ensure_smem((const void*)tile_index_kernel, one_block_smem(kOneBlockWords))) return VOID_ERR_CUDA;
    *ordered = row_order != nullptr && nbr <= kOneBlockOrder;
    return status_of(launch_pdl(tile_index_kernel, 1, 1024, smem, st, block_rows, block_cols, (int)nnz, nbr, nbc, pitch, row_ptr, block_indices,
                                *ordered ? row_order : nullptr));
  }
  uint32_t* bitmap = reinterpret_cast<uint32_t*>(ws);
  int32_t* counts = reinterpret_cast<int32_t*>(bitmap + (size_t)nbr * wpr);
  if (cudaMemsetAsync(bitmap, 0, (size_t)nbr * wpr * 4, st) != cudaSuccess) return VOID_ERR_CUDA;
  const unsigned blocks = (unsigned)((nnz + 255) / 256);
  Launches on(st);
  if (nnz > 0) on.run(mark_tiles_kernel, blocks, 256, block_rows, block_cols, nnz, nbr, nbc, wpr, bitmap, block_indices);
  if ((int64_t)nbr * wpr <= kOneBlockBitmap) {
    on.run(count_scan_rows_kernel, 1, 1024, bitmap, nbr, wpr, counts, row_ptr);
  } else {
    on.run(count_rows_kernel, (unsigned)(((int64_t)nbr * 32 + 255) / 256), 256, bitmap, nbr, wpr, counts);
    on.run(scan_rows_kernel, 1, 1024, counts, row_ptr, nbr);
  }
  if (nnz > 0) on.run(rank_tiles_kernel, blocks, 256, block_rows, block_cols, nnz, nbr, nbc, wpr, bitmap, row_ptr, block_indices);
  return on.status();
}

int void_build_tile_index(const int32_t* block_rows, const int32_t* block_cols, int64_t nnz, int32_t nbr,
                          int32_t nbc, int32_t* row_ptr, int32_t* block_indices, void* ws, size_t ws_bytes,
                          void_stream_t stream) {
  bool ordered = false;
  return build_tile_index(block_rows, block_cols, nnz, nbr, nbc, row_ptr, block_indices, nullptr, &ordered, ws, ws_bytes, stream);
}

int void_build_tile_index_order(const int32_t* block_rows, const int32_t* block_cols, int64_t nnz, int32_t nbr, int32_t nbc,
                                int32_t* row_ptr, int32_t* block_indices, int32_t* row_order, void* ws, size_t ws_bytes,
                                void_stream_t stream) {
  if (nbr > 0 && row_order == nullptr) return VOID_ERR_BAD_ARG;
  bool ordered = false;
  const int st = build_tile_index(block_rows, block_cols, nnz, nbr, nbc, row_ptr, block_indices, row_order, &ordered, ws, ws_bytes, stream);
  return st != VOID_OK || ordered ? st : void_row_order(row_ptr, nbr, row_order, stream);
}

int void_row_order(const int32_t* row_ptr, int32_t nbr, int32_t* order, void_stream_t stream) {
  if (nbr < 0) return VOID_ERR_BAD_ARG;
  if (nbr == 0) return VOID_OK;
  if (row_ptr == nullptr || order == nullptr) return VOID_ERR_BAD_ARG;
  return status_of(launch_pdl(row_order_kernel, (int)(((int64_t)nbr * 32 + 255) / 256), 256, 0, as_stream(stream), row_ptr, nbr, order));
}

int void_pack_tiles(const void* values, const float* scales, int64_t n_scales, const int32_t* block_cols,
                    const int32_t* block_indices, const int32_t* row_ptr, int64_t nnz, int32_t nbr, void* packed,
                    int32_t* tile_cols, float* tile_scales, float* row_scale, void_stream_t stream) {
  if (nnz < 0 || nbr < 0) return VOID_ERR_BAD_ARG;
  cudaStream_t st = as_stream(stream);
  if (nnz > 0) {
    if (values == nullptr || block_cols == nullptr || block_indices == nullptr || packed == nullptr ||
        tile_cols == nullptr)
      return VOID_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(values) & 15u) != 0 || (reinterpret_cast<uintptr_t>(packed) & 1023u) != 0)
      return VOID_ERR_ALIGN;
    if (scales != nullptr && n_scales != 1 && n_scales != nnz) return VOID_ERR_BAD_ARG;
  }
  RowScales rows = {row_ptr, row_scale, 0, (unsigned)((nnz * 64 + 255) / 256)};
  if (row_scale != nullptr && nbr > 0) {
    if (row_ptr == nullptr || (nnz > 0 && tile_scales == nullptr)) return VOID_ERR_BAD_ARG;
    rows.nbr = nbr;
  }
  const unsigned blocks = rows.pack_blocks + (unsigned)((rows.nbr + 7) / 8);
  if (blocks == 0) return VOID_OK;
  return status_of(launch_pdl(pack_tiles_kernel, (int)blocks, 256, 0, st, reinterpret_cast<const uint4*>(values), block_indices, nnz,
                              reinterpret_cast<uint4*>(packed), TileMeta{block_cols, scales, n_scales, tile_cols, tile_scales}, rows));
}

int void_pack_tiles_f8_split(const void* values, const float* scales, int64_t n_scales, const int32_t* block_rows,
                             const int32_t* block_cols, const int32_t* block_indices, const int32_t* row_ptr, int64_t nnz,
                             int32_t nbr, int32_t terms, void* packed, int32_t* tile_cols, float* tile_scales,
                             float* row_scale, void_stream_t stream) {
  if (nnz < 0 || nbr < 0 || (terms != 2 && terms != 3)) return VOID_ERR_BAD_ARG;
  if (row_ptr == nullptr || row_scale == nullptr) return VOID_ERR_BAD_ARG;
  cudaStream_t st = as_stream(stream);
  if (nnz > 0) {
    if (values == nullptr || block_rows == nullptr || block_cols == nullptr || block_indices == nullptr ||
        packed == nullptr || tile_cols == nullptr || tile_scales == nullptr)
      return VOID_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(values) & 15u) != 0 || (reinterpret_cast<uintptr_t>(packed) & 1023u) != 0)
      return VOID_ERR_ALIGN;
    if (scales != nullptr && n_scales != 1 && n_scales != nnz) return VOID_ERR_BAD_ARG;
  }
  Launches on(st);
  if (nnz > 0)
    on.run(gather_tile_meta_kernel, (unsigned)((nnz + 255) / 256), 256, block_cols, scales, n_scales, block_indices, nnz, tile_cols, tile_scales);
  if (nbr > 0) on.run(row_max_scale_kernel, (unsigned)((nbr + 255) / 256), 256, row_ptr, tile_scales, nbr, row_scale);
  if (nnz > 0)
    on.run(terms == 2 ? pack_tiles_f8_split_kernel<2> : pack_tiles_f8_split_kernel<3>, (unsigned)((nnz * 64 + 255) / 256), 256,
           reinterpret_cast<const uint4*>(values), scales, n_scales, block_rows, block_indices, row_scale, nnz, nbr, reinterpret_cast<uint4*>(packed));
  return on.status();
}

int void_reduce_slots(const void* slots, const uint8_t* contrib, int32_t n_ranks, int32_t rows_owned, int32_t row0,
                      int32_t n_panels, int32_t panels_per_item, const float* row_scale, const float* col_scale, float b_scale, const float* bias,
                      int32_t act, void* out, int64_t ldc, int32_t out_dtype, int32_t M, int32_t N, void_stream_t stream) {
  if (n_ranks < 1 || n_ranks > 8 || rows_owned < 0 || n_panels < 1 || N < 1 || M < 0) return VOID_ERR_BAD_ARG;
  if (panels_per_item != 1 && panels_per_item != 2 && panels_per_item != 4) return VOID_ERR_BAD_ARG;
  if (out_dtype < VOID_OUT_F32 || out_dtype > VOID_OUT_BF16 || act < VOID_ACT_NONE || act > VOID_ACT_SILU) return VOID_ERR_BAD_ARG;
  if (rows_owned == 0) return VOID_OK;
  if (slots == nullptr || contrib == nullptr || row_scale == nullptr || out == nullptr || ldc < N) return VOID_ERR_BAD_ARG;
  if ((long long)n_panels * 128 < N) return VOID_ERR_SHAPE;
  Launches on(as_stream(stream));
  on.run(reduce_slots_kernel, (unsigned)(rows_owned * n_panels), 128, reinterpret_cast<const int32_t*>(slots), contrib, n_ranks, rows_owned, row0,
         n_panels, panels_per_item, row_scale, col_scale, b_scale, bias, act, out, ldc, out_dtype, M, N);
  return on.status();
}

int void_pack_tiles_fp(const void* values, int32_t elem_bytes, const int32_t* block_cols, const int32_t* block_indices,
                       int64_t nnz, void* packed, int32_t* tile_cols, void_stream_t stream) {
  if (nnz < 0 || (elem_bytes != 2 && elem_bytes != 4)) return VOID_ERR_BAD_ARG;
  if (nnz == 0) return VOID_OK;
  if (values == nullptr || block_cols == nullptr || block_indices == nullptr || packed == nullptr || tile_cols == nullptr)
    return VOID_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(values) & 15u) != 0 || (reinterpret_cast<uintptr_t>(packed) & 1023u) != 0)
    return VOID_ERR_ALIGN;
  Launches on(as_stream(stream));
  on.run(elem_bytes == 2 ? pack_tiles_fp_kernel<2> : pack_tiles_fp_kernel<4>, (unsigned)((nnz * 64 * elem_bytes + 255) / 256), 256,
         reinterpret_cast<const uint4*>(values), block_indices, nnz, reinterpret_cast<uint4*>(packed),
         TileMeta{block_cols, nullptr, 0, tile_cols, nullptr});
  return on.status();
}

int void_repack_tiles_fp(const void* values, int32_t elem_bytes, const int32_t* block_indices, int64_t nnz,
                         int32_t transposed, void* packed, void_stream_t stream) {
  if (nnz < 0 || (elem_bytes != 2 && elem_bytes != 4)) return VOID_ERR_BAD_ARG;
  if (nnz == 0) return VOID_OK;
  if (values == nullptr || block_indices == nullptr || packed == nullptr) return VOID_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(values) & 15u) != 0 || (reinterpret_cast<uintptr_t>(packed) & 1023u) != 0)
    return VOID_ERR_ALIGN;
  const unsigned blocks = (unsigned)((nnz * 64 * elem_bytes + 255) / 256);   // one thread per 16 bytes in both forms
  uint4* o = reinterpret_cast<uint4*>(packed);
  Launches on(as_stream(stream));
  if (transposed) on.run(elem_bytes == 2 ? pack_tiles_fp_t_kernel<2> : pack_tiles_fp_t_kernel<4>, blocks, 256, values, block_indices, nnz, o);
  else
    on.run(elem_bytes == 2 ? pack_tiles_fp_kernel<2> : pack_tiles_fp_kernel<4>, blocks, 256, reinterpret_cast<const uint4*>(values), block_indices,
           nnz, o, TileMeta{});
  return on.status();
}

int void_copy_rows(const void* in, int64_t ld_in, void* out, int64_t ld_out, int32_t elem_bytes, int64_t rows, int32_t cols,
                   void_stream_t stream) {
  if (rows < 0 || cols < 0 || (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4)) return VOID_ERR_BAD_ARG;
  if (rows == 0 || cols == 0) return VOID_OK;
  if (in == nullptr || out == nullptr) return VOID_ERR_BAD_ARG;
  if (ld_in % elem_bytes != 0 || ld_out % 16 != 0 || (reinterpret_cast<uintptr_t>(out) & 15u) != 0 ||
      (reinterpret_cast<uintptr_t>(in) & (uintptr_t)(elem_bytes - 1)) != 0)
    return VOID_ERR_ALIGN;
  if (ld_out < (int64_t)cols * elem_bytes) return VOID_ERR_SHAPE;
  const int64_t pieces = ld_out / 16, blocks = (rows * pieces + 255) / 256;
  if (blocks > 0x7fffffffLL) return VOID_ERR_TOO_LARGE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(256);
  cfg.stream = as_stream(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  uint4* dst = reinterpret_cast<uint4*>(out);
  cudaError_t rc;
  const int early = blocks <= 8ll * device_info().sms ? 1 : 0;   // 2048 threads per SM
  if (elem_bytes == 1) rc = cudaLaunchKernelEx(&cfg, copy_rows_kernel<uint8_t>, reinterpret_cast<const uint8_t*>(in), ld_in, dst, pieces, rows, cols, early);
  else if (elem_bytes == 2) rc = cudaLaunchKernelEx(&cfg, copy_rows_kernel<uint16_t>, reinterpret_cast<const uint16_t*>(in), ld_in / 2, dst, pieces, rows, cols, early);
  else rc = cudaLaunchKernelEx(&cfg, copy_rows_kernel<uint32_t>, reinterpret_cast<const uint32_t*>(in), ld_in / 4, dst, pieces, rows, cols, early);
  return status_of(rc);
}

int void_transpose(const void* in, int64_t ld_in, void* out, int64_t ld_out, int32_t elem_bytes, int32_t rows, int32_t cols,
                   void_stream_t stream) {
  if (rows < 0 || cols < 0 || (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4)) return VOID_ERR_BAD_ARG;
  if (rows == 0 || cols == 0) return VOID_OK;
  if (in == nullptr || out == nullptr) return VOID_ERR_BAD_ARG;
  if (ld_in % elem_bytes != 0 || ld_out % 16 != 0 || (reinterpret_cast<uintptr_t>(out) & 15u) != 0 ||
      (reinterpret_cast<uintptr_t>(in) & (uintptr_t)(elem_bytes - 1)) != 0)
    return VOID_ERR_ALIGN;
  if (ld_out < (int64_t)rows * elem_bytes || (rows > 1 && ld_in < (int64_t)cols * elem_bytes)) return VOID_ERR_SHAPE;
  const int side = 128 / elem_bytes, whole = (ld_in % 16 == 0 && (reinterpret_cast<uintptr_t>(in) & 15u) == 0) ? 1 : 0;
  const dim3 grid((unsigned)((cols + side - 1) / side), (unsigned)((rows + side - 1) / side));
  if (grid.y > 65535u) return VOID_ERR_TOO_LARGE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(256);
  cfg.stream = as_stream(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int64_t li = ld_in / elem_bytes, lo = ld_out / elem_bytes;
  cudaError_t rc;
  if (elem_bytes == 1) rc = cudaLaunchKernelEx(&cfg, transpose_kernel<uint8_t>, reinterpret_cast<const uint8_t*>(in), li, reinterpret_cast<uint8_t*>(out), lo, rows, cols, whole);
  else if (elem_bytes == 2) rc = cudaLaunchKernelEx(&cfg, transpose_kernel<uint16_t>, reinterpret_cast<const uint16_t*>(in), li, reinterpret_cast<uint16_t*>(out), lo, rows, cols, whole);
  else rc = cudaLaunchKernelEx(&cfg, transpose_kernel<uint32_t>, reinterpret_cast<const uint32_t*>(in), li, reinterpret_cast<uint32_t*>(out), lo, rows, cols, whole);
  return status_of(rc);
}

int void_column_sum(const void* in, int32_t elem, int64_t ld, int32_t rows, int32_t cols, void* out, void_stream_t stream) {
  if (rows < 0 || cols < 0 || ld < cols || elem < VOID_ELEM_F32 || elem > VOID_ELEM_BF16) return VOID_ERR_BAD_ARG;
  if (cols == 0) return VOID_OK;
  if (out == nullptr || (rows > 0 && in == nullptr)) return VOID_ERR_BAD_ARG;
  cudaStream_t st = as_stream(stream);
  const bool ok = elem == VOID_ELEM_F32   ? launch_column_sum<float>(in, ld, rows, cols, out, st)
                  : elem == VOID_ELEM_F16 ? launch_column_sum<__half>(in, ld, rows, cols, out, st)
                                          : launch_column_sum<__nv_bfloat16>(in, ld, rows, cols, out, st);
  return ok ? VOID_OK : VOID_ERR_CUDA;
}

int void_quant_tiles(const void* values, int32_t elem, int64_t nnz, int32_t kind, void* q, float* scale, float* scale_inv,
                     float* amax, int8_t* zero_points, const int32_t* block_rows, const int32_t* block_cols,
                     int32_t* rows_out, int32_t* cols_out, void_stream_t stream) {
  if (nnz < 0 || elem < VOID_ELEM_F32 || elem > VOID_ELEM_BF16 || (kind != VOID_KIND_I8 && kind != VOID_KIND_F8E4M3))
    return VOID_ERR_BAD_ARG;
  if (nnz == 0) return VOID_OK;
  if (values == nullptr || q == nullptr || scale == nullptr) return VOID_ERR_BAD_ARG;
  if ((rows_out != nullptr && block_rows == nullptr) || (cols_out != nullptr && block_cols == nullptr)) return VOID_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(values) & 15u) != 0 || (reinterpret_cast<uintptr_t>(q) & 3u) != 0) return VOID_ERR_ALIGN;
  const StoreExtras x{zero_points, block_rows, block_cols, rows_out, cols_out};
  const unsigned blocks = (unsigned)((nnz * 32 + 255) / 256);
  uint8_t* dst = reinterpret_cast<uint8_t*>(q);
  cudaStream_t st = as_stream(stream);
#define VB_QUANT(T)                                                                                                            \
  status_of(launch_pdl(kind == VOID_KIND_I8 ? quant_tiles_kernel<VOID_KIND_I8, T> : quant_tiles_kernel<VOID_KIND_F8E4M3, T>,    \
                       (int)blocks, 256, 0, st, reinterpret_cast<const T*>(values), nnz, dst, scale, scale_inv, amax, x))
  if (elem == VOID_ELEM_F32) return VB_QUANT(float);
  return elem == VOID_ELEM_F16 ? VB_QUANT(__half) : VB_QUANT(__nv_bfloat16);
#undef VB_QUANT
}

int void_quant_i8_tiles(const float* values, int64_t nnz, int8_t* q, float* scales, void_stream_t stream) {
  return void_quant_tiles(values, VOID_ELEM_F32, nnz, VOID_KIND_I8, q, scales, nullptr, nullptr, nullptr, nullptr, nullptr,
                          nullptr, nullptr, stream);
}

int void_quant_fp8_tiles(const float* values, int64_t nnz, uint8_t* q, float* scale, float* scale_inv, float* amax,
                         void_stream_t stream) {
  return void_quant_tiles(values, VOID_ELEM_F32, nnz, VOID_KIND_F8E4M3, q, scale, scale_inv, amax, nullptr, nullptr, nullptr,
                          nullptr, nullptr, stream);
}

static void quant_pass(const float* b, int64_t ldb, int K, int N, int kind, void* q, int64_t ldq, const float* scale,
                       int scale_stride, Launches& on) {
  const bool words = (ldq % 4 == 0) && ((reinterpret_cast<uintptr_t>(q) & 3u) == 0);
  const bool vec4 = words && (N % 4 == 0) && (ldb % 4 == 0) && ((reinterpret_cast<uintptr_t>(b) & 15u) == 0) &&
                    ((reinterpret_cast<uintptr_t>(scale) & 15u) == 0);
  // blockIdx.y is limited to 65535: quantise in slabs of rows
  for (int k0 = 0; k0 < K; k0 += 65535) {
    const int kk = (K - k0) < 65535 ? (K - k0) : 65535;
    const float* src = b + (size_t)k0 * ldb;
    uint8_t* dst = reinterpret_cast<uint8_t*>(q) + (size_t)k0 * ldq;
    if (words) {
      dim3 g2((unsigned)((ldq / 4 + 127) / 128), (unsigned)((kk + kColRows - 1) / kColRows));
      on.run(vec4 ? quant_cols4_kernel<true> : quant_cols4_kernel<false>, g2, 128, src, ldb, kk, N, kind, dst, ldq, scale, scale_stride);
    } else {
      dim3 g2((unsigned)((ldq + 255) / 256), kk);
      on.run(quant_cols_kernel, g2, 256, src, ldb, kk, N, kind, dst, ldq, scale, scale_stride);
    }
  }
}

int void_quant_cols(const float* b, int64_t ldb, int32_t K, int32_t N, int32_t kind, void* q, int64_t ldq,
                    float* col_scale, float* col_scale_inv, void_stream_t stream) {
  if (K < 0 || N < 0 || (kind != VOID_KIND_I8 && kind != VOID_KIND_F8E4M3)) return VOID_ERR_BAD_ARG;
  if (K == 0 || N == 0) return VOID_OK;
  if (b == nullptr || q == nullptr || col_scale == nullptr) return VOID_ERR_BAD_ARG;
  if (ldb < N || ldq < N) return VOID_ERR_SHAPE;
  if (K > 65535 * kRowSlab) return VOID_ERR_TOO_LARGE;
  cudaStream_t st = as_stream(stream);
  if (quant_cols_fused(b, ldb, K, N, kind, q, ldq, col_scale, col_scale_inv, st)) return VOID_OK;
  if (cudaMemsetAsync(col_scale, 0, (size_t)N * 4, st) != cudaSuccess) return VOID_ERR_CUDA;
  dim3 g1((N + kColBlock - 1) / kColBlock, (K + kRowSlab - 1) / kRowSlab);
  Launches on(st);
  on.run(col_amax_kernel, g1, kColBlock, b, ldb, K, N, col_scale);
  on.run(col_scale_kernel, (unsigned)((N + 255) / 256), 256, col_scale, col_scale_inv, N, kind);
  quant_pass(b, ldb, K, N, kind, q, ldq, col_scale, 1, on);
  return on.status();
}

int void_quant_i8_tensor(const float* b, int64_t ldb, int32_t K, int32_t N, void* q, int64_t ldq, float* scale,
                         void_stream_t stream) {
  if (K < 0 || N < 0) return VOID_ERR_BAD_ARG;
  if (b == nullptr || q == nullptr || scale == nullptr) return VOID_ERR_BAD_ARG;
  cudaStream_t st = as_stream(stream);
  if (cudaMemsetAsync(scale, 0, 4, st) != cudaSuccess) return VOID_ERR_CUDA;
  if (K == 0 || N == 0) return VOID_OK;
  if (ldb < N || ldq < N) return VOID_ERR_SHAPE;
  if (K > 65535 * kRowSlab) return VOID_ERR_TOO_LARGE;
  dim3 g1((N + kColBlock - 1) / kColBlock, (K + kRowSlab - 1) / kRowSlab);
  Launches on(st);
  on.run(tensor_amax_kernel, g1, kColBlock, b, ldb, K, N, scale);
  on.run(col_scale_kernel, 1, 32, scale, nullptr, 1, VOID_KIND_I8);
  quant_pass(b, ldb, K, N, VOID_KIND_I8, q, ldq, scale, 0, on);
  return on.status();
}

int64_t void_streamk_table_capacity(int64_t nnz, int32_t nbr) {
  (void)nbr;
  return nnz > 0 ? nnz : 1;
}

int32_t void_streamk_target(int64_t nnz, int32_t n_workers_req, int32_t max_work) {
  // target_work of compute_stream_k_workload, void/stream_k.py:61-67
  if (nnz <= 0) return 0;
  int64_t n_workers = n_workers_req > 0 ? n_workers_req : (nnz < 1024 ? nnz : 1024);
  int64_t target = (nnz + n_workers - 1) / n_workers;
  if (target > max_work) target = max_work;
  return (int32_t)target;
}

int void_streamk_table(const int32_t* row_ptr, int32_t nbr, int64_t nnz, int32_t n_workers_req, int32_t max_work,
                       int32_t* worker_rows, int32_t* worker_block_start, int32_t* worker_block_end,
                       uint8_t* worker_needs_atomic, int32_t* n_workers_out, int32_t* ws, void_stream_t stream) {
  if (row_ptr == nullptr || nbr <= 0 || nnz <= 0 || max_work <= 0) return VOID_ERR_BAD_ARG;
  if (worker_rows == nullptr || worker_block_start == nullptr || worker_block_end == nullptr ||
      worker_needs_atomic == nullptr || n_workers_out == nullptr || ws == nullptr)
    return VOID_ERR_BAD_ARG;
  const int target = void_streamk_target(nnz, n_workers_req, max_work);
  if (target <= 0) return VOID_ERR_BAD_ARG;
  Launches on(as_stream(stream));
  on.run(streamk_offsets_kernel, 1, 1024, row_ptr, nbr, target, ws, n_workers_out);
  on.run(streamk_fill_kernel, (unsigned)((nbr + 255) / 256), 256, row_ptr, nbr, target, ws, worker_rows, worker_block_start, worker_block_end,
         worker_needs_atomic);
  return on.status();
}

}  // extern "C"
