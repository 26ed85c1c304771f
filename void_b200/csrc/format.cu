// On-device construction of the VOID format: which 32x32 tiles of a dense or CSR matrix are kept,
// their Morton (Z-order) ranking, and the tile values.
//
// The reference builds the format on the host: dense_to_void (void/format.py:352-446) finds the
// active tiles with torch ops but computes and sorts the Morton codes in numpy, csr_to_void
// (:248-349) does everything in numpy with a Python loop over the nonzeros (:321-327).  Here the
// ranking is a bitmap in Morton-code space: bit morton(r, c) is set for every kept tile, a prefix
// sum of the words' population counts gives every set bit its rank, and rank order IS ascending
// Morton order - no sort.  All kernels are bandwidth-bound passes; none waits on another CTA.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/void_b200.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace vbf {

constexpr int kTile = 32;
constexpr int kChunkWords = 1024;  // words of the bitmap summed by one block
constexpr int kOneBlockWords = 32768;  // up to this many words (a grid side of 1024 tiles) one block ranks the bitmap
constexpr size_t kBitmapAt = 256;  // workspace: unsigned long long counts[2] (kept tiles, nonzero elements), then the bitmap

static inline cudaStream_t as_stream(void_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }
using vb::Launches;

// morton(r, c): bits of r on the even positions, bits of c on the odd ones (void/format.py:41-51)
__host__ __device__ inline uint32_t spread16(uint32_t v) {
  v = (v | (v << 8)) & 0x00FF00FFu;
  v = (v | (v << 4)) & 0x0F0F0F0Fu;
  v = (v | (v << 2)) & 0x33333333u;
  v = (v | (v << 1)) & 0x55555555u;
  return v;
}
__host__ __device__ inline uint32_t compact16(uint32_t v) {
  v &= 0x55555555u;
  v = (v | (v >> 1)) & 0x33333333u;
  v = (v | (v >> 2)) & 0x0F0F0F0Fu;
  v = (v | (v >> 4)) & 0x00FF00FFu;
  v = (v | (v >> 8)) & 0x0000FFFFu;
  return v;
}
__host__ __device__ inline uint32_t morton(uint32_t r, uint32_t c) { return spread16(r) | (spread16(c) << 1); }

// Side of the Morton square that holds the block grid (a power of two), and its bitmap size.
static int morton_side(int nbr, int nbc) {
  int s = 1;
  while (s < nbr || s < nbc) s <<= 1;
  return s;
}
struct WsLayout {
  int64_t words;       // 32-bit words of the bitmap
  int64_t chunks;      // blocks of kChunkWords words
  size_t clear_bytes;  // counts and bitmap stand first and are cleared together
  size_t off_prefix;   // int32 word_prefix[words + 1]
  size_t off_chunk;    // int32 chunk_ptr[chunks + 1]
  size_t bytes;
};
static bool ws_layout(int nbr, int nbc, WsLayout* w) {
  if (nbr <= 0 || nbc <= 0) { nbr = nbr > 0 ? nbr : 1; nbc = nbc > 0 ? nbc : 1; }
  const int64_t side = morton_side(nbr, nbc);
  if (side > 16384) return false;  // 2^28 bits = 32 MiB of bitmap is the largest grid built here
  const int64_t bits = side * side;
  w->words = (bits + 31) / 32;
  w->chunks = (w->words + kChunkWords - 1) / kChunkWords;
  size_t off = kBitmapAt + (size_t)w->words * 4;
  w->clear_bytes = off;
  off = (off + 255) & ~(size_t)255;
  w->off_prefix = off;
  off += (size_t)(w->words + 1) * 4;
  off = (off + 255) & ~(size_t)255;
  w->off_chunk = off;
  off += (size_t)(w->chunks + 1) * 4;
  w->bytes = off;
  return true;
}

template <typename T>
__device__ __forceinline__ float to_float(T v);
template <>
__device__ __forceinline__ float to_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// L1 norm and nonzero count per tile of the block grid (elements outside the matrix count as the zero padding of
// void/format.py:374-378); a tile is kept when its norm exceeds the threshold (:391-394).  A warp takes the 32 rows of a
// strip of 32 * V columns, every lane V of them: V elements are one 16-byte load where the rows allow it, otherwise V = 1
// and the strip is one tile.  Bound by reading the matrix once; the nonzero counts meet in shared memory first, since one
// atomic per tile on the same word cost as much as the reading (4096^2 fp32: 20.7 us before, 12.4 us now).
template <typename T, int V>
__global__ void __launch_bounds__(256) dense_mark_kernel(const T* __restrict__ a, int64_t ld, int M, int N, int nbr, int strips,
                                                         float threshold, uint32_t* __restrict__ bitmap,
                                                         unsigned long long* __restrict__ counts) {
  __shared__ int block_nz;
  if (threadIdx.x == 0) block_nz = 0;
  __syncthreads();
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const bool mine = warp < (int64_t)nbr * strips;
  const int r = mine ? (int)(warp / strips) : 0, strip = mine ? (int)(warp - (int64_t)r * strips) : 0;
  const int col = (strip * 32 + lane) * V;
  float norm = 0.0f;
  int nz = 0;
  auto add = [&](float v) {
    norm += fabsf(v);
    nz += (v != 0.0f) ? 1 : 0;
  };
  if (mine && col < N) {
    const int rows = M - r * kTile < kTile ? M - r * kTile : kTile;
    const T* src = a + (size_t)r * kTile * ld + col;
    if (V == 1 || col + V <= N) {
      if (rows == kTile) {
#pragma unroll
        for (int k0 = 0; k0 < kTile; k0 += 8) {
          T v[8][V];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if constexpr (V > 1) *reinterpret_cast<uint4*>(v[k]) = *reinterpret_cast<const uint4*>(src + (size_t)(k0 + k) * ld);
            else v[k][0] = src[(size_t)(k0 + k) * ld];
          }
#pragma unroll
          for (int k = 0; k < 8; ++k)
#pragma unroll
            for (int e = 0; e < V; ++e) add(to_float<T>(v[k][e]));
        }
      } else {
        for (int k = 0; k < rows; ++k)
#pragma unroll
          for (int e = 0; e < V; ++e) add(to_float<T>(src[(size_t)k * ld + e]));
      }
    } else {   // the last columns of a width that is no multiple of V
      for (int k = 0; k < rows; ++k)
        for (int e = 0; col + e < N; ++e) add(to_float<T>(src[(size_t)k * ld + e]));
    }
  }
  constexpr int kLanes = 32 / V;   // lanes of one tile
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) norm += __shfl_xor_sync(0xffffffffu, norm, o);
  nz = __reduce_add_sync(0xffffffffu, nz);
  if (mine && (lane & (kLanes - 1)) == 0 && col < N && norm > threshold) {
    const uint32_t code = morton((uint32_t)r, (uint32_t)(strip * V + lane / kLanes));
    atomicOr(bitmap + (code >> 5), 1u << (code & 31));
  }
  if (lane == 0 && nz) atomicAdd(&block_nz, nz);
  __syncthreads();
  if (threadIdx.x == 0 && block_nz) atomicAdd(counts + 1, (unsigned long long)block_nz);
}

// One warp per matrix row of a CSR matrix: every stored entry, zero or not, activates its tile
// (void/format.py:287-296).
__global__ void csr_mark_kernel(const int32_t* __restrict__ crow, const int32_t* __restrict__ col, int M,
                                uint32_t* __restrict__ bitmap) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= M) return;
  const int r = (int)warp / kTile;
  uint32_t last = 0xffffffffu;
  for (int i = crow[warp] + lane; i < crow[warp + 1]; i += 32) {
    const uint32_t code = morton((uint32_t)r, (uint32_t)(col[i] / kTile));
    if (code != last) atomicOr(bitmap + (code >> 5), 1u << (code & 31));
    last = code;
  }
}

// Rank of the first set bit of every word and the counts, by one block: the three levels below in one launch for the
// grids that most matrices have.
__global__ void __launch_bounds__(1024) rank_bitmap_kernel(const uint32_t* bitmap, int words,
                                                           int32_t* word_prefix,
                                                           const unsigned long long* counts,
                                                           int64_t* counts_out) {
  __shared__ int32_t warp_sum[32];
  vb::grid_dependency_wait();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int per = (words + 1023) / 1024;
  const int lo = tid * per < words ? tid * per : words, hi = lo + per < words ? lo + per : words;
  int c = 0;
  for (int i = lo; i < hi; ++i) c += __popc(bitmap[i]);
  int incl = c;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int s = warp_sum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += v;
    }
    warp_sum[lane] = s;
  }
  __syncthreads();
  int run = (wid ? warp_sum[wid - 1] : 0) + incl - c;
  for (int i = lo; i < hi; ++i) {
    word_prefix[i] = run;
    run += __popc(bitmap[i]);
  }
  if (tid == 1023) {
    word_prefix[words] = run;
    counts_out[0] = run;
    counts_out[1] = (int64_t)counts[1];
  }
}

// Level 1 of the prefix sum: set bits per chunk of kChunkWords words.
__global__ void __launch_bounds__(kChunkWords) chunk_count_kernel(const uint32_t* __restrict__ bitmap, int64_t words,
                                                                  int32_t* __restrict__ chunk_ptr) {
  __shared__ int32_t warp_sum[32];
  const int64_t w = (int64_t)blockIdx.x * kChunkWords + threadIdx.x;
  int c = (w < words) ? __popc(bitmap[w]) : 0;
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x < 32) {
    int s = warp_sum[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) chunk_ptr[blockIdx.x] = s;
  }
}

// Level 2: exclusive scan of the chunk counts by one block; the total is the number of kept tiles.
__global__ void __launch_bounds__(1024) chunk_scan_kernel(int32_t* chunk_ptr, int64_t chunks,
                                                          const unsigned long long* __restrict__ counts,
                                                          int64_t* __restrict__ counts_out) {
  __shared__ int32_t part[1024];
  const int tid = threadIdx.x;
  const int64_t per = (chunks + 1023) / 1024;
  const int64_t lo = tid * per < chunks ? tid * per : chunks;
  const int64_t hi = lo + per < chunks ? lo + per : chunks;
  int32_t s = 0;
  for (int64_t i = lo; i < hi; ++i) s += chunk_ptr[i];
  part[tid] = s;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    const int32_t v = (tid >= off) ? part[tid - off] : 0;
    __syncthreads();
    part[tid] += v;
    __syncthreads();
  }
  int32_t run = part[tid] - s;
  for (int64_t i = lo; i < hi; ++i) {
    const int32_t v = chunk_ptr[i];
    chunk_ptr[i] = run;
    run += v;
  }
  if (tid == 1023) {
    chunk_ptr[chunks] = part[1023];
    counts_out[0] = part[1023];
    counts_out[1] = (int64_t)counts[1];
  }
}

// Level 3: rank of the first set bit of every word.
__global__ void __launch_bounds__(kChunkWords) word_prefix_kernel(const uint32_t* __restrict__ bitmap, int64_t words,
                                                                  const int32_t* __restrict__ chunk_ptr,
                                                                  int32_t* __restrict__ word_prefix) {
  __shared__ int32_t warp_sum[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t w = (int64_t)blockIdx.x * kChunkWords + threadIdx.x;
  const int c = (w < words) ? __popc(bitmap[w]) : 0;
  int incl = c;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int s = warp_sum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += v;
    }
    warp_sum[lane] = s;  // inclusive over warps
  }
  __syncthreads();
  const int before = (wid ? warp_sum[wid - 1] : 0) + incl - c;
  if (w < words) word_prefix[w] = chunk_ptr[blockIdx.x] + before;
  if (w == words - 1) word_prefix[words] = chunk_ptr[blockIdx.x] + before + c;
}

// One thread per word: writes block_rows / block_cols / morton_codes of its set bits at their ranks.
__global__ void emit_index_kernel(const uint32_t* __restrict__ bitmap, const int32_t* __restrict__ word_prefix,
                                  int64_t words, int32_t* __restrict__ brow, int32_t* __restrict__ bcol,
                                  int64_t* __restrict__ codes) {
  const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= words) return;
  uint32_t bits = bitmap[w];
  int rank = word_prefix[w];
  while (bits) {
    const int b = __ffs(bits) - 1;
    bits &= bits - 1;
    const uint32_t code = (uint32_t)(w * 32 + b);
    brow[rank] = (int32_t)compact16(code);
    bcol[rank] = (int32_t)compact16(code >> 1);
    codes[rank] = (int64_t)code;
    ++rank;
  }
}

// values[i] = tile (block_rows[i], block_cols[i]) of the dense matrix, zero outside the matrix.
// 128 threads per tile, eight elements each (tile rows e/32, e/32 + 4, ...): eight independent loads in flight
// per thread, every warp reading and writing 128 contiguous bytes per instruction.
template <typename T>
__global__ void dense_gather_kernel(const T* __restrict__ a, int64_t ld, int M, int N,
                                    const int32_t* __restrict__ brow, const int32_t* __restrict__ bcol, int64_t n_blocks,
                                    T* __restrict__ values) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t t = g >> 7;
  if (t >= n_blocks) return;
  const int e0 = (int)(g & 127);
  const int row0 = brow[t] * kTile + (e0 >> 5), col = bcol[t] * kTile + (e0 & 31);
  T v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int row = row0 + 4 * k;
    v[k] = (row < M && col < N) ? a[(size_t)row * ld + col] : T(0.0f);
  }
  T* dst = values + t * (kTile * kTile) + e0;
#pragma unroll
  for (int k = 0; k < 8; ++k) dst[k * 128] = v[k];
}

// Both for the grids that most matrices have: a block takes a word of the bitmap, each of its eight warps four bits of it, and
// copies the tiles that are set, writing their coordinates on the way.  V elements are a 16-byte piece of a row, or 1.
// 4096^2, 80 %, fp32 (13 MB each way, cold): 7.1 us against 3.8 + 5.1 and the gap between two launches.
constexpr int kFusedWords = 8192;   // a grid side of 512 tiles
template <typename T, int V>
__global__ void __launch_bounds__(256) emit_tiles_kernel(const uint32_t* __restrict__ bitmap, const int32_t* __restrict__ word_prefix,
                                                         const T* __restrict__ a, int64_t ld, int M, int N, int64_t n_blocks,
                                                         int32_t* __restrict__ brow, int32_t* __restrict__ bcol,
                                                         int64_t* __restrict__ codes, T* __restrict__ values) {
  constexpr int PER_ROW = kTile / V, ROWS = 32 / PER_ROW;   // lanes of a tile row, rows a warp reads at once
  const int lane = threadIdx.x & 31, first = (int)(threadIdx.x >> 5) * 4;
  const uint32_t word = bitmap[blockIdx.x];
  const int row = lane / PER_ROW, col = lane % PER_ROW * V;
  for (uint32_t bits = word & (0xfu << first); bits != 0u; bits &= bits - 1u) {
    const int b = __ffs((int)bits) - 1;
    const uint32_t code = blockIdx.x * 32u + (uint32_t)b;
    const int64_t rank = word_prefix[blockIdx.x] + __popc(word & ((1u << b) - 1u));
    if (rank >= n_blocks) return;
    const int r = (int)compact16(code), c = (int)compact16(code >> 1);
    if (lane == 0) {
      brow[rank] = r;
      bcol[rank] = c;
      codes[rank] = (int64_t)code;
    }
    const T* src = a + (size_t)(r * kTile + row) * ld + c * kTile + col;
    T* dst = values + rank * (kTile * kTile) + row * kTile + col;
    if constexpr (V > 1) {
      if ((r + 1) * kTile <= M && (c + 1) * kTile <= N) {
        uint4 v[kTile / ROWS];
#pragma unroll
        for (int k = 0; k < kTile / ROWS; ++k) v[k] = *reinterpret_cast<const uint4*>(src + (size_t)(k * ROWS) * ld);
#pragma unroll
        for (int k = 0; k < kTile / ROWS; ++k) *reinterpret_cast<uint4*>(dst + k * ROWS * kTile) = v[k];
        continue;
      }
    }
#pragma unroll 8
    for (int k = 0; k < kTile / ROWS; ++k)
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const bool in = r * kTile + row + k * ROWS < M && c * kTile + col + e < N;
        dst[k * ROWS * kTile + e] = in ? src[(size_t)(k * ROWS) * ld + e] : T(0.0f);
      }
  }
}

// One warp per matrix row of the CSR matrix: every stored entry goes to its place in its tile.
// Two entries with the same coordinates (a non-canonical CSR) race; the reference keeps the later one.
__global__ void csr_scatter_kernel(const int32_t* __restrict__ crow, const int32_t* __restrict__ col,
                                   const float* __restrict__ data, int M, const uint32_t* __restrict__ bitmap,
                                   const int32_t* __restrict__ word_prefix, float* __restrict__ values) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= M) return;
  const int r = (int)warp / kTile, rr = (int)warp % kTile;
  for (int i = crow[warp] + lane; i < crow[warp + 1]; i += 32) {
    const int c = col[i];
    const uint32_t code = morton((uint32_t)r, (uint32_t)(c / kTile));
    const int rank = word_prefix[code >> 5] + __popc(bitmap[code >> 5] & ((1u << (code & 31)) - 1u));
    values[(size_t)rank * (kTile * kTile) + rr * kTile + (c % kTile)] = data[i];
  }
}

static uint32_t* bitmap_of(void* ws) { return reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(ws) + kBitmapAt); }
static const uint32_t* bitmap_of(const void* ws) {
  return reinterpret_cast<const uint32_t*>(static_cast<const unsigned char*>(ws) + kBitmapAt);
}

static int rank_bitmap(const WsLayout& w, unsigned char* ws, int64_t* counts_out, cudaStream_t st) {
  const uint32_t* bitmap = bitmap_of(ws);
  int32_t* word_prefix = reinterpret_cast<int32_t*>(ws + w.off_prefix);
  int32_t* chunk_ptr = reinterpret_cast<int32_t*>(ws + w.off_chunk);
  const unsigned long long* counts = reinterpret_cast<const unsigned long long*>(ws);
  if (w.words <= kOneBlockWords) {
    return vb::status_of(vb::launch_pdl(rank_bitmap_kernel, 1, 1024, 0, st, bitmap, (int)w.words, word_prefix, counts, counts_out));
  }
  Launches on(st);
  on.run(chunk_count_kernel, (unsigned)w.chunks, kChunkWords, bitmap, w.words, chunk_ptr);
  on.run(chunk_scan_kernel, 1, 1024, chunk_ptr, w.chunks, counts, counts_out);
  on.run(word_prefix_kernel, (unsigned)w.chunks, kChunkWords, bitmap, w.words, chunk_ptr, word_prefix);
  return on.status();
}

template <typename T>
static int launch_dense_mark(const void* matrix, int64_t ld, int M, int N, float threshold, void* ws, cudaStream_t st) {
  constexpr int kVec = 16 / (int)sizeof(T);
  const int nbr = (M + kTile - 1) / kTile;
  const T* a = static_cast<const T*>(matrix);
  const bool vec = ld % kVec == 0 && (reinterpret_cast<uintptr_t>(matrix) & 15u) == 0;
  const int strips = (N + 32 * (vec ? kVec : 1) - 1) / (32 * (vec ? kVec : 1));
  const unsigned blocks = (unsigned)(((int64_t)nbr * strips + 7) / 8);
  unsigned long long* counts = static_cast<unsigned long long*>(ws);
  Launches on(st);
  on.run(vec ? dense_mark_kernel<T, kVec> : dense_mark_kernel<T, 1>, blocks, 256, a, ld, M, N, nbr, strips, threshold, bitmap_of(ws), counts);
  return on.status();
}

template <typename T>
static int launch_emit_tiles(const WsLayout& w, const void* ws, const void* matrix, int64_t ld, int M, int N, int64_t n_blocks,
                             int32_t* brow, int32_t* bcol, int64_t* codes, void* values, cudaStream_t st) {
  constexpr int kVec = 16 / (int)sizeof(T);
  const int32_t* prefix = reinterpret_cast<const int32_t*>(static_cast<const unsigned char*>(ws) + w.off_prefix);
  const T* a = static_cast<const T*>(matrix);
  const bool vec = ld % kVec == 0 && ((reinterpret_cast<uintptr_t>(matrix) | reinterpret_cast<uintptr_t>(values)) & 15u) == 0;
  Launches on(st);
  on.run(vec ? emit_tiles_kernel<T, kVec> : emit_tiles_kernel<T, 1>, (unsigned)w.words, 256, bitmap_of(ws), prefix, a, ld, M, N, n_blocks, brow, bcol,
         codes, static_cast<T*>(values));
  return on.status();
}

}  // namespace vbf

extern "C" {

size_t void_format_ws_bytes(int32_t nbr, int32_t nbc) {
  vbf::WsLayout w;
  return vbf::ws_layout(nbr, nbc, &w) ? w.bytes : 0;
}

int void_dense_mark(const void* matrix, int32_t elem, int64_t ld, int32_t M, int32_t N, float threshold, void* ws,
                    size_t ws_bytes, int64_t* counts_out, void_stream_t stream) {
  if (M < 0 || N < 0 || ld < N || counts_out == nullptr) return VOID_ERR_BAD_ARG;
  if (elem < VOID_ELEM_F32 || elem > VOID_ELEM_BF16) return VOID_ERR_BAD_ARG;
  const int nbr = (M + vbf::kTile - 1) / vbf::kTile, nbc = (N + vbf::kTile - 1) / vbf::kTile;
  vbf::WsLayout w;
  if (!vbf::ws_layout(nbr, nbc, &w)) return VOID_ERR_TOO_LARGE;
  if (ws == nullptr || ws_bytes < w.bytes) return VOID_ERR_WORKSPACE;
  if ((int64_t)nbr * nbc > 0 && matrix == nullptr) return VOID_ERR_BAD_ARG;
  cudaStream_t st = vbf::as_stream(stream);
  if (cudaMemsetAsync(ws, 0, w.clear_bytes, st) != cudaSuccess) return VOID_ERR_CUDA;
  if ((int64_t)nbr * nbc > 0) {
    const int rc = elem == VOID_ELEM_F32   ? vbf::launch_dense_mark<float>(matrix, ld, M, N, threshold, ws, st)
                   : elem == VOID_ELEM_F16 ? vbf::launch_dense_mark<__half>(matrix, ld, M, N, threshold, ws, st)
                                           : vbf::launch_dense_mark<__nv_bfloat16>(matrix, ld, M, N, threshold, ws, st);
    if (rc != VOID_OK) return rc;
  }
  return vbf::rank_bitmap(w, static_cast<unsigned char*>(ws), counts_out, st);
}

int void_csr_mark(const int32_t* crow, const int32_t* col, int32_t M, int32_t N, void* ws, size_t ws_bytes,
                  int64_t* counts_out, void_stream_t stream) {
  if (M < 0 || N < 0 || counts_out == nullptr) return VOID_ERR_BAD_ARG;
  const int nbr = (M + vbf::kTile - 1) / vbf::kTile, nbc = (N + vbf::kTile - 1) / vbf::kTile;
  vbf::WsLayout w;
  if (!vbf::ws_layout(nbr, nbc, &w)) return VOID_ERR_TOO_LARGE;
  if (ws == nullptr || ws_bytes < w.bytes) return VOID_ERR_WORKSPACE;
  if (M > 0 && crow == nullptr) return VOID_ERR_BAD_ARG;  // col may be null for a matrix without entries
  cudaStream_t st = vbf::as_stream(stream);
  if (cudaMemsetAsync(ws, 0, w.clear_bytes, st) != cudaSuccess) return VOID_ERR_CUDA;
  if (M > 0) {
    vbf::Launches on(st);
    on.run(vbf::csr_mark_kernel, (unsigned)(((int64_t)M * 32 + 255) / 256), 256, crow, col, M, vbf::bitmap_of(ws));
    if (on.status() != VOID_OK) return on.status();
  }
  return vbf::rank_bitmap(w, static_cast<unsigned char*>(ws), counts_out, st);
}

int void_morton_emit(const void* ws, int32_t nbr, int32_t nbc, int64_t n_blocks, int32_t* block_rows,
                     int32_t* block_cols, int64_t* morton_codes, void_stream_t stream) {
  vbf::WsLayout w;
  if (!vbf::ws_layout(nbr, nbc, &w)) return VOID_ERR_TOO_LARGE;
  if (n_blocks < 0 || ws == nullptr) return VOID_ERR_BAD_ARG;
  if (n_blocks == 0) return VOID_OK;
  if (block_rows == nullptr || block_cols == nullptr || morton_codes == nullptr) return VOID_ERR_BAD_ARG;
  const unsigned char* base = static_cast<const unsigned char*>(ws);
  vbf::Launches on(vbf::as_stream(stream));
  on.run(vbf::emit_index_kernel, (unsigned)((w.words + 255) / 256), 256, vbf::bitmap_of(ws), reinterpret_cast<const int32_t*>(base + w.off_prefix),
         w.words, block_rows, block_cols, morton_codes);
  return on.status();
}

int void_dense_gather(const void* matrix, int32_t elem, int64_t ld, int32_t M, int32_t N, const int32_t* block_rows,
                      const int32_t* block_cols, int64_t n_blocks, void* values, void_stream_t stream) {
  if (n_blocks < 0 || M < 0 || N < 0 || ld < N) return VOID_ERR_BAD_ARG;
  if (elem < VOID_ELEM_F32 || elem > VOID_ELEM_BF16) return VOID_ERR_BAD_ARG;
  if (n_blocks == 0) return VOID_OK;
  if (matrix == nullptr || block_rows == nullptr || block_cols == nullptr || values == nullptr) return VOID_ERR_BAD_ARG;
  vbf::Launches on(vbf::as_stream(stream));
  const unsigned blocks = (unsigned)((n_blocks * 128 + 255) / 256);
  if (elem == VOID_ELEM_F32)
    on.run(vbf::dense_gather_kernel<float>, blocks, 256, static_cast<const float*>(matrix), ld, M, N, block_rows, block_cols, n_blocks,
           static_cast<float*>(values));
  else if (elem == VOID_ELEM_F16)
    on.run(vbf::dense_gather_kernel<__half>, blocks, 256, static_cast<const __half*>(matrix), ld, M, N, block_rows, block_cols, n_blocks,
           static_cast<__half*>(values));
  else
    on.run(vbf::dense_gather_kernel<__nv_bfloat16>, blocks, 256, static_cast<const __nv_bfloat16*>(matrix), ld, M, N, block_rows, block_cols,
           n_blocks, static_cast<__nv_bfloat16*>(values));
  return on.status();
}

int void_dense_emit(const void* ws, const void* matrix, int32_t elem, int64_t ld, int32_t M, int32_t N, int64_t n_blocks,
                    int32_t* block_rows, int32_t* block_cols, int64_t* morton_codes, void* values, void_stream_t stream) {
  if (n_blocks < 0 || M < 0 || N < 0 || ld < N || ws == nullptr) return VOID_ERR_BAD_ARG;
  if (elem < VOID_ELEM_F32 || elem > VOID_ELEM_BF16) return VOID_ERR_BAD_ARG;
  if (n_blocks == 0) return VOID_OK;
  const int nbr = (M + vbf::kTile - 1) / vbf::kTile, nbc = (N + vbf::kTile - 1) / vbf::kTile;
  vbf::WsLayout w;
  if (!vbf::ws_layout(nbr, nbc, &w)) return VOID_ERR_TOO_LARGE;
  if (w.words > vbf::kFusedWords) {
    const int st = void_morton_emit(ws, nbr, nbc, n_blocks, block_rows, block_cols, morton_codes, stream);
    return st != VOID_OK ? st : void_dense_gather(matrix, elem, ld, M, N, block_rows, block_cols, n_blocks, values, stream);
  }
  if (matrix == nullptr || block_rows == nullptr || block_cols == nullptr || morton_codes == nullptr || values == nullptr)
    return VOID_ERR_BAD_ARG;
  cudaStream_t st = vbf::as_stream(stream);
  if (elem == VOID_ELEM_F32) return vbf::launch_emit_tiles<float>(w, ws, matrix, ld, M, N, n_blocks, block_rows, block_cols, morton_codes, values, st);
  if (elem == VOID_ELEM_F16) return vbf::launch_emit_tiles<__half>(w, ws, matrix, ld, M, N, n_blocks, block_rows, block_cols, morton_codes, values, st);
  return vbf::launch_emit_tiles<__nv_bfloat16>(w, ws, matrix, ld, M, N, n_blocks, block_rows, block_cols, morton_codes, values, st);
}

int void_csr_scatter(const int32_t* crow, const int32_t* col, const float* data, int32_t M, int32_t N, const void* ws,
                     int64_t n_blocks, float* values, void_stream_t stream) {
  if (M < 0 || N < 0 || n_blocks < 0) return VOID_ERR_BAD_ARG;
  if (n_blocks == 0 || M == 0) return VOID_OK;
  if (crow == nullptr || col == nullptr || data == nullptr || ws == nullptr || values == nullptr) return VOID_ERR_BAD_ARG;
  const int nbr = (M + vbf::kTile - 1) / vbf::kTile, nbc = (N + vbf::kTile - 1) / vbf::kTile;
  vbf::WsLayout w;
  if (!vbf::ws_layout(nbr, nbc, &w)) return VOID_ERR_TOO_LARGE;
  cudaStream_t st = vbf::as_stream(stream);
  if (cudaMemsetAsync(values, 0, (size_t)n_blocks * 4096, st) != cudaSuccess) return VOID_ERR_CUDA;
  const unsigned char* base = static_cast<const unsigned char*>(ws);
  vbf::Launches on(st);
  on.run(vbf::csr_scatter_kernel, (unsigned)(((int64_t)M * 32 + 255) / 256), 256, crow, col, data, M, vbf::bitmap_of(ws),
         reinterpret_cast<const int32_t*>(base + w.off_prefix), values);
  return on.status();
}

}  // extern "C"
