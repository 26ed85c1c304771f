// Device-side work splitter of the SpMM kernels.
//
// The work of one launch is the sequence of "virtual rows" v = (column chunk c, tile row r),
// v = c * nbr + r, each worth (tiles in row r) + row_cost units.  row_cost stands for the epilogue:
// reading the accumulator back, dequantising, activating and storing 32 x chunk columns costs as
// much as several tiles of products, and empty rows still have to be written as zeros.  Because
// row_ptr is already a prefix sum, the start position of a virtual row on that axis is closed-form:
// P(v) = c * (nnz + row_cost * nbr) + row_ptr[r] + row_cost * r.  The axis is cut into n_cta shares of
// equal length; cut k lands inside some row and is then moved
//   mode 0  to the nearer tile-row boundary (rows are never split),
//   mode 1  to the nearer tile-row boundary if the row is light, else to the nearest multiple of
//           `chunk_tiles` inside the row (the chunk boundaries of the Stream-K worker table,
//           void/stream_k.py:84-97), so that a heavy row is shared by several CTAs,
//   mode 2  always to the nearest chunk boundary, and every chunk becomes a segment of its
//           own (one segment per worker of the reference table; used to check partial sums).
// Mode 3 deals segments out instead of cutting an axis (deal_kernel below).
// A row that ends up in several segments gets a counter and one partial-sum slot per segment;
// the SpMM kernel's last arriver adds the slots up.
//
// The same code runs as one 1024-thread block on the device (the product path) and, for
// tests of the splitting arithmetic on machines without a GPU, as plain loops on the host.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/void_b200.h"
#include "launch.cuh"

namespace vb {

struct PlanIn {
  const int32_t* row_ptr;
  const int32_t* woff;  // mode 2: workers before each row (nbr + 1), else null
  int nbr, n_chunks, n_cta, mode, chunk_tiles;
  int row_cost;  // what finishing one (tile row, chunk) costs, in units of one tile's work
};

struct PlanWs {       // all arrays have n_cta + 2 entries
  int32_t* bv;        // boundary: virtual row
  int32_t* bo;        // boundary: tile offset inside the row
  int32_t* lead_nseg; // segments of the split row whose first interior cut is this boundary, else 0
  int32_t* lead_flag; // 1 at such a boundary
  int32_t* slot_off;  // exclusive scans of the two above
  int32_t* ctr_off;
  int32_t* nseg_cta;  // segments per CTA, scanned into cta_seg_ptr
};

__host__ __device__ inline int row_cnt(const PlanIn& in, int v) {
  const int r = v % in.nbr;
  return in.row_ptr[r + 1] - in.row_ptr[r];
}

// phase 1: boundary j in [0, n_cta]
__host__ __device__ inline void plan_boundary(const PlanIn& in, const PlanWs& ws, int j) {
  const long long c0 = in.row_cost;
  const long long nnz = in.row_ptr[in.nbr];
  const long long wrow = nnz + c0 * in.nbr;
  const long long W = wrow * in.n_chunks;
  const int V = in.nbr * in.n_chunks;
  if (j >= in.n_cta) {
    ws.bv[j] = V;
    ws.bo[j] = 0;
    return;
  }
  const long long x = (W * j) / in.n_cta;
  const int c = (int)(x / wrow);
  const long long y = x - (long long)c * wrow;
  int lo = 0, hi = in.nbr - 1;  // largest r with row_ptr[r] + c0 * r <= y
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((long long)in.row_ptr[mid] + c0 * mid <= y) lo = mid;
    else hi = mid - 1;
  }
  const int r = lo;
  const long long d = y - ((long long)in.row_ptr[r] + c0 * r);  // 0 .. cnt + c0 - 1
  const int cnt = in.row_ptr[r + 1] - in.row_ptr[r];
  int v = c * in.nbr + r, o = 0;
  const long long share = W / in.n_cta;
  const bool splittable = in.chunk_tiles > 0 && cnt > 0 &&
                          (in.mode == 2 || (in.mode == 1 && (long long)cnt + c0 > share));
  if (d == 0) {
    o = 0;
  } else if (!splittable) {
    if (2 * d >= (long long)cnt + c0) v += 1;  // nearer end of the row
    o = 0;
  } else {
    const int T = in.chunk_tiles;
    const long long tile = d > c0 ? d - c0 : 0;  // the row's own cost comes first on the axis
    o = (int)(((tile + T / 2) / T) * T);
    if (o >= cnt) { v += 1; o = 0; }
  }
  ws.bv[j] = v;
  ws.bo[j] = o;
}

// number of distinct interior offsets of row bv[j] among boundaries j, j+1, ... (bo[j] > 0)
__host__ __device__ inline int distinct_from(const PlanWs& ws, int j, int n_cta) {
  const int v = ws.bv[j];
  int m = 1, prev = ws.bo[j];
  for (int i = j + 1; i <= n_cta && ws.bv[i] == v; ++i) {
    if (ws.bo[i] != prev) { ++m; prev = ws.bo[i]; }
  }
  return m;
}

// phase 2: leaders of split rows (modes 0/1), segments per CTA
__host__ __device__ inline void plan_leaders(const PlanIn& in, const PlanWs& ws, int j) {
  int lead = 0, nseg = 0;
  if (in.mode != 2 && j <= in.n_cta && ws.bo[j] > 0) {
    const bool first = (j == 0) || ws.bv[j - 1] != ws.bv[j] || ws.bo[j - 1] == 0;
    if (first) { lead = 1; nseg = distinct_from(ws, j, in.n_cta) + 1; }
  }
  ws.lead_flag[j] = lead;
  ws.lead_nseg[j] = nseg;
  if (j < in.n_cta) {
    const int va = ws.bv[j], oa = ws.bo[j], vb = ws.bv[j + 1], ob = ws.bo[j + 1];
    const int T = in.chunk_tiles;
    int n;
    if (in.mode != 2) {
      n = (va == vb) ? (ob > oa ? 1 : 0) : 1 + (vb - va - 1) + (ob > 0 ? 1 : 0);
    } else {
      if (va == vb) {
        n = (ob - oa + T - 1) / T;
      } else {
        const int ca = row_cnt(in, va);
        n = (ca - oa + T - 1) / T;
        if (ca == 0) n = 1;
        for (int v = va + 1; v < vb; ++v) {
          const int cv = row_cnt(in, v);
          n += cv == 0 ? 1 : (cv + T - 1) / T;
        }
        n += (ob + T - 1) / T;
      }
    }
    ws.nseg_cta[j] = n;
  } else {
    ws.nseg_cta[j] = 0;
  }
}

__host__ __device__ inline void put_seg(int32_t* segs, long long idx, int row, int chunk, int t0, int t1, int nseg,
                                        int slot0, int my_idx, int ctr) {
  int32_t* s = segs + idx * 8;
  s[0] = row; s[1] = chunk; s[2] = t0; s[3] = t1; s[4] = nseg; s[5] = slot0; s[6] = my_idx; s[7] = ctr;
}

// emits the piece [a, b) of virtual row v (tile offsets inside the row); returns segments written
__host__ __device__ inline int emit_piece(const PlanIn& in, const PlanWs& ws, int32_t* segs, long long at,
                                          long long capacity, int v, int a, int b, int k_start) {
  const int r = v % in.nbr, c = v / in.nbr;
  const int rs = in.row_ptr[r], cnt = in.row_ptr[r + 1] - rs;
  if (in.mode == 2) {
    const int T = in.chunk_tiles;
    const int nseg = cnt == 0 ? 1 : (cnt + T - 1) / T;
    const int n_workers = in.woff[in.nbr];
    const int slot0 = c * n_workers + in.woff[r];
    int n = 0;
    if (cnt == 0) {
      if (at < capacity) put_seg(segs, at, r, c, rs, rs, 1, 0, 0, 0);
      return 1;
    }
    for (int t = a; t < b; t += T, ++n) {
      const int e = (t + T) < b ? (t + T) : b;
      if (at + n < capacity) put_seg(segs, at + n, r, c, rs + t, rs + e, nseg, slot0, t / T, v);
    }
    return n;
  }
  int nseg = 1, slot0 = 0, my_idx = 0, ctr = 0;
  if (a > 0 || b < cnt) {
    // find the first interior boundary (leader) of this row: k_start is a boundary index inside or
    // at the edge of the row; walk back while the previous boundary is interior to the same row
    int j = k_start;
    if (!(ws.bv[j] == v && ws.bo[j] > 0)) j = k_start + 1;  // piece starts at the row start
    while (j > 0 && ws.bv[j - 1] == v && ws.bo[j - 1] > 0) --j;
    nseg = ws.lead_nseg[j];
    slot0 = ws.slot_off[j];
    ctr = ws.ctr_off[j];
    if (a > 0) {
      int prev = -1;
      for (int i = j; i <= in.n_cta && ws.bv[i] == v && ws.bo[i] <= a; ++i)
        if (ws.bo[i] != prev) { ++my_idx; prev = ws.bo[i]; }
    }
  }
  if (at < capacity) put_seg(segs, at, r, c, rs + a, rs + b, nseg, slot0, my_idx, ctr);
  return 1;
}

// phase 4: CTA k writes its segments starting at cta_seg_ptr[k]
__host__ __device__ inline void plan_emit(const PlanIn& in, const PlanWs& ws, const int32_t* cta_seg_ptr,
                                          int32_t* segs, long long capacity, int k) {
  const int va = ws.bv[k], oa = ws.bo[k], vb = ws.bv[k + 1], ob = ws.bo[k + 1];
  long long at = cta_seg_ptr[k];
  if (va == vb) {
    if (ob > oa) at += emit_piece(in, ws, segs, at, capacity, va, oa, ob, k);
    return;
  }
  at += emit_piece(in, ws, segs, at, capacity, va, oa, row_cnt(in, va), k);
  for (int v = va + 1; v < vb; ++v) at += emit_piece(in, ws, segs, at, capacity, v, 0, row_cnt(in, v), k);
  if (ob > 0) at += emit_piece(in, ws, segs, at, capacity, vb, 0, ob, k);
}

// single-block exclusive scan, n + 1 outputs (out[n] = total); in/out may alias
__device__ void plan_scan(const int32_t* in, int32_t* out, int n) {
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
  int32_t run = part[tid] - s;
  for (int i = lo; i < hi; ++i) {
    const int32_t v = in[i];
    out[i] = run;
    run += v;
  }
  if (tid == 1023) out[n] = part[1023];
  __syncthreads();
}

__global__ void __launch_bounds__(1024) plan_kernel(PlanIn in, PlanWs ws, int32_t* segs, long long capacity,
                                                    int32_t* cta_seg_ptr, int32_t* counts) {
  const int G = in.n_cta;
  for (int j = threadIdx.x; j <= G; j += blockDim.x) plan_boundary(in, ws, j);
  __syncthreads();
  for (int j = threadIdx.x; j <= G; j += blockDim.x) plan_leaders(in, ws, j);
  __syncthreads();
  plan_scan(ws.lead_nseg, ws.slot_off, G + 1);
  plan_scan(ws.lead_flag, ws.ctr_off, G + 1);
  plan_scan(ws.nseg_cta, cta_seg_ptr, G);
  for (int k = threadIdx.x; k < G; k += blockDim.x) plan_emit(in, ws, cta_seg_ptr, segs, capacity, k);
  if (threadIdx.x == 0) {
    counts[0] = cta_seg_ptr[G];
    if (in.mode == 2) {
      counts[1] = in.n_chunks * in.woff[in.nbr];
      counts[2] = in.n_chunks * in.nbr;
    } else {
      counts[1] = ws.slot_off[G + 1];
      counts[2] = ws.ctr_off[G + 1];
    }
    counts[3] = (cta_seg_ptr[G] > capacity) ? 1 : 0;  // overflow flag
  }
}

// ------------------------------------------------------------------------------------------ mode 3: segments dealt out
// Every virtual row is a segment; one heavier than kDealLimit shares is cut into pieces.  The segments go, the heaviest first, each
// to a CTA that has the least so far.  A piece costs what its tiles do and `piece` units more, since its sums travel through memory
// and its last arriver reads them back: from time stamps, a CTA's end moves by 0.14 us per tile, 1.7 per whole row and 2.5 - 4 per
// piece (16384^2, N = 256, power-law rows), so contiguous shares of equal tiles and rows ended between 8 and 15 us.  us, shares of
// mode 1 and dealt, products of a graph: 16384^2, N = 256 13.5 12.2, N = 500 28.5 25.3, N = 1024 34.4 31.3; 32768 x 8192, N = 512 27.0 24.0;
// 8192 x 32768, N = 200 16.6 15.1; 30000 x 3000, N = 60 10.7 8.7; 4096 x 8192, N = 128 8.1 6.0; 2048 x 16384, N = 128 8.6 6.2.  (Launched one by one, 16384^2,
// N = 256: a piece at 2, 3, 4, 6 row costs 13.5 13.2 13.0 14.8; limits of 1.15, 1.3, 1.5, 2 shares 13.1 13.0 13.0 14.1, N = 1024 36.8 35.1 32.6 -;
// dealt back and forth without regard to the load 17.)
constexpr double kDealLimit = 1.5;
constexpr int kDealMaxSegs = 8192, kDealMaxCtas = 1024;   // sorted and kept in one block's shared memory
constexpr int kDealThreads = 1024;

// Pieces of a row of cnt tiles when a CTA's share is `share`.
__host__ __device__ inline int deal_pieces(int cnt, int row_cost, int piece, double share) {
  if (cnt < 2 || (double)(cnt + row_cost) <= kDealLimit * share) return 1;
  const double most = kDealLimit * share - piece, tiles = most > 0.5 * share ? most : 0.5 * share;
  const double k = ceil((double)cnt / tiles);
  return k < 2.0 ? 1 : (k < (double)cnt ? (int)k : cnt);
}
__host__ __device__ inline int deal_cost(int cnt, int k, int row_cost, int piece) { return k > 1 ? cnt + k * piece : cnt + row_cost; }
// Rounds in which the share is taken from the work at the share before.  Pieces make work and a larger share makes fewer pieces, so it
// swings about the one at which the work fits, and an odd number of rounds ends on the high side.  With many rows the two are close
// (512 rows, two chunks: 40.7, 63.9, 51.6, 54.5; 54.2 fits), with few long ones far apart (64 rows of 27 tiles: 3.8, 28.3, 5.3, 21.0; 11.4
// fits), and then fewer segments than CTAs are the better plan: 155 against 336 of 592, 2048 x 32768, N = 60 7.6 against 10.1 us.  Three rounds, the
// share that fits (found by halving), contiguous shares: N = 256 there 7.6 9.5 9.4; 2048 x 16384, N = 128 6.2 8.7 8.6; 4096 x 32768, N = 128 8.0 9.4
// 9.4; 4096 x 16384, N = 256 8.1 9.3 10.7.  Between, where the segments nearly fill the CTAs, the other way round: 8192 x 16384, N = 256 10.1 9.0
// 10.9; 8192 x 32768, N = 200 15.1 14.9 16.6.  From two segments per CTA on no difference.
constexpr int kDealRounds = 3;
// What a piece costs: four row costs, two where that leaves CTAs without a segment.
__host__ __device__ inline int deal_piece(int row_cost, int attempt) { return (attempt == 0 ? 4 : 2) * row_cost; }
// The heaviest first, of equal ones the first.
__host__ __device__ inline unsigned long long deal_key(int cost, int idx) {
  return ((unsigned long long)(0x7fffffffu - (uint32_t)cost) << 32) | (uint32_t)idx;
}
__host__ __device__ inline int deal_key_cost(unsigned long long key) { return (int)(0x7fffffffu - (uint32_t)(key >> 32)); }
// CTAs are compared by load and number in 32 bits; loads that do not fit are compared without their last bits.
__host__ __device__ inline int deal_shift(long long total) {
  int s = 0;
  while ((total >> s) >= (1ll << 21)) ++s;
  return s;
}
// CTAs that take a segment at the same time: the least loaded ones.
__host__ __device__ inline int deal_batch(int n_cta) { return n_cta >= 4 ? n_cta / 4 : 1; }

struct DealWs {          // per tile row, and their totals behind them (nbr + 1 entries each)
  int32_t* seg_off;      // segments before the row
  int32_t* split_off;    // split rows before it
  int32_t* slot_off;     // pieces of split rows before it
};
__host__ __device__ inline void deal_segment(const PlanIn& in, const DealWs& ws, int idx, int32_t* out) {
  const int per_chunk = ws.seg_off[in.nbr], c = idx / per_chunk, j = idx - c * per_chunk;
  int lo = 0, hi = in.nbr - 1;   // the row whose segments hold j: every row has at least one
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (ws.seg_off[mid] <= j) lo = mid;
    else hi = mid - 1;
  }
  const int rs = in.row_ptr[lo], cnt = in.row_ptr[lo + 1] - rs, k = ws.seg_off[lo + 1] - ws.seg_off[lo], i = j - ws.seg_off[lo];
  const int t0 = (int)((long long)cnt * i / k), t1 = (int)((long long)cnt * (i + 1) / k);
  const bool split = k > 1;
  put_seg(out, 0, lo, c, rs + t0, rs + t1, k, split ? c * ws.slot_off[in.nbr] + ws.slot_off[lo] : 0, split ? i : 0,
          split ? c * ws.split_off[in.nbr] + ws.split_off[lo] : 0);
}
// Key of segment i of k of a row.
__host__ __device__ inline unsigned long long deal_row_key(int cnt, int k, int i, int row_cost, int piece, int idx) {
  const int tiles = (int)((long long)cnt * (i + 1) / k - (long long)cnt * i / k);
  return deal_key(tiles + (k > 1 ? piece : row_cost), idx);
}

__device__ __forceinline__ unsigned long long deal_packed(int k) {
  return (unsigned long long)k + (k > 1 ? (1ull << 20) + ((unsigned long long)k << 40) : 0ull);
}
__device__ __forceinline__ void put_offsets(const DealWs& ws, int r, unsigned long long packed) {
  ws.seg_off[r] = (int32_t)(packed & 0xfffffu);
  ws.split_off[r] = (int32_t)((packed >> 20) & 0xfffffu);
  ws.slot_off[r] = (int32_t)(packed >> 40);
}
// Sum of the values of the threads before this one, over the block; shared: 33 words, behind them the whole sum.
__device__ unsigned long long deal_scan(unsigned long long v, unsigned long long* shared) {
  const int tid = threadIdx.x, lane = tid & 31;
  unsigned long long incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  __syncthreads();
  if (lane == 31) shared[tid >> 5] = incl;
  __syncthreads();
  if (tid < 32) {
    unsigned long long w = shared[lane], t = w;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long x = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += x;
    }
    shared[lane] = t - w;
    if (lane == 31) shared[32] = t;
  }
  __syncthreads();
  return shared[tid >> 5] + incl - v;
}
__device__ long long deal_sum(long long v, unsigned long long* shared) {   // every thread has the sum
  deal_scan((unsigned long long)v, shared);
  return (long long)shared[32];
}

// The block's values in ascending order, thread k has the k-th: bitonic, within a warp by shuffles.
__device__ uint32_t deal_sort(uint32_t v, uint32_t* shared) {
  const int tid = threadIdx.x;
  for (int size = 2; size <= kDealThreads; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      uint32_t other;
      if (stride >= 32) {
        __syncthreads();
        shared[tid] = v;
        __syncthreads();
        other = shared[tid ^ stride];
      } else {
        other = __shfl_xor_sync(0xffffffffu, v, stride);
      }
      const bool smaller = ((tid & stride) == 0) == ((tid & size) == 0);
      v = smaller ? min(v, other) : max(v, other);
    }
  return v;
}

// One block: it is run once per tensor and width, and takes some 40 us for a thousand segments (the sort of the keys, then a
// batch of CTAs at a time).
__global__ void __launch_bounds__(kDealThreads) deal_kernel(PlanIn in, DealWs ws, int32_t* segs, long long capacity, int32_t* cta_seg_ptr,
                                                            int32_t* counts) {
  extern __shared__ unsigned long long keys[];                      // [kDealMaxSegs]
  __shared__ unsigned long long wide[33];
  uint16_t* taken_by = reinterpret_cast<uint16_t*>(keys + kDealMaxSegs);   // [kDealMaxSegs]
  uint16_t* place = taken_by + kDealMaxSegs;                         // [kDealMaxSegs]
  int32_t* load = reinterpret_cast<int32_t*>(place + kDealMaxSegs);   // [kDealMaxCtas]
  int32_t* held = load + kDealMaxCtas;                               // [kDealMaxCtas]
  uint32_t* order = reinterpret_cast<uint32_t*>(held + kDealMaxCtas);  // [kDealThreads]
  int32_t* tiles = reinterpret_cast<int32_t*>(order + kDealThreads);   // [kDealMaxSegs], of each row
  const int tid = threadIdx.x, G = in.n_cta, c0 = in.row_cost;
  int piece = 0;
  double share = 0.0;
  long long S = 0;
  const int per = (in.nbr + kDealThreads - 1) / kDealThreads, lo = min(tid * per, in.nbr), hi = min(lo + per, in.nbr);   // this thread's rows
  for (int r = lo; r < hi; ++r) tiles[r] = in.row_ptr[r + 1] - in.row_ptr[r];
  const long long base = ((long long)in.row_ptr[in.nbr] + (long long)c0 * in.nbr) * in.n_chunks;
  for (int attempt = 0; attempt < 2; ++attempt) {
    piece = deal_piece(c0, attempt);
    share = (double)base / G;
    for (int round = 0; round < kDealRounds; ++round) {
      long long w = 0;
      for (int r = lo; r < hi; ++r) {
        const int cnt = tiles[r];
        w += deal_cost(cnt, deal_pieces(cnt, c0, piece, share), c0, piece);
      }
      share = (double)(deal_sum(w, wide) * in.n_chunks) / G;
    }
    long long n = 0;
    for (int r = lo; r < hi; ++r) n += deal_pieces(tiles[r], c0, piece, share);
    S = deal_sum(n, wide) * in.n_chunks;
    if (S >= G) break;
  }
  unsigned long long sum = 0, before;   // segments | split rows << 20 | pieces of split rows << 40 (8192 at most each)
  for (int r = lo; r < hi; ++r) sum += deal_packed(deal_pieces(tiles[r], c0, piece, share));
  before = deal_scan(sum, wide);
  for (int r = lo; r < hi; ++r) {
    put_offsets(ws, r, before);
    before += deal_packed(deal_pieces(tiles[r], c0, piece, share));
  }
  if (tid == kDealThreads - 1) put_offsets(ws, in.nbr, before);
  __syncthreads();
  const int per_chunk = ws.seg_off[in.nbr];
  if (tid == 0) {
    counts[0] = (int32_t)S;
    counts[1] = in.n_chunks * ws.slot_off[in.nbr];
    counts[2] = in.n_chunks * ws.split_off[in.nbr];
    counts[3] = (S > capacity || S > kDealMaxSegs) ? 1 : 0;
  }
  if (S > capacity || S > kDealMaxSegs) {   // (not with the capacity asked for)
    for (int j = tid; j <= G; j += kDealThreads) cta_seg_ptr[j] = 0;
    return;
  }
  int P = 1;
  while (P < (int)S) P <<= 1;
  for (int i = tid; i < P; i += kDealThreads) keys[i] = ~0ull;
  for (int j = tid; j < G; j += kDealThreads) load[j] = held[j] = 0;
  __syncthreads();
  for (int r = lo; r < hi; ++r) {
    const int cnt = tiles[r], at = ws.seg_off[r], k = ws.seg_off[r + 1] - at;
    for (int c = 0; c < in.n_chunks; ++c)
      for (int i = 0; i < k; ++i) keys[c * per_chunk + at + i] = deal_row_key(cnt, k, i, c0, piece, c * per_chunk + at + i);
  }
  __syncthreads();
  for (int size = 2; size <= P; size <<= 1)   // bitonic sort, ascending
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = tid; t < P / 2; t += kDealThreads) {
        const int lo = 2 * t - (t & (stride - 1)), hi = lo + stride;
        const unsigned long long a = keys[lo], b = keys[hi];
        if ((a > b) == ((lo & size) == 0)) { keys[lo] = b; keys[hi] = a; }
      }
      __syncthreads();
    }
  // the CTAs take one each, then batch by batch the least loaded ones
  const int batch = deal_batch(G), shift = deal_shift((long long)(share * G));
  const int each = (int)S < G / batch * batch ? (int)S : G / batch * batch;
  for (int k = tid; k < each; k += kDealThreads) {
    taken_by[k] = (uint16_t)k;
    place[k] = 0;
    held[k] = 1;
    load[k] = deal_key_cost(keys[k]);
  }
  for (int first = each; first < (int)S; first += batch) {
    __syncthreads();
    const uint32_t cta = deal_sort(tid < G ? ((uint32_t)load[tid] >> shift) << 10 | (uint32_t)tid : ~0u, order) & 1023u;
    if (tid < batch && first + tid < (int)S) {
      const int k = first + tid;
      taken_by[k] = (uint16_t)cta;
      place[k] = (uint16_t)held[cta]++;
      load[cta] += deal_key_cost(keys[k]);
    }
  }
  __syncthreads();
  const int taken = tid < G ? held[tid] : 0, at = (int)deal_scan((unsigned long long)taken, wide);
  __syncthreads();
  if (tid < G) {
    cta_seg_ptr[tid] = at;
    load[tid] = at;
  }
  if (tid == 0) cta_seg_ptr[G] = (int32_t)S;
  __syncthreads();
  for (int k = tid; k < (int)S; k += kDealThreads)
    deal_segment(in, ws, (int)(uint32_t)keys[k], segs + ((size_t)load[taken_by[k]] + place[k]) * 8);
}
constexpr int kDealSmem = kDealMaxSegs * (8 + 2 + 2 + 4) + kDealMaxCtas * 8 + kDealThreads * 4;

static DealWs carve_deal(int32_t* base, int nbr) {
  const size_t n = (size_t)nbr + 1;
  return DealWs{base, base + n, base + 2 * n};
}
// The same on the host.
static void deal_host(const PlanIn& in, const DealWs& ws, int32_t* segs, long long capacity, int32_t* cta_seg_ptr, int32_t* counts) {
  const int G = in.n_cta, c0 = in.row_cost, nbr = in.nbr;
  int piece = 0;
  double share = 0.0;
  long long S = 0;
  auto tiles = [&](int r) { return in.row_ptr[r + 1] - in.row_ptr[r]; };
  for (int attempt = 0; attempt < 2; ++attempt) {
    piece = deal_piece(c0, attempt);
    share = (double)(((long long)in.row_ptr[nbr] + (long long)c0 * nbr) * in.n_chunks) / G;
    for (int round = 0; round < kDealRounds; ++round) {
      long long w = 0;
      for (int r = 0; r < nbr; ++r) w += deal_cost(tiles(r), deal_pieces(tiles(r), c0, piece, share), c0, piece);
      share = (double)(w * in.n_chunks) / G;
    }
    S = 0;
    for (int r = 0; r < nbr; ++r) S += deal_pieces(tiles(r), c0, piece, share);
    S *= in.n_chunks;
    if (S >= G) break;
  }
  ws.seg_off[0] = ws.split_off[0] = ws.slot_off[0] = 0;
  for (int r = 0; r < nbr; ++r) {
    const int k = deal_pieces(tiles(r), c0, piece, share);
    ws.seg_off[r + 1] = ws.seg_off[r] + k;
    ws.split_off[r + 1] = ws.split_off[r] + (k > 1 ? 1 : 0);
    ws.slot_off[r + 1] = ws.slot_off[r] + (k > 1 ? k : 0);
  }
  counts[0] = (int32_t)S;
  counts[1] = in.n_chunks * ws.slot_off[nbr];
  counts[2] = in.n_chunks * ws.split_off[nbr];
  counts[3] = (S > capacity || S > kDealMaxSegs) ? 1 : 0;
  std::vector<int32_t> load(G, 0), held(G, 0);
  for (int j = 0; j <= G; ++j) cta_seg_ptr[j] = 0;
  if (counts[3]) return;
  std::vector<unsigned long long> keys;
  for (int c = 0; c < in.n_chunks; ++c)
    for (int r = 0; r < nbr; ++r) {
      const int k = ws.seg_off[r + 1] - ws.seg_off[r];
      for (int i = 0; i < k; ++i) keys.push_back(deal_row_key(tiles(r), k, i, c0, piece, (int)keys.size()));
    }
  std::sort(keys.begin(), keys.end());
  std::vector<int32_t> taken_by((size_t)S), place((size_t)S), order(G);
  const int batch = deal_batch(G), shift = deal_shift((long long)(share * G));
  for (int first = 0; first < (int)S; first += batch) {
    for (int j = 0; j < G; ++j) order[j] = j;
    if (first >= G / batch * batch)   // (before, the CTAs take one each)
      std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return (load[a] >> shift) < (load[b] >> shift); });
    else
      std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return (load[a] != 0) < (load[b] != 0); });
    for (int rank = 0; rank < batch && first + rank < (int)S; ++rank) {
      const int j = order[rank];
      taken_by[first + rank] = j;
      place[first + rank] = held[j]++;
      load[j] += deal_key_cost(keys[first + rank]);
    }
  }
  for (int j = 0; j < G; ++j) cta_seg_ptr[j + 1] = cta_seg_ptr[j] + held[j];
  for (int k = 0; k < (int)S; ++k) deal_segment(in, ws, (int)(uint32_t)keys[k], segs + ((size_t)cta_seg_ptr[taken_by[k]] + place[k]) * 8);
}

static void host_scan(const int32_t* in, int32_t* out, int n) {
  int32_t run = 0;
  for (int i = 0; i < n; ++i) {
    const int32_t v = in[i];
    out[i] = run;
    run += v;
  }
  out[n] = run;
}

static PlanWs carve_ws(int32_t* base, int n_cta) {
  const size_t n = (size_t)n_cta + 2;
  PlanWs ws;
  ws.bv = base;
  ws.bo = base + n;
  ws.lead_nseg = base + 2 * n;
  ws.lead_flag = base + 3 * n;
  ws.slot_off = base + 4 * n;
  ws.ctr_off = base + 5 * n;
  ws.nseg_cta = base + 6 * n;
  return ws;
}

}  // namespace vb

using namespace vb;

extern "C" {

int64_t void_plan_capacity(int64_t nnz, int32_t nbr, int32_t n_chunks, int32_t n_cta, int32_t split_rows,
                           int32_t chunk_tiles) {
  if (nnz < 0 || nbr < 0 || n_chunks <= 0 || n_cta <= 0) return 0;
  int64_t per_chunk = nbr;
  if (split_rows == 2 && chunk_tiles > 0) per_chunk = nnz / chunk_tiles + nbr + 1;
  // (a row of cnt tiles makes at most cnt / (share / 2) + 1 segments, and the shares together are no less than all tiles)
  if (split_rows == 3) return per_chunk * n_chunks + 2 * (int64_t)n_cta + 2;
  return per_chunk * n_chunks + n_cta + 1;
}

size_t void_plan_ws_bytes(int32_t nbr, int32_t n_cta) {
  if (n_cta <= 0) return 0;
  const size_t shares = 7 * ((size_t)n_cta + 2), dealt = nbr > 0 ? 3 * ((size_t)nbr + 1) : 0;
  return (shares > dealt ? shares : dealt) * sizeof(int32_t);
}

static int plan_check(const int32_t* row_ptr, int32_t nbr, int32_t n_chunks, int32_t n_cta, int32_t split_rows,
                      int32_t chunk_tiles, const int32_t* woff, const int32_t* segs, const int32_t* cta_seg_ptr,
                      const int32_t* counts) {
  if (row_ptr == nullptr || segs == nullptr || cta_seg_ptr == nullptr || counts == nullptr) return VOID_ERR_BAD_ARG;
  if (nbr <= 0 || n_chunks <= 0 || n_cta <= 0 || split_rows < 0 || split_rows > 3) return VOID_ERR_BAD_ARG;
  if (split_rows > 0 && split_rows < 3 && chunk_tiles <= 0) return VOID_ERR_BAD_ARG;
  if (split_rows == 2 && woff == nullptr) return VOID_ERR_BAD_ARG;
  if ((long long)nbr * n_chunks > 0x7fffffffLL) return VOID_ERR_TOO_LARGE;
  if (split_rows == 3 && (n_cta > kDealMaxCtas || (long long)nbr * n_chunks + 2ll * n_cta + 2 > kDealMaxSegs)) return VOID_ERR_TOO_LARGE;
  return VOID_OK;
}

int void_plan_segments(const int32_t* row_ptr, int32_t nbr, int32_t n_chunks, int32_t n_cta, int32_t split_rows,
                       int32_t chunk_tiles, int32_t row_cost, const int32_t* woff, int32_t* segs,
                       int64_t segs_capacity, int32_t* cta_seg_ptr, int32_t* counts, void* ws, size_t ws_bytes,
                       void_stream_t stream) {
  const int st = plan_check(row_ptr, nbr, n_chunks, n_cta, split_rows, chunk_tiles, woff, segs, cta_seg_ptr, counts);
  if (st != VOID_OK) return st;
  if (ws == nullptr || ws_bytes < void_plan_ws_bytes(nbr, n_cta)) return VOID_ERR_WORKSPACE;
  if (row_cost < 1) return VOID_ERR_BAD_ARG;
  PlanIn in{row_ptr, woff, nbr, n_chunks, n_cta, split_rows, chunk_tiles, row_cost};
  if (split_rows == 3) {
    if (ensure_smem((const void*)deal_kernel, kDealSmem)) return VOID_ERR_CUDA;
    return status_of(launch_kernel(false, deal_kernel, 1, kDealThreads, kDealSmem, reinterpret_cast<cudaStream_t>(stream), in,
                                   carve_deal(reinterpret_cast<int32_t*>(ws), nbr), segs, segs_capacity, cta_seg_ptr, counts));
  }
  const PlanWs w = carve_ws(reinterpret_cast<int32_t*>(ws), n_cta);
  return status_of(launch_kernel(false, plan_kernel, 1, 1024, 0, reinterpret_cast<cudaStream_t>(stream), in, w, segs, segs_capacity, cta_seg_ptr, counts));
}

// Host twin of void_plan_segments over HOST arrays: the same splitting arithmetic run as plain
// loops.  It exists so that the splitter can be tested where there is no GPU; nothing in the
// SpMM path calls it.
int void_plan_segments_host(const int32_t* row_ptr, int32_t nbr, int32_t n_chunks, int32_t n_cta,
                            int32_t split_rows, int32_t chunk_tiles, int32_t row_cost, const int32_t* woff,
                            int32_t* segs, int64_t segs_capacity, int32_t* cta_seg_ptr, int32_t* counts) {
  const int st = plan_check(row_ptr, nbr, n_chunks, n_cta, split_rows, chunk_tiles, woff, segs, cta_seg_ptr, counts);
  if (st != VOID_OK) return st;
  std::vector<int32_t> buf(void_plan_ws_bytes(nbr, n_cta) / sizeof(int32_t), 0);
  if (row_cost < 1) return VOID_ERR_BAD_ARG;
  PlanIn in{row_ptr, woff, nbr, n_chunks, n_cta, split_rows, chunk_tiles, row_cost};
  if (split_rows == 3) {
    deal_host(in, carve_deal(buf.data(), nbr), segs, segs_capacity, cta_seg_ptr, counts);
    return VOID_OK;
  }
  const PlanWs w = carve_ws(buf.data(), n_cta);
  const int G = n_cta;
  for (int j = 0; j <= G; ++j) plan_boundary(in, w, j);
  for (int j = 0; j <= G; ++j) plan_leaders(in, w, j);
  host_scan(w.lead_nseg, w.slot_off, G + 1);
  host_scan(w.lead_flag, w.ctr_off, G + 1);
  host_scan(w.nseg_cta, cta_seg_ptr, G);
  for (int k = 0; k < G; ++k) plan_emit(in, w, cta_seg_ptr, segs, segs_capacity, k);
  counts[0] = cta_seg_ptr[G];
  if (split_rows == 2) {
    counts[1] = n_chunks * woff[nbr];
    counts[2] = n_chunks * nbr;
  } else {
    counts[1] = w.slot_off[G + 1];
    counts[2] = w.ctr_off[G + 1];
  }
  counts[3] = (cta_seg_ptr[G] > segs_capacity) ? 1 : 0;
  return VOID_OK;
}

}  // extern "C"
