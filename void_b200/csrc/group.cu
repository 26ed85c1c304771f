// Products of groups of tile rows that share B's panels:  C = act(dequant(A . B) + bias).
//
// The row-accumulate kernel of rowacc.cuh fetches a panel of B for every stored tile.  Its large products bring 58 - 68 bytes per
// clock into an SM, where a kernel that does nothing but load from L2 reaches 66 - 70 with every SM loading, so fewer bytes are
// what makes them faster.  Here a CTA (two per SM) owns up to eight tile rows at once, their accumulators for a panel of 128
// columns in tensor memory, and walks the block columns that ANY of its rows stores: a panel is fetched once and multiplied
// by the 1 ... R tiles of that column.  With density d a panel serves R d / (1 - (1 - d)^R) tiles: 1.4 at 90 % sparsity and
// R = 8, 2.3 at 70 % and R = 7, 3.5 at 50 %.  Measured against that kernel, us (back to back, one size after the other): fp16
// 8192^2, N = 1024 50 % 120 -> 79, 70 % 85 -> 63, 80 % 57 -> 46, 90 % 31 -> 29; 4096 x 16384, N = 2048 90 % 65 -> 56; fp32 8192^2 50 % 255
// -> 152, 70 % 157 -> 119, 80 % 108 -> 86; INT8 50 % 60 -> 42, 70 % 40 -> 33, slower from 85 % on.
//
// What is left is the chain of a CTA's stages: wait, products, commit take its warps about 550 clocks a stage whatever is in it
// (an answered wait 100, a product 44 - 60, the bookkeeping the rest), so a stage takes what a third of the CTA's shared memory holds.
// One CTA per SM with 16 rows, which would fetch a fifth less, has one such chain instead of two: bf16 16384 x 4096, 90 %, N = 2048 68
// us, 8 rows and two panels per item 80, this form 59.  One thread that waits and issues for itself takes 170 clocks for an answered
// wait and spins through those that are not: fp16 8192^2, 80 % 53 us against 46.
//
// The packed tiles are laid out in the order the CTA uses them, stage by stage (up to E block columns and T tiles), so that one bulk
// copy brings a stage's tiles and E tensor copies its panels.  A stage's tiles of consecutive rows in one block column form a run,
// which is one instruction of 32 to 128 rows (an instruction reads the 4 KB panel whatever its width: 40 clocks for 32 rows, 48 for
// 64, 64 for 128).  Groups are made of rows of falling length dealt out back and forth, so that they hold nearly the same
// number of tiles.
//
// Roles as in pipeline.cuh: two producer warps take the stages in turn, two warps issue the products of four rows each, four warps
// finish rows, one per lane quadrant of tensor memory; the products of the next item begin when four rows of this one are in
// registers.  Every wait is bounded.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cudaTypedefs.h>

#include "../../include/void_b200.h"
#include "epilogue.cuh"
#include "kinds.cuh"
#include "launch.cuh"
#include "ptx.cuh"

namespace vb {

namespace {

constexpr int kCtas = 2, kProducers = 2, kClasses = 2, kEpiWarps = 4;
constexpr int kMmaWarp0 = kProducers, kEpiWarp0 = kMmaWarp0 + kClasses;
constexpr int kClassRows = 4;                    // tile rows whose products one MMA warp issues
constexpr int kMaxRows = kClasses * kClassRows;   // tile rows of a group: their accumulators fill the CTA's tensor memory
constexpr int kMaxGroupRows = 16;                 // and the places group_rows has for them (callers size it by the header)
constexpr int kMaxEntries = 6;       // block columns per stage (what a record holds)
constexpr int kMaxStageTiles = 32;   // tiles per stage (a lane each while they are laid out)
constexpr int kRecordWords = 8;
constexpr int kHeadBytes = 16;       // of a stage, per class: its first tile, its number of runs, then a byte for each run
constexpr int kMaxRuns = kHeadBytes - 2;
static_assert(kClasses * kHeadBytes == VOID_GROUP_HEAD_BYTES, "room for the heads of as many stages as there are tiles");
constexpr int kMaxRing = 12;
constexpr int kThreads = 32 * (kProducers + kClasses + kEpiWarps);
constexpr int kNone = 0x7fffffff;

constexpr int kPartBytes = 32 * 32 * 2;   // staging of a 32 x 32 part of 16-bit results

struct GroupParams {
  const uint8_t* blob;         // tiles in the order they are used, then heads [class][tiles: as many stages as there can be]
  const int32_t* records;      // 8 per stage: first tile, tiles | entries << 8, block columns
  const int32_t* stage_ptr;    // [groups + 1]
  const int32_t* group_rows;   // [groups][16]: tile rows, -1 for none
  const int32_t* row_ptr;
  const float* row_scale;
  const float* col_scale;
  const float* bias;
  float b_scale;
  OutDesc out;
  int32_t* status;
  int nbr, n_groups, n_chunks, n_items, rows;
  int classes;                 // MMA warps with rows
  int panel_bytes;             // panels of a stage (their tiles follow)
  int stage_bytes, stages;
  int use3d, staged, out_tr, a_stable;
  int wait_limit_ms;
  unsigned long long desc_hi_a, desc_hi_b;
  unsigned int idesc;
};

struct __align__(8) Bars {
  uint64_t full[kMaxRing], empty[kMaxRing];
  uint64_t acc_full[2][kClasses], acc_empty[2][kClasses];
};

template <int KIND>
__global__ void __launch_bounds__(kThreads, kCtas) group_kernel(const __grid_constant__ CUtensorMap tmap_b,
                                                            const __grid_constant__ GroupParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ Bars bars;
  __shared__ uint32_t tmem_base_s;
  __shared__ int ctl_s[2];   // abort flag, wait limit in ms
  constexpr int ES = Elem<KIND>::ES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  volatile int* ctl = ctl_s;
  const int buf_cols = p.rows * kTile;
  const int n_buf = 2 * buf_cols <= 512 / kCtas ? 2 : 1;
  uint32_t tmem_cols = 32;
  while ((int)tmem_cols < n_buf * buf_cols) tmem_cols <<= 1;

  if (threadIdx.x == 0) {
    ctl_s[0] = 0;
    ctl_s[1] = p.wait_limit_ms;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&bars.full[s]), 1);
      mbar_init(smem_u32(&bars.empty[s]), p.classes);
    }
    for (int b = 0; b < 2; ++b)
      for (int c = 0; c < kClasses; ++c) {
        mbar_init(smem_u32(&bars.acc_full[b][c]), 1);
        mbar_init(smem_u32(&bars.acc_empty[b][c]), 4);
      }
    fence_mbar_init();
    prefetch_tmap(&tmap_b);
  }
  if (warp == kMmaWarp0) {
    tmem_alloc(smem_u32(&tmem_base_s), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;

  if (warp < kProducers) {
    bool waited = p.a_stable == 0;
    if (waited) grid_dependency_wait();
    const int S = p.stages;
    int slot = warp, first = 0;   // ring slot of this warp's next stage; CTA stages before the current item, mod kProducers
    uint32_t phase = 0;
    while (slot >= S) { slot -= S; phase ^= 1u; }
    bool ok = true;
    for (int i = blockIdx.x; i < p.n_items && ok; i += gridDim.x) {
      const int g = i / p.n_chunks, chunk = i - g * p.n_chunks;
      const int s0 = p.stage_ptr[g], s1 = p.stage_ptr[g + 1];
      int s = s0 + ((warp - first) & (kProducers - 1));
      // records of this warp's next four stages, fetched four stages ahead
      const int mine = s + (lane >> 3) * kProducers;
      int rec = 0, rec_next = mine < s1 ? p.records[(size_t)mine * kRecordWords + (lane & 7)] : 0;
      for (int k = 0; s < s1; s += kProducers, ++k) {
        const int word = (k & 3) * kRecordWords;
        if (word == 0) {
          rec = rec_next;
          const int ahead = s + ((lane >> 3) + 4) * kProducers;
          if (ahead < s1) rec_next = p.records[(size_t)ahead * kRecordWords + (lane & 7)];
        }
        const int at = __shfl_sync(0xffffffffu, rec, word);
        const int meta = __shfl_sync(0xffffffffu, rec, word + 1);
        const int tiles = meta & 0xff, entries = (meta >> 8) & 0xff;
        const int col = __shfl_sync(0xffffffffu, rec, word + 2 + (lane < kMaxEntries ? lane : 0));
        const uint32_t full = smem_u32(&bars.full[slot]), base = ring + (uint32_t)slot * (uint32_t)p.stage_bytes;
        const uint32_t blob_bytes = (uint32_t)(tiles * kTileBytes * ES);
        ok = mbar_wait_warp(smem_u32(&bars.empty[slot]), phase ^ 1u, ctl);
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(full, blob_bytes + (uint32_t)(entries * kPanelBytes * ES));
          bulk_load(base + (uint32_t)p.panel_bytes, p.blob + (size_t)at * (size_t)(kTileBytes * ES), blob_bytes, full);
        }
        __syncwarp();
        if (!waited) {   // B may be the output of the previous kernel
          grid_dependency_wait();
          waited = true;
        }
        if (lane < entries) {
          const uint32_t dst = base + (uint32_t)lane * (kPanelBytes * ES);
          if (p.use3d) tma_load_3d(dst, &tmap_b, 0, col * kTile, chunk * ES, full);
          else
            for (int q = 0; q < ES; ++q)
              tma_load_2d(dst + (uint32_t)q * kPanelBytes, &tmap_b, chunk * kPanelN + q * (kPanelN / ES), col * kTile, full);
        }
        slot += kProducers;
        while (slot >= S) { slot -= S; phase ^= 1u; }
      }
      first = (first + (s1 - s0)) & (kProducers - 1);
    }
    if (!waited) grid_dependency_wait();
  } else if (warp < kMmaWarp0 + p.classes) {
    // Each MMA warp issues the products of its own rows of the group.  It walks its chain of waits, products and commits as a warp,
    // the heads of its next stages in registers before their stages have landed.
    if (!p.a_stable) grid_dependency_wait();
    const bool leader = elect_one();
    const int cls = warp - kMmaWarp0;
    const size_t tiles = (size_t)p.row_ptr[p.nbr];
    const uint4* heads = reinterpret_cast<const uint4*>(p.blob + tiles * (size_t)(kTileBytes * ES)) + (size_t)cls * tiles;
    const uint32_t idesc = p.idesc;
    constexpr uint32_t kTileStep = (kTileBytes * ES) >> 4, kPanelStep = (kPanelBytes * ES) >> 4;
    constexpr uint32_t kPanelKStep = (kPanelBytes / ES) >> 4, kTileKStep = 256 >> 4;
    const uint32_t a_hi = (uint32_t)(p.desc_hi_a >> 32), b_hi = (uint32_t)(p.desc_hi_b >> 32);
    // the place in the ring: barriers, operand descriptors of the stage's first panel and first tile
    const uint32_t full0 = smem_u32(&bars.full[0]), empty_off = smem_u32(&bars.empty[0]) - full0, full_end = full0 + 8u * (uint32_t)p.stages;
    const uint32_t a_first = (uint32_t)p.desc_hi_a | (ring >> 4), b_first = (uint32_t)p.desc_hi_b | ((ring + (uint32_t)p.panel_bytes) >> 4);
    const uint32_t stage_step = (uint32_t)p.stage_bytes >> 4;
    uint32_t full = full0, a_at = a_first, b_at = b_first, phase = 0, it = 0;
    bool ok = true;
    int s0 = 0, s1 = 0;
    uint4 h0 = {}, h1 = {}, h2 = {};   // heads of the next three stages
    if ((int)blockIdx.x < p.n_items) {
      const int g = blockIdx.x / p.n_chunks;
      s0 = p.stage_ptr[g];
      s1 = p.stage_ptr[g + 1];
    }
    for (int i = blockIdx.x; i < p.n_items && ok; i += gridDim.x, ++it) {
      if (s0 < s1) h0 = heads[s0];
      if (s0 + 1 < s1) h1 = heads[s0 + 1];
      if (s0 + 2 < s1) h2 = heads[s0 + 2];
      int n0 = 0, n1 = 0;   // stages of the item after this one
      if (i + (int)gridDim.x < p.n_items) {
        const int g = (i + (int)gridDim.x) / p.n_chunks;
        n0 = p.stage_ptr[g];
        n1 = p.stage_ptr[g + 1];
      }
      const uint32_t buf = n_buf == 2 ? (it & 1u) : 0u, use = n_buf == 2 ? (it >> 1) : it;
      ok = mbar_wait_warp(smem_u32(&bars.acc_empty[buf][cls]), (use & 1u) ^ 1u, ctl);
      if (!ok) break;
      tc_fence_after();
      const uint32_t d0 = tmem_base + buf * (uint32_t)buf_cols + (uint32_t)(cls * kClassRows * kTile);
#pragma unroll 1
      for (int s = s0; s < s1; ++s) {
        uint4 h = h0;
        h0 = h1;
        h1 = h2;
        if (s + 3 < s1) h2 = heads[s + 3];
        const uint32_t n = (h.x >> 8) & 0xffu;
        uint32_t bt = b_at + (h.x & 0xffu) * kTileStep;
        ok = mbar_wait_warp(full, phase, ctl);
        if (!ok) break;
        uint32_t left = n, w = h.x >> 16;
#pragma unroll 1
        for (uint32_t t = 2; left > 0; ++t, --left) {
          // a run: bits 0, 1 its first row, bits 2, 3 how many following rows' tiles of the same block column go with it, bit 4 whether these
          // are its rows' first tiles, then the block column's place in the stage
          const uint32_t more = (w >> 2) & 3u, d = d0 + (w & 3u) * kTile, a = a_at + ((w >> 5) & 7u) * kPanelStep;
          const uint32_t keep = ((w >> 4) & 1u) ^ 1u, id = idesc + (more << 19);
#pragma unroll
          for (int kk = 0; kk < ES; ++kk)
            mma_halves<KIND>(leader, d, a + (uint32_t)(kk * kPanelKStep), a_hi, bt + (uint32_t)(kk * kTileKStep), b_hi, id, kk > 0 ? 1u : keep);
          bt += (more + 1u) * kTileStep;
          w >>= 8;
          if ((t & 3u) == 3u) { w = h.y; h.y = h.z; h.z = h.w; }
        }
        tc_commit_if(leader, full + empty_off);
        full += 8u;
        a_at += stage_step;
        b_at += stage_step;
        if (full == full_end) { full = full0; a_at = a_first; b_at = b_first; phase ^= 1u; }
      }
      if (!ok) break;
      tc_commit_if(leader, smem_u32(&bars.acc_full[buf][cls]));
      s0 = n0;
      s1 = n1;
    }
    __syncwarp();
  } else if (warp >= kEpiWarp0) {
    const int quad = warp & 3;
    const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
    const OutDesc od = p.out;
    const uint32_t part = ring + (uint32_t)p.stages * (uint32_t)p.stage_bytes + (uint32_t)(warp - kEpiWarp0) * kPartBytes;
    grid_dependency_wait();
    uint32_t it = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < p.n_items && ok; i += gridDim.x, ++it) {
      const int g = i / p.n_chunks, chunk = i - g * p.n_chunks;
      const uint32_t buf = n_buf == 2 ? (it & 1u) : 0u, use = n_buf == 2 ? (it >> 1) : it;
      // this lane's row of the group, with what its epilogue needs; scales and biases of the columns
      const int my_row = lane < p.rows ? p.group_rows[g * kMaxGroupRows + lane] : -1;
      int my_has = 0;
      float my_scale = 1.0f;
      if (my_row >= 0) {
        my_has = p.row_ptr[my_row + 1] > p.row_ptr[my_row] ? 1 : 0;
        if (p.row_scale != nullptr && my_has) my_scale = p.row_scale[my_row];
      }
      const int n = chunk * kPanelN + quad * 32 + lane;
      float cs = p.b_scale, bias = 0.0f;
      if (n < od.N) {
        if (p.col_scale != nullptr) cs *= p.col_scale[n];
        if (p.bias != nullptr) bias = p.bias[n];
      }
#pragma unroll 1
      for (int cls = 0; cls < p.classes; ++cls) {
        ok = mbar_wait_warp(smem_u32(&bars.acc_full[buf][cls]), use & 1u, ctl);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int r = cls * kClassRows; r < (cls + 1) * kClassRows && r < p.rows; ++r) {
          const int row = __shfl_sync(0xffffffffu, my_row, r);
          if (row < 0) continue;
          const int has = __shfl_sync(0xffffffffu, my_has, r);
          const float rs = __shfl_sync(0xffffffffu, my_scale, r);
          const uint32_t acc = tmem_base + lane_sel + buf * (uint32_t)buf_cols + (uint32_t)(r * kTile);
          if (p.staged) {
            // 16-bit results: the warp's 32 x 32 part is put together in shared memory and leaves in 16-byte pieces, four
            // lanes per row.  (A tiled store by the copy engine waits there behind the panels' loads: 2.4 us per part.)
            uint32_t lo[16], hi[16];
            if (has) {
              tmem_ld_fragments(acc, lo, hi);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int k = 0; k < 16; ++k) lo[k] = hi[k] = 0u;
            }
            finish_fragments<KIND, true>(od, row * kTile, lo, hi, rs, cs, bias, p.bias != nullptr, part, lane);
            __syncwarp();
            const int c = n - lane + (lane & 3) * 8;
            uint16_t* dst = reinterpret_cast<uint16_t*>(od.out) + (size_t)row * kTile * (size_t)od.ldc + c;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int m = k * 8 + (lane >> 2);
              uint32_t x[4];   // (the pieces of a row lie as finish_fragments puts them)
              ld_shared_v4(part + (uint32_t)(m * 64 + (((lane & 3) ^ ((m >> 1) & 3)) << 4)), x);
              if (c < od.N && row * kTile + m < od.M) *reinterpret_cast<uint4*>(dst + (size_t)m * od.ldc) = make_uint4(x[0], x[1], x[2], x[3]);
            }
            __syncwarp();
          } else {
            uint32_t v[32];
            if (has) {
              tmem_ld_32x32(acc, v);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int k = 0; k < 32; ++k) v[k] = 0u;
            }
            if (p.out_tr) {
              finish16_tr<KIND>(od, row, n, 0, &v[0], rs, cs, bias);
              finish16_tr<KIND>(od, row, n, 16, &v[16], rs, cs, bias);
            } else {
              finish16<KIND>(od, row, n, 0, &v[0], rs, cs, bias);
              finish16<KIND>(od, row, n, 16, &v[16], rs, cs, bias);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars.acc_empty[buf][cls]));
      }
    }
  }

  grid_launch_dependents();   // (late, see pipeline_teardown in pipeline.cuh)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (ctl_s[0]) {
    const uint64_t t0 = globaltimer_ns();   // let copies still in flight land before shared memory is given back
    while (globaltimer_ns() - t0 < 200000ull) {
    }
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, 1);
    __syncthreads();
  }
  if (warp == kMmaWarp0) tmem_dealloc(tmem_base, tmem_cols);
}

// ------------------------------------------------------------------------------------------ building a group store
// Rows of falling length (row_order, or their own order) dealt to the groups back and forth.
__global__ void group_rows_kernel(const int32_t* __restrict__ row_order, int nbr, int n_groups, int32_t* __restrict__ group_rows) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_groups * kMaxGroupRows) return;
  const int g = i / kMaxGroupRows, slot = i - g * kMaxGroupRows;
  const long long k = (long long)slot * n_groups + ((slot & 1) ? n_groups - 1 - g : g);
  int row = -1;
  if (k < nbr) {
    row = row_order != nullptr ? row_order[k] : (int)k;
    if (row < 0 || row >= nbr) row = -1;
  }
  group_rows[i] = row;
}

constexpr unsigned kClassStarts = 0x11u;        // first rows of the classes
static_assert(kClasses == 2 && kClassRows == 4, "kClassStarts");
constexpr uint32_t kRunStart = 1u << 8;         // (marks a run's byte while a stage is open)
__device__ __forceinline__ unsigned class_lanes(int k) { return ((1u << kClassRows) - 1u) << (k * kClassRows); }   // rows of MMA warp k
// One warp per group merges its rows' sorted column lists, lane r holding row r's place.  Pass 1 counts the group's stages;
// pass 2 writes their records and headers and where every tile goes.
template <bool EMIT>
__global__ void __launch_bounds__(128) group_walk_kernel(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ tile_cols,
                                                         const int32_t* __restrict__ group_rows, int n_groups, int max_entries,
                                                         int max_tiles,
                                                         const int32_t* __restrict__ stage_ptr,
                                                         const int32_t* __restrict__ tile_base, int32_t* __restrict__ counts,
                                                         int32_t* __restrict__ records, uint8_t* __restrict__ heads, int64_t head_stages,
                                                         int32_t* __restrict__ tile_at) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (g >= n_groups) return;
  int at = 0, end = 0, begin = 0;
  if (lane < kMaxGroupRows) {
    const int row = group_rows[g * kMaxGroupRows + lane];
    if (row >= 0) { begin = at = row_ptr[row]; end = row_ptr[row + 1]; }
  }
  int stage = EMIT ? stage_ptr[g] : 0;
  int placed = EMIT ? tile_base[g] : 0;   // tiles before the open stage
  int entries = 0, tiles = 0;
  int rec = 0;                      // lane k < 8: word k of the open stage's record
  uint32_t word = 0;                // lane k < tiles: the k-th tile of the open stage: the word of the run it starts (0 where it
  int src = 0, cls = kClasses;      // only continues one), its packed position and its class
  int in_class = 0;                 // lane k < classes: runs of class k in the open stage
  auto close = [&]() {
    if (EMIT) {
      // tiles go class by class: a tile's place is the number of tiles of lower classes and of its own before it
      int before = 0;
      for (int c = 0; c < kClasses; ++c) {
        const unsigned below = (1u << lane) - 1u, m = __ballot_sync(0xffffffffu, cls == c);
        const unsigned starts = __ballot_sync(0xffffffffu, cls == c && word != 0u);
        uint8_t* head = heads + ((size_t)c * head_stages + stage) * kHeadBytes;
        if (cls == c) {
          if (word != 0u) head[2 + __popc(starts & below)] = (uint8_t)word;
          tile_at[src] = placed + before + __popc(m & below);
        }
        if (lane == 0) {
          head[0] = (uint8_t)before;
          head[1] = (uint8_t)__popc(starts);
        }
        before += __popc(m);
      }
      if (lane == 0) rec = placed;
      if (lane == 1) rec = tiles | entries << 8;
      if (lane < kRecordWords) records[(size_t)stage * kRecordWords + lane] = rec;
      placed += tiles;
    }
    ++stage;
    entries = tiles = 0;
    rec = 0;
    cls = kClasses;
  };
  while (true) {
    const int col = at < end ? tile_cols[at] : kNone;
    const int c = __reduce_min_sync(0xffffffffu, col);
    if (c == kNone) break;
    // the rows that store it; where they are more than a stage takes, the rest come with the next one (and its panel again)
    unsigned mask = __ballot_sync(0xffffffffu, col == c);
    while (__popc(mask) > max_tiles) mask &= ~(0x80000000u >> __clz(mask));
    const int n = __popc(mask);
    const bool taken = (mask >> lane) & 1u;
    // Tiles of consecutive rows of a class make a run, unless one is its row's first and the other is not.  (A class's runs
    // have to fit its words of the header.)
    const unsigned fresh = __ballot_sync(0xffffffffu, taken && at == begin);
    const unsigned starts = mask & (~(mask << 1) | (fresh ^ (fresh << 1)) | kClassStarts);
    bool full = entries == max_entries || tiles + n > max_tiles;
    for (int k = 0; k < kClasses; ++k) {
      const int of_class = __popc(starts & class_lanes(k));
      if (__shfl_sync(0xffffffffu, in_class, k) + of_class > kMaxRuns) full = true;
    }
    if (full) {
      close();
      in_class = 0;
    }
    if (lane < kClasses) in_class += __popc(starts & class_lanes(lane));
    if (EMIT) {
      // (the byte of a run: see group_kernel)
      const unsigned after = (mask & ~starts) >> 1 >> lane;   // rows that continue a run, from the next on
      const uint32_t more = (uint32_t)(__ffs(~after) - 1);
      const uint32_t mine = (starts >> lane) & 1u ? (uint32_t)(lane & (kClassRows - 1)) | more << 2 | (at == begin ? 16u : 0u) | (uint32_t)entries << 5 | kRunStart : 0u;
      for (unsigned m = mask; m != 0u; m &= m - 1u) {
        const int from = __ffs(m) - 1;
        const uint32_t b = __shfl_sync(0xffffffffu, mine, from);
        const int place = __shfl_sync(0xffffffffu, at, from);
        if (lane == tiles) { word = b; src = place; cls = from / kClassRows; }
        ++tiles;
      }
      if (lane == 2 + entries) rec = c;
    } else {
      tiles += n;
    }
    ++entries;
    if (taken) ++at;
  }
  if (entries > 0) close();
  if (!EMIT && lane == 0) counts[g] = stage;
}

// stage_ptr and tile_base from the groups' stage and tile counts, by one block
__global__ void __launch_bounds__(1024) group_scan_kernel(const int32_t* __restrict__ counts, const int32_t* __restrict__ row_ptr,
                                                          const int32_t* __restrict__ group_rows, int n_groups,
                                                          int32_t* __restrict__ stage_ptr, int32_t* __restrict__ tile_base) {
  __shared__ int s_sum[1024], u_sum[1024];
  const int tid = threadIdx.x, per = (n_groups + 1023) / 1024;
  const int lo = tid * per < n_groups ? tid * per : n_groups, hi = lo + per < n_groups ? lo + per : n_groups;
  auto tiles_of = [&](int g) {
    int t = 0;
    for (int r = 0; r < kMaxGroupRows; ++r) {
      const int row = group_rows[g * kMaxGroupRows + r];
      if (row >= 0) t += row_ptr[row + 1] - row_ptr[row];
    }
    return t;
  };
  int s = 0, u = 0;
  for (int g = lo; g < hi; ++g) { s += counts[g]; u += tiles_of(g); }
  s_sum[tid] = s;
  u_sum[tid] = u;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const int a = tid >= o ? s_sum[tid - o] : 0, b = tid >= o ? u_sum[tid - o] : 0;
    __syncthreads();
    s_sum[tid] += a;
    u_sum[tid] += b;
    __syncthreads();
  }
  s = s_sum[tid] - s;
  u = u_sum[tid] - u;
  for (int g = lo; g < hi; ++g) {
    stage_ptr[g] = s;
    tile_base[g] = u;
    s += counts[g];
    u += tiles_of(g);
  }
  if (tid == 1023) stage_ptr[n_groups] = s_sum[1023];
}

__global__ void __launch_bounds__(256) group_copy_kernel(const uint4* __restrict__ tiles, const int32_t* __restrict__ tile_at,
                                                         int64_t nnz, int pieces, uint4* __restrict__ blob) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t t = i / pieces;
  if (t >= nnz) return;
  blob[(size_t)tile_at[t] * (size_t)pieces + (size_t)(i - t * pieces)] = tiles[i];
}

template <int KIND>
int launch_group(const GroupParams& p, const CUtensorMap& mb, int grid, int smem, cudaStream_t st) {
  auto kernel = group_kernel<KIND>;
  if (ensure_smem((const void*)kernel, smem)) return VOID_ERR_CUDA;
  return status_of(launch_pdl(kernel, grid, kThreads, smem, st, mb, p));
}

}  // namespace

}  // namespace vb

extern "C" {

int void_group_build(const int32_t* row_ptr, const int32_t* row_order, const int32_t* tile_cols, const void* tiles, int32_t nbr,
                     int64_t nnz, int32_t elem_bytes, int32_t n_groups, int32_t max_entries, int32_t max_tiles,
                     int32_t* group_rows, int32_t* stage_ptr, int32_t* records, void* blob, int32_t* ws, void_stream_t stream) {
  using namespace vb;
  if (nbr <= 0 || nnz <= 0 || n_groups <= 0 || (long long)n_groups * kMaxGroupRows < nbr) return VOID_ERR_BAD_ARG;
  if ((elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4)) return VOID_ERR_BAD_ARG;
  const int tile_bytes = kTileBytes * elem_bytes;
  if (max_entries < 1 || max_entries > kMaxEntries || max_tiles < 1 ||
      max_tiles > kMaxStageTiles || (nbr + n_groups - 1) / n_groups > kMaxRows)
    return VOID_ERR_BAD_ARG;
  if (nnz > 0x7fffffffLL / 8) return VOID_ERR_TOO_LARGE;
  if (row_ptr == nullptr || tile_cols == nullptr || tiles == nullptr || group_rows == nullptr || stage_ptr == nullptr ||
      records == nullptr || blob == nullptr || ws == nullptr)
    return VOID_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(tiles) & 15u) != 0 || (reinterpret_cast<uintptr_t>(blob) & 127u) != 0) return VOID_ERR_ALIGN;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int32_t *counts = ws, *tile_base = ws + n_groups, *tile_at = ws + 2 * (size_t)n_groups;
  uint8_t* heads = static_cast<uint8_t*>(blob) + (size_t)nnz * tile_bytes;
  const int blocks = (n_groups + 3) / 4;
  const int64_t pieces = nnz * (tile_bytes / 16);
  Launches on(st);
  on.run(group_rows_kernel, (unsigned)((n_groups * kMaxGroupRows + 255) / 256), 256, row_order, nbr, n_groups, group_rows);
  on.run(group_walk_kernel<false>, (unsigned)blocks, 128, row_ptr, tile_cols, group_rows, n_groups, max_entries, max_tiles,
         nullptr, nullptr, counts, nullptr, nullptr, nnz, nullptr);
  on.run(group_scan_kernel, 1, 1024, counts, row_ptr, group_rows, n_groups, stage_ptr, tile_base);
  on.run(group_walk_kernel<true>, (unsigned)blocks, 128, row_ptr, tile_cols, group_rows, n_groups, max_entries, max_tiles,
         stage_ptr, tile_base, counts, records, heads, nnz, tile_at);
  on.run(group_copy_kernel, (unsigned)((pieces + 255) / 256), 256, reinterpret_cast<const uint4*>(tiles), tile_at, nnz, tile_bytes / 16,
         reinterpret_cast<uint4*>(blob));
  return on.status();
}

int void_spmm_grouped(const void_spmm_args* a, const void_group_store* s, int32_t kind, void_stream_t stream) {
  using namespace vb;
  if (a == nullptr || s == nullptr || kind < VOID_KIND_I8 || kind > VOID_KIND_TF32 || kind == VOID_KIND_F8E4M3) return VOID_ERR_BAD_ARG;
  if (a->M <= 0 || a->N <= 0 || a->K <= 0 || a->nbr <= 0) return VOID_ERR_BAD_ARG;
  if (a->out == nullptr || a->b == nullptr || a->row_ptr == nullptr || s->blob == nullptr || s->records == nullptr ||
      s->stage_ptr == nullptr || s->group_rows == nullptr)
    return VOID_ERR_BAD_ARG;
  if (a->out_dtype < VOID_OUT_F32 || a->out_dtype > VOID_OUT_BF16 || a->act < VOID_ACT_NONE || a->act > VOID_ACT_SILU ||
      a->scale_mode != VOID_SCALE_ROW_MEAN || a->acc_out != nullptr || a->segs != nullptr || a->worker_partials != nullptr ||
      a->n_peers != 0 || a->trace != nullptr)
    return VOID_ERR_BAD_ARG;
  const int es = (kind == VOID_KIND_TF32) ? 4 : ((kind == VOID_KIND_F16 || kind == VOID_KIND_BF16) ? 2 : 1);
  if (a->tile_terms > 1 || (es > 1 && a->row_scale != nullptr)) return VOID_ERR_BAD_ARG;
  if (a->transposed != 0 && a->transposed != 2) return VOID_ERR_BAD_ARG;
  const bool tr = a->transposed != 0;
  if ((long long)a->nbr * kTile < a->M || a->ldc < (tr ? a->M : a->N)) return VOID_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(a->b) & 15u) != 0 || (a->ldb & 15) != 0 || a->ldb < (long long)a->N * es) return VOID_ERR_ALIGN;
  const int rows = (a->nbr + s->n_groups - 1) / (s->n_groups > 0 ? s->n_groups : 1);
  if (s->n_groups <= 0 || rows < 1 || rows > kMaxRows) return VOID_ERR_BAD_ARG;
  if (s->max_entries < 1 || s->max_entries > kMaxEntries || s->max_tiles < 1 || s->max_tiles > kMaxStageTiles) return VOID_ERR_BAD_ARG;
  const DeviceInfo dev = device_info();
  if (!dev.ok) return VOID_ERR_CUDA;
  if (dev.cc_major != 10) return VOID_ERR_ARCH;

  GroupParams p;
  p.blob = reinterpret_cast<const uint8_t*>(s->blob);
  p.records = s->records;
  p.stage_ptr = s->stage_ptr;
  p.group_rows = s->group_rows;
  p.row_ptr = a->row_ptr;
  p.row_scale = a->row_scale;
  p.col_scale = a->col_scale;
  p.bias = a->bias;
  p.b_scale = a->b_scale;
  p.out.out = a->out;
  p.out.ldc = a->ldc;
  p.out.acc_out = nullptr;
  p.out.row_bias = a->row_bias;
  p.out.M = a->M;
  p.out.N = a->N;
  p.out.dtype = a->out_dtype;
  p.out.act = a->act;
  p.status = a->status;
  p.nbr = a->nbr;
  p.n_groups = s->n_groups;
  p.n_chunks = (a->N + kPanelN - 1) / kPanelN;
  p.classes = (rows + kClassRows - 1) / kClassRows;
  if ((long long)p.n_groups * p.n_chunks > 0x7fffffffLL) return VOID_ERR_TOO_LARGE;
  p.n_items = p.n_groups * p.n_chunks;
  p.rows = rows;
  p.out_tr = tr ? 1 : 0;
  p.staged = (!tr && a->out_dtype != VOID_OUT_F32 && a->N % 8 == 0 && a->ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(a->out) & 15u) == 0) ? 1 : 0;
  p.a_stable = (a->flags & 4) ? 1 : 0;
  p.wait_limit_ms = (a->test_hooks & 0xffff) ? (a->test_hooks & 0xffff) : kDefaultWaitLimitMs;
  p.panel_bytes = s->max_entries * kPanelBytes * es;
  p.stage_bytes = (p.panel_bytes + s->max_tiles * kTileBytes * es + 1023) / 1024 * 1024;
  const int staging = p.staged ? kEpiWarps * kPartBytes : 0;
  const int room = dev.smem_per_sm / kCtas - 1024 - 1024 - 1024 - staging;   // less alignment slack and the kernel's static variables
  p.stages = room / p.stage_bytes;
  if (a->stages > 0 && a->stages < p.stages) p.stages = a->stages;
  if (p.stages > kMaxRing) p.stages = kMaxRing;
  if (p.stages < kProducers) return VOID_ERR_SHAPE;   // (a producer warp may run that many stages ahead, see pipeline.cuh)
  const int smem = p.stages * p.stage_bytes + staging + 1024;
  p.desc_hi_b = smem_desc_hi(128, 256 * es, kLayoutNone);
  p.desc_hi_a = es == 4 ? smem_desc_hi(4096, 512, kLayoutSw128Base32)
                        : (es == 2 ? smem_desc_hi(4096, 1024, kLayoutSw128) : smem_desc_hi(1024, 1024, kLayoutSw128));
  if (kind == VOID_KIND_I8) p.idesc = instr_desc(/*c s32*/ 2, /*s8*/ 1, 1, /*a MN*/ 1, /*b K*/ 0, 128, 32);
  else if (kind == VOID_KIND_F16) p.idesc = instr_desc(1, 0, 0, 1, 0, 128, 32);
  else if (kind == VOID_KIND_BF16) p.idesc = instr_desc(1, 1, 1, 1, 0, 128, 32);
  else p.idesc = instr_desc(1, 2, 2, 1, 0, 128, 32);

  CUtensorMap mb;
  memset(&mb, 0, sizeof(mb));
  bool whole = a->N % (kPanelN / es) == 0;
  if (!panel_map(&mb, a->b, a->ldb, a->K, a->N, es, 1, &whole)) return VOID_ERR_TENSOR_MAP;
  p.use3d = whole ? 1 : 0;
  int grid = a->grid > 0 ? a->grid : dev.sms * kCtas;
  if (grid > p.n_items) grid = p.n_items;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (kind) {
    case VOID_KIND_I8: return launch_group<VOID_KIND_I8>(p, mb, grid, smem, st);
    case VOID_KIND_TF32: return launch_group<VOID_KIND_TF32>(p, mb, grid, smem, st);
    default: return launch_group<VOID_KIND_F16>(p, mb, grid, smem, st);
  }
}

}  // extern "C"

