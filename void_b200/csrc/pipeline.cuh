// Block-sparse SpMM for B200 (sm_100a):  C = act(dequant(A . B) + bias), A quantized to 8 bits (INT8 or
// FP8 E4M3 with per-block scales) or floating point (fp16 / bf16, or fp32 multiplied as TF32).
//
// A is the packed VOID tensor (tile-row-major 32x32 tiles, each stored as 8-row x 16-byte core
// matrices), B is a row-major [K, N] matrix of the same element size.  The product is computed
// transposed on the tensor cores so that the 32-row tile sits in the N slot of the instruction:
//
//     D[n, m] (+)= sum_k  B[kcol*32 + k, n0 + n] * A_tile[m, k]        n < 128, m < 32, k < 32
//
// i.e. tcgen05.mma (M=128, N=32, 32 bytes of k) once per (tile, 128-column panel of B) for 8-bit
// elements, twice for 16-bit, four times for 32-bit.  The "A" operand of the instruction is the B
// panel exactly as it lies in memory (n contiguous: MN-major, 128-byte swizzle, written by a tiled
// TMA load); the "B" operand is the packed tile (K-major, no swizzle, written by a linear bulk
// copy).  Accumulators live in tensor memory: lane = output column n, column = tile row m.
//
// Warp roles (struct Shape): producer warps stream tiles and panels into a shared-memory ring, one
// warp issues the MMAs and owns the tensor-memory allocation, epilogue warps read accumulators back
// (one or two warps per 32-lane TMEM quadrant), apply scales / bias / activation and store C.
//
// The ring moves GROUPS of up to `group` consecutive tiles of a tile row per stage: a group needs one
// wait + one expect_tx + one bulk copy (its tiles are contiguous in the packed store) and one tiled TMA
// per tile, the TMAs issued by different lanes in the same instruction, and the producer warps take the
// groups round-robin so that several stage turns are in flight at once.  Measured on B200, a stage's
// round trip (copies requested, landed, MMAs issued and retired, stage handed back) takes 1.2 - 1.3 us
// whatever its size, so a CTA streams what its ring holds per round trip and the launcher gives the
// ring all the shared memory that four CTAs per SM leave each other.  When N is a whole number of
// 128-byte column blocks the TMA is 3-D (B viewed as [column block][k][128 bytes]) and fetches all panels
// of the work item at once.
//
// Two kernels share this pipeline:
//   spmm_rowacc_kernel  one accumulator per (tile row, column chunk), scaled once by the
//                       row's mean tile scale (the INT8 semantic of void/int_quant.py:479-526), by
//                       the row's reference scale (FP8 tiles packed with their scales folded in: each
//                       tile is then two or three E4M3 terms that multiply the same panel), or
//                       not at all (floating point, void/ops.py:93-146); rows cut into several
//                       segments by a work plan are finished by the CTA that arrives last - the
//                       segments of a row may belong to different GPUs (sum over ranks: partial tiles
//                       go to the owning rank through peer pointers).
//   spmm_drain_kernel   every tile's product lands in its own TMEM slot and is folded into
//                       registers with that tile's scale (the exact FP8 semantic of
//                       void/fp8.py:638-659; also exact per-block INT8 dequantisation).
//
// Launch order: the kernels use programmatic dependent launch.  Set-up touches no global memory; every
// role then waits for the previous kernel of the stream where it first needs data that kernel may have
// written.  When the caller vouches that the packed A is not being written by any kernel in flight, the
// index of A and the first tiles are read ahead of that wait.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cudaTypedefs.h>

#include "../../include/void_b200.h"
#include "epilogue.cuh"
#include "kinds.cuh"
#include "launch.cuh"
#include "ptx.cuh"

namespace vb {

constexpr int kMaxStages = 16;
constexpr int kMaxSlots = 16;
// Warp roles of a CTA: PW producer warps (0..PW-1) stream tiles and panels, warp PW issues the MMAs
// and owns the TMEM allocation, EW epilogue warps follow (EW/4 per TMEM lane quadrant, each taking
// 32/(EW/4) accumulator columns).  Three shapes serve the row-accumulate kernel: a wide one (4 + 1 + 8 warps, two CTAs per
// SM), a slim one (2 + 1 + 4 warps, four CTAs per SM) and a mid one (slim, three per SM).  A CTA's stream is bound by the round trip
// of its ring: 8-bit tiles move faster through four slim CTAs per SM than through two wide ones, 16- and 32-bit tiles of small
// products through two wide CTAs, whose rings are twice as deep, those of large products through mid CTAs, or slim ones where
// rows are short.  The rule and its figures are in spmm.cu.
template <int PW_, int EW_, int CTAS_>
struct Shape {
  static constexpr int PW = PW_;
  static constexpr int EW = EW_;
  static constexpr int MMA = PW_;
  static constexpr int EPI0 = PW_ + 1;
  static constexpr int EPI_THREADS = 32 * EW_;
  static constexpr int THREADS = 32 * (PW_ + 1 + EW_);
  static constexpr int COLS = 32 / (EW_ / 4);  // accumulator columns one epilogue warp reads
  static constexpr int CTAS_PER_SM = CTAS_;
};
using Wide = Shape<4, 8, 2>;
using Slim = Shape<2, 4, 4>;
using Mid = Shape<2, 4, 3>;   // slim warps, three CTAs per SM: large products of 16- and 32-bit tiles
// Shapes of the per-tile kernel, three CTAs per SM so that an epilogue thread can hold 32 raw products in
// registers next to its running sums: four epilogue warps with all 32 accumulator columns each, or eight
// with 16 each (two tiles per round trip to tensor memory).
// (The register file is split over the four schedulers of an SM, so what a thread may use follows from the
// warps per scheduler: 28 warps -> 72 registers, 24 or 21 -> 80, 30 -> 64.)
using Slim3 = Shape<2, 4, 3>;
using Drain8 = Shape<1, 8, 3>;
using Slim1 = Shape<1, 4, 4>;
constexpr int kDefaultDrainShape = 2;   // cta_shape the one-panel per-tile kernel runs with by default

// device status codes (written to the status word)
constexpr int kStatusTimeout = 1;
constexpr int kStatusBadPlan = 2;   // a split row of the plan points outside the scratch the caller provided

// The order in which the work items (tile row, chunk of columns) of a launch without a plan are taken: pass by pass over all
// tile rows, a pass with the chunks whose part of B stays in L2 while every tile fetches its panels from it.  A is read once
// more per pass, which memory delivers beside the panels (four to nine times A's bytes).  Measured with all chunks
// together and with the passes of this rule, us (graphs of launches): INT8 65536^2, 95 %, N = 1024 (B 67 MB, two passes) 526 ->
// 481, 32768^2, N = 2048 292 -> 251, at 98 % 142 -> 126; bf16 4096 x 16384, 90 %, N = 2048 72 -> 68; fp32 8192^2, 95 %,
// N = 2048 85 -> 81.  Passes of half that size: 513, 252, 126, 69, 81.  In the first of them DRAM reads fall from 1094 to 620 MB per
// launch, L2 hits rise from 74 to 86 %.
struct Passes {
  int pass_chunks, pass_items, last_chunks, n_full;   // chunks and items of a pass, chunks of the last one, passes before it
  unsigned inverse, last_inverse;                     // 2^31 / chunks of a pass, rounded up
  __device__ __forceinline__ void item(int i, int& row, int& chunk) const {
    int first = 0, n = pass_chunks;
    unsigned inv = inverse;
    for (int pass = 0; pass < n_full && i >= pass_items; ++pass, i -= pass_items) first += pass_chunks;
    if (first == n_full * pass_chunks) { n = last_chunks; inv = last_inverse; }
    // i / n without a division, which every role of a CTA would start with; the rounding adds less than one
    row = (int)(((unsigned long long)(unsigned)i * inv) >> 31);
    chunk = i - row * n;
    if (chunk < 0) { --row; chunk += n; }
    chunk += first;
  }
};

struct SpmmParams {
  const uint8_t* tiles;
  const int32_t* tile_cols;
  const float* tile_scales;
  const int32_t* row_ptr;
  const int32_t* row_order;  // launches without a plan: tile row of the k-th row taken, or null for k
  const float* row_scale;
  int nbr, nbc, n_chunks, N, M;
  long long nnz;
  const float* col_scale;
  float b_scale;
  const float* bias;
  const float* row_bias;
  void* out;
  long long ldc;
  int out_dtype, act;
  void* acc_out;
  const int32_t* segs;
  const int32_t* cta_seg_ptr;
  int32_t* partials;
  int32_t* counters;
  int32_t* worker_partials;
  int n_peers;      // sums over ranks: PeerParams below
  int peer_slots;   // 1: every contributing rank stores its partial tile into its own slot of the owner's scratch
                    // (plain stores, no counters); a second kernel on the owner adds the slots (void_reduce_slots)
  int32_t* status;
  unsigned long long* trace;  // diagnostic instantiations only: 64 timestamps per CTA
  int np;       // panels per work item
  int terms;    // packed tiles per stored tile: 1, or 2 / 3 when an FP8 tile is stored as a sum of E4M3 terms
  int group;    // tiles per ring stage
  int stages;   // ring depth
  int last_group;   // tiles of the ring's last stage (1 .. group): the shared memory left over by the full stages
  int part_off;     // staging of 16-bit results, bytes from the ring's start: behind the ring, or in it (spmm.cu)
  int use3d;    // B panels of a tile fetched by one 3-D TMA
  int tmem_cols;  // tensor-memory columns of the drain kernel (256: two CTAs per SM, 512: one)
  int n_items;  // without a plan: nbr * n_chunks
  Passes passes;  // and the order they are taken in
  int a_stable;   // A's packed arrays and the plan were complete before the stream's kernels in flight started:
                  // they may be read before the wait on the previous kernel
  int ctr_limit;  // split rows the scratch (partials, counters) has room for
  int wait_limit_ms;  // limit of every device-side wait
  int drop_group;     // test hook: the producers never fill the ring stage of each CTA's first group of tiles
  unsigned long long desc_hi_a;  // B panel  (instruction operand A: MN-major, 128B swizzle)
  unsigned long long desc_hi_b;  // A tile   (instruction operand B: K-major, no swizzle)
  unsigned int idesc;
};

// Split rows whose sums live on other GPUs (reduction across ranks): n_peers > 0 makes field slot0 of a segment the owner of its
// tile row; the row's accumulator, arrival counter and rows of C are the owner's, reached through peer pointers (out is
// offset so that the GLOBAL tile row indexes it).
struct PeerParams {
  int32_t* partials[8];
  int32_t* counters[8];
  void* out[8];
};

// Time stamps exist in the diagnostic instantiations (TRACE) only; the kernels every ordinary launch runs
// are compiled without them.
template <bool TRACE>
__device__ __forceinline__ void stamp(const SpmmParams& p, int slot) {
  if constexpr (TRACE) {
    if (p.trace != nullptr) p.trace[(size_t)blockIdx.x * 64 + slot] = globaltimer_ns();
  }
}

struct Seg {
  int row, chunk, t0, t1, nseg, slot0, my_idx, ctr;
};

// PLAN: the launch may come with a work plan.
template <bool PLAN>
__device__ __forceinline__ Seg load_seg(const SpmmParams& p, int i) {
  Seg s;
  if (PLAN && p.segs != nullptr) {
    const int4* q = reinterpret_cast<const int4*>(p.segs) + 2 * (size_t)i;
    const int4 a = q[0], b = q[1];
    s.row = a.x; s.chunk = a.y; s.t0 = a.z; s.t1 = a.w;
    s.nseg = b.x; s.slot0 = b.y; s.my_idx = b.z; s.ctr = b.w;
  } else {
    int k;   // k-th tile row taken
    p.passes.item(i, k, s.chunk);
    s.row = k;
    if (p.row_order != nullptr) {
      const int r = p.row_order[k];
      s.row = r < 0 ? 0 : (r >= p.nbr ? p.nbr - 1 : r);
    }
    s.t0 = p.row_ptr[s.row];
    s.t1 = p.row_ptr[s.row + 1];
    s.nseg = 1; s.slot0 = 0; s.my_idx = 0; s.ctr = 0;
  }
  return s;
}

// The same for a warp that waits with many values in registers: lane k holds word k (in the order of Seg's fields).
template <bool PLAN>
__device__ __forceinline__ int load_seg_word(const SpmmParams& p, int i, int lane) {
  if (PLAN && p.segs != nullptr) return p.segs[8 * (size_t)i + (lane & 7)];   // (without a branch, whose register costs 0.1 us of 14.9)
  int k, chunk;
  p.passes.item(i, k, chunk);
  int row = k;
  if (p.row_order != nullptr) {
    const int r = p.row_order[k];
    row = r < 0 ? 0 : (r >= p.nbr ? p.nbr - 1 : r);
  }
  if (lane == 2 || lane == 3) return p.row_ptr[row + lane - 2];
  return lane == 0 ? row : (lane == 1 ? chunk : (lane == 4 ? 1 : 0));
}
__device__ __forceinline__ int word_of(int words, int k) { return __shfl_sync(0xffffffffu, words, k); }

// Range of segment indices of this CTA: [begin, end) with stride step.
template <bool PLAN>
__device__ __forceinline__ void seg_range(const SpmmParams& p, int& begin, int& end, int& step) {
  if (PLAN && p.segs != nullptr) {
    begin = p.cta_seg_ptr[blockIdx.x];
    end = p.cta_seg_ptr[blockIdx.x + 1];
    step = 1;
  } else {
    begin = blockIdx.x;
    end = p.n_items;
    step = gridDim.x;
  }
}

__device__ __forceinline__ int panels_in_chunk(const SpmmParams& p, int chunk) {
  const int total = (p.N + kPanelN - 1) / kPanelN;
  const int left = total - chunk * p.np;
  return left < p.np ? left : p.np;
}

__device__ __forceinline__ OutDesc out_desc(const SpmmParams& p) {
  OutDesc o;
  o.out = p.out; o.ldc = p.ldc; o.acc_out = p.acc_out; o.row_bias = p.row_bias; o.M = p.M; o.N = p.N; o.dtype = p.out_dtype; o.act = p.act;
  return o;
}

struct __align__(8) PipeBars {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t acc_full[kMaxSlots];
  uint64_t acc_empty[kMaxSlots];
};

// shared-memory offsets inside one ring stage
template <int ES>
__device__ __forceinline__ uint32_t panel_off(const SpmmParams& p, int j, int q) {
  return (uint32_t)(j * p.np + q) * (kPanelBytes * ES);
}
// A stage holds the panels of its tiles first, then the tiles; `cap` is the stage's capacity in tiles
template <int ES>
__device__ __forceinline__ uint32_t tile_off(const SpmmParams& p, int cap, int j) {
  return (uint32_t)(cap * p.np) * (kPanelBytes * ES) + (uint32_t)(j * p.terms) * (kTileBytes * ES);
}
// Capacity of a ring stage: every stage takes p.group tiles except the last, which takes what is left of the
// shared memory (p.last_group).  The groups of a tile row follow the stages they fall on: a group is
// min(capacity of its stage, tiles left in the row) consecutive tiles.
__device__ __forceinline__ int stage_cap(const SpmmParams& p, int stage) {
  return stage == p.stages - 1 ? p.last_group : p.group;
}

// Producer warp `pw` of C::PW: the CTA's groups of tiles are numbered in the order the MMA warp
// consumes them; group g uses ring stage g % stages and belongs to warp g % C::PW.
//
// The wait on the previous kernel of the stream sits where the first read of data that kernel may
// have produced is.  When the caller vouches for A (p.a_stable: the packed tiles, their index arrays
// and the plan were complete before the kernels now in flight started) the warp reads the index,
// claims its first ring stage and starts the bulk copy of that stage's tiles BEFORE the wait, while the
// previous kernel is still draining; only the panels of B - typically that kernel's output - are
// requested after it.
template <class C, int ES, int TR, bool PLAN, bool TRACE>
__device__ __forceinline__ void producer_loop(const SpmmParams& p, const CUtensorMap* tmap, PipeBars* bars,
                                              uint32_t ring_base, uint32_t stage_bytes, volatile int* ctl,
                                              int lane, int pw) {
  bool waited = p.a_stable == 0;
  if (waited) grid_dependency_wait();
  if (TRACE && pw == 0 && lane == 0) stamp<TRACE>(p, 56);   // producer starts
  int begin, end, step;
  seg_range<PLAN>(p, begin, end, step);
  const int S = p.stages;
  // position of the next group in the ring: its stage, the parity of the stage's use, the warp it belongs to
  int stage = 0, owner = 0, gcount = 0;
  uint32_t phase = 0;
  Seg seg_next = {};  // the next segment's descriptor is fetched one item ahead
  if (begin < end) seg_next = load_seg<PLAN>(p, begin);
  for (int i = begin; i < end; i += step) {
    const Seg s = seg_next;
    if (i + step < end) seg_next = load_seg<PLAN>(p, i + step);
    const int npan = panels_in_chunk(p, s.chunk);
    const int n0 = s.chunk * p.np * kPanelN;
    const uint32_t unit_bytes = (uint32_t)((kTileBytes * p.terms + ((p.use3d && TR != 1) ? p.np : npan) * kPanelBytes) * ES);
    if (TRACE && i == begin && pw == 0 && lane == 0) {
      asm volatile("" ::"r"(s.t1) : "memory");
      stamp<TRACE>(p, 57);   // the row's tile range has arrived
    }
    // block column of this lane's tile in the warp's next group, fetched one group of its own ahead; (ct, cs):
    // first tile and stage of that group
    int ct = s.t0, cs = stage;
    for (int o = owner; o != pw && ct < s.t1; o = (o + 1 == C::PW) ? 0 : o + 1) {
      ct += stage_cap(p, cs);
      cs = (cs + 1 == S) ? 0 : cs + 1;
    }
    int col = 0;
    if (ct + lane < s.t1 && lane < stage_cap(p, cs)) col = p.tile_cols[ct + lane];
    if (TRACE && i == begin && pw == 0 && lane == 0) {
      asm volatile("" ::"r"(col) : "memory");
      stamp<TRACE>(p, 58);   // the first block columns have arrived
    }
    int k = 0;   // group of the segment
    for (int t = s.t0; t < s.t1; ++k, ++gcount) {
      const int cap = stage_cap(p, stage);
      const int gcnt = (s.t1 - t) < cap ? (s.t1 - t) : cap;
      if (owner == pw) {
        // this warp's group after this one
        int nt = t, ns = stage;
        for (int o = 0; o < C::PW && nt < s.t1; ++o) {
          nt += stage_cap(p, ns);
          ns = (ns + 1 == S) ? 0 : ns + 1;
        }
        int col_next = 0;
        if (nt + lane < s.t1 && lane < stage_cap(p, ns)) col_next = p.tile_cols[nt + lane];
        const uint32_t full = smem_u32(&bars->full[stage]);
        const uint32_t sbase = ring_base + (uint32_t)stage * stage_bytes;
        // test hook: the first group of the CTA is never delivered, so the consumer's bounded wait runs out
        const bool drop = p.drop_group != 0 && gcount == 0;
        if (!mbar_wait_warp(smem_u32(&bars->empty[stage]), phase ^ 1u, ctl)) return;
        if (lane == 0 && !drop) {
          mbar_expect_tx(full, unit_bytes * (uint32_t)gcnt);
          bulk_load(sbase + tile_off<ES>(p, cap, 0), p.tiles + (size_t)t * (size_t)(kTileBytes * ES * p.terms),
                    (uint32_t)(gcnt * p.terms) * (kTileBytes * ES), full);
        }
        __syncwarp();
        if (TRACE && i == begin && pw == 0 && lane == 0 && k == 0) stamp<TRACE>(p, 59);   // tiles of the first group requested
        if (!waited) {  // B may be the output of the previous kernel
          grid_dependency_wait();
          waited = true;
        }
        if (TRACE && i == begin && pw == 0 && lane == 0 && k == 0) stamp<TRACE>(p, 60);   // past the wait on the previous kernel
        if (lane < gcnt && !drop) {
          if (TR == 1) {
            // B stored transposed ([N, K], k contiguous): one box of 128 rows of n x 32 k per panel
            for (int q = 0; q < npan; ++q)
              tma_load_2d(sbase + panel_off<ES>(p, lane, q), tmap, col * kTile, n0 + q * kPanelN, full);
          } else if (p.use3d) {
            tma_load_3d(sbase + panel_off<ES>(p, lane, 0), tmap, 0, col * kTile, s.chunk * p.np * ES, full);
          } else {
            // one copy per 128-byte-wide block of columns: ES blocks of 128 / ES columns per panel
            for (int q = 0; q < npan * ES; ++q)
              tma_load_2d(sbase + panel_off<ES>(p, lane, 0) + (uint32_t)q * kPanelBytes, tmap,
                          n0 + q * (kPanelN / ES), col * kTile, full);
          }
        }
        if (TRACE && lane == 0 && i == begin && k < 16) stamp<TRACE>(p, 32 + k);
        col = col_next;
      }
      t += gcnt;
      owner = (owner + 1 == C::PW) ? 0 : owner + 1;
      if (++stage == S) { stage = 0; phase ^= 1u; }
    }
  }
  if (!waited) grid_dependency_wait();
}

// Barriers, tensor memory and the launch of the next kernel's set-up.  Nothing here touches global memory,
// so all of it overlaps the tail of the previous kernel of the stream (programmatic dependent launch);
// every role then waits for that kernel where it first needs data the kernel may have written.
template <class C, int ES, bool TRACE>
__device__ __forceinline__ void pipeline_setup(const SpmmParams& p, const CUtensorMap* tmap, PipeBars& bars,
                                               uint32_t* tmem_base_s, int* ctl_s, int n_acc, uint32_t tmem_cols) {
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) stamp<TRACE>(p, 62);
  if constexpr (TRACE) {   // slot 63: the SM this CTA runs on
    if (threadIdx.x == 0 && p.trace != nullptr) {
      uint32_t smid;
      asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
      p.trace[(size_t)blockIdx.x * 64 + 63] = smid;
    }
  }
  if (threadIdx.x == 0) {
    ctl_s[0] = 0;
    ctl_s[1] = p.wait_limit_ms;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&bars.full[s]), 1);
      mbar_init(smem_u32(&bars.empty[s]), 1);
    }
    for (int b = 0; b < n_acc; ++b) {
      mbar_init(smem_u32(&bars.acc_full[b]), 1);
      mbar_init(smem_u32(&bars.acc_empty[b]), C::EW);
    }
    fence_mbar_init();
    if (p.tiles != nullptr) prefetch_tmap(tmap);
  }
  if (warp == C::MMA) {
    tmem_alloc(smem_u32(tmem_base_s), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x == 0) stamp<TRACE>(p, 1);
}

template <class C, bool TRACE>
__device__ __forceinline__ void pipeline_teardown(const SpmmParams& p, int* ctl_s, uint32_t tmem_base,
                                                  uint32_t tmem_cols) {
  // The next kernel may start when every CTA is through with its work: started with this one, it settles beside CTAs that
  // have yet to come, on few SMs, and keeps that placement (graphs of launches, 4096^2, N = 512: fp32 90 % 13.1 -> 12.8 us,
  // its transposed form 14.1 -> 13.1; INT8 16384^2, 95 % 21.7 -> 20.6; not at all early: 15.5 and 23.5).
  grid_launch_dependents();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x == 0) stamp<TRACE>(p, 7);
  if (ctl_s[0]) {
    // let copies that may still be in flight land before shared memory is given back
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, kStatusTimeout);
    __syncthreads();
  }
  if ((threadIdx.x >> 5) == C::MMA) tmem_dealloc(tmem_base, tmem_cols);
}

// How a row-accumulate kernel is launched; defined in rowacc.cuh, built for one kind per source file.  `epilogue`: what its
// epilogue has to be able to do, a sum of
//   kStaged  16-bit results through shared memory and tiled stores
//   kSplit   a work plan, raw sums for the caller
//   kActive  activation, row bias
//   kTraced  time stamps (slim INT8 only, with kActive)
constexpr int kStaged = 1, kSplit = 2, kActive = 4, kTraced = 8;
struct RowaccLaunch {
  int shape;   // 1 wide, 2 slim, 6 mid
  int transposed;
  int epilogue;
  int grid, smem_bytes;
  cudaStream_t stream;
  const CUtensorMap& b;
  const CUtensorMap& c;
  const PeerParams& peers;
  const SpmmParams& p;
};
template <int KIND>
int launch_rowacc(const RowaccLaunch& l);

}  // namespace vb
