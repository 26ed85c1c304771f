// Launches of the block-sparse products (pipeline.cuh, rowacc.cuh, skinny.cu), and the per-tile kernel.
#include <mutex>

#include "pipeline.cuh"
#include "skinny.cuh"

namespace vb {

// ------------------------------------------------------------------------------------------
// Per-tile drain kernel: every tile's product is scaled by that tile's scale.
// ------------------------------------------------------------------------------------------
template <int KIND, int NP, class C, bool TRACE = false>
__global__ void __launch_bounds__(C::THREADS, (NP == 4) ? 1 : C::CTAS_PER_SM) spmm_drain_kernel(const __grid_constant__ CUtensorMap tmap_b,
                                                              const __grid_constant__ SpmmParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ PipeBars bars;
  __shared__ uint32_t tmem_base_s;
  __shared__ int ctl_s[2];   // abort flag, wait limit in ms

  // Tensor memory is cut into slot groups: one group receives the products of the tiles of one ring
  // stage (up to p.group tiles, NP panels each), so that MMA warp and epilogue hand over once per
  // stage, not once per tile.
  constexpr uint32_t kTileCols = NP * 32;   // TMEM columns of one tile's product
  const uint32_t kTmemCols = (uint32_t)p.tmem_cols;
  constexpr int CW = C::COLS;
  // Products are read back in batches of 32 registers per thread with ONE wait per batch: both halves of a
  // tile for a warp that owns all 32 accumulator columns, the halves of two tiles for a warp that owns 16.
  // A read of tensor memory is a round trip of a few hundred cycles whatever its width, and the fold that
  // follows depends on it, so the number of round trips per tile is what this role's speed hangs on.
  constexpr int TPW = 32 / CW;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t ring_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t stage_bytes = (uint32_t)(p.group * (NP * kPanelBytes + kTileBytes));
  const uint32_t group_cols = (uint32_t)p.group * kTileCols;
  const int n_slots = (int)(kTmemCols / group_cols);   // >= 2: checked at launch
  volatile int* ctl = ctl_s;

  pipeline_setup<C, 1, TRACE>(p, &tmap_b, bars, &tmem_base_s, ctl_s, n_slots, kTmemCols);
  const uint32_t tmem_base = tmem_base_s;

  if (warp < C::PW) {
    producer_loop<C, 1, 0, false, TRACE>(p, &tmap_b, &bars, ring_base, stage_bytes, ctl, lane, warp);
    if (warp == 0 && lane == 0) stamp<TRACE>(p, 2);
  } else if (warp == C::MMA) {
    {
      // as in the row-accumulate kernel: the warp walks the loop together, one elected lane issues
      const bool leader = elect_one();
      if (!p.a_stable) grid_dependency_wait();
      const uint32_t idesc = p.idesc;
      const uint64_t hi_a = p.desc_hi_a, hi_b = p.desc_hi_b;
      const int G = p.group, S = p.stages;   // (the per-tile kernel runs with stages of equal size)
      const uint32_t tiles_at = (uint32_t)(G * NP) * kPanelBytes;
      constexpr uint64_t kPanelStep = kPanelBytes >> 4, kTileStep = kTileBytes >> 4;
      int begin, end, step;
      seg_range<false>(p, begin, end, step);
      int stage = 0, slot = 0;
      uint32_t phase = 0, sphase = 0;
      uint32_t sbase = ring_base;
      bool ok = true;
      Seg seg_next = {};  // the next segment's descriptor is fetched one item ahead
      if (begin < end) seg_next = load_seg<false>(p, begin);
      for (int i = begin; i < end && ok; i += step) {
        const Seg s = seg_next;
        if (i + step < end) seg_next = load_seg<false>(p, i + step);
        const int npan = panels_in_chunk(p, s.chunk);
        for (int t = s.t0; t < s.t1; t += G) {
          const int gcnt = (s.t1 - t) < G ? (s.t1 - t) : G;
          ok = mbar_wait_warp(smem_u32(&bars.full[stage]), phase, ctl);
          if (!ok) break;
          ok = mbar_wait_warp(smem_u32(&bars.acc_empty[slot]), sphase ^ 1u, ctl);
          if (!ok) break;
          tc_fence_after();
          uint64_t ad = smem_desc(hi_a, sbase);
          uint64_t bd = smem_desc(hi_b, sbase + tiles_at);
          uint32_t d = tmem_base + (uint32_t)slot * group_cols;
          for (int j = 0; j < gcnt; ++j) {
            uint64_t adq = ad;
            uint32_t dq = d;
            for (int q = 0; q < npan; ++q) {
              issue_mma<KIND>(leader, dq, adq, bd, idesc, 0u);
              adq += kPanelStep;
              dq += 32u;
            }
            ad += kPanelStep * (uint64_t)NP;
            bd += kTileStep;
            d += kTileCols;
          }
          if (leader) {
            tc_commit(smem_u32(&bars.acc_full[slot]));
            tc_commit(smem_u32(&bars.empty[stage]));
          }
          if (++slot == n_slots) { slot = 0; sphase ^= 1u; }
          sbase += stage_bytes;
          if (++stage == S) { stage = 0; phase ^= 1u; sbase = ring_base; }
        }
      }
      if (leader) stamp<TRACE>(p, 4);
    }
    __syncwarp();
  } else {
    const int quad = warp & 3;
    const int half = (warp - C::EPI0) >> 2;
    const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
    const int m_first = half * CW;
    const int G = p.group;
    grid_dependency_wait();
    int begin, end, step;
    seg_range<false>(p, begin, end, step);
    int slot = 0;
    uint32_t sphase = 0;
    bool alive = true;
    Seg seg_next = {};  // the next segment's descriptor is fetched one item ahead
    if (begin < end) seg_next = load_seg<false>(p, begin);
    for (int i = begin; i < end && alive; i += step) {
      const Seg s = seg_next;
      if (i + step < end) seg_next = load_seg<false>(p, i + step);
      const int npan = panels_in_chunk(p, s.chunk);
      float acc[NP][CW];
#pragma unroll
      for (int q = 0; q < NP; ++q)
#pragma unroll
        for (int m = 0; m < CW; ++m) acc[q][m] = 0.0f;
      for (int t = s.t0; t < s.t1; t += G) {
        const int gcnt = (s.t1 - t) < G ? (s.t1 - t) : G;
        // scale of lane j's tile, fetched before the products are ready
        const float my_ts = (lane < gcnt) ? p.tile_scales[t + lane] : 0.0f;
        alive = mbar_wait_warp(smem_u32(&bars.acc_full[slot]), sphase, ctl);
        if (!alive) break;
        tc_fence_after();
        const uint32_t slot_addr = tmem_base + lane_sel + (uint32_t)slot * group_cols + (uint32_t)m_first;
        for (int j = 0; j < gcnt; j += TPW) {
#pragma unroll
          for (int q = 0; q < NP; ++q) {
            if (q < npan) {
              uint32_t r[TPW][CW];
#pragma unroll
              for (int u = 0; u < TPW; ++u) {
                if (j + u < gcnt) {
#pragma unroll
                  for (int c = 0; c < CW; c += 16)
                    tmem_ld_32x16p(slot_addr + (uint32_t)(j + u) * kTileCols + (uint32_t)(q * 32 + c), &r[u][c]);
                }
              }
              tmem_ld_wait();
              if (j + TPW >= gcnt && q == npan - 1) {  // this warp has read the whole slot group
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars.acc_empty[slot]));
              }
#pragma unroll
              for (int u = 0; u < TPW; ++u) {
                if (j + u < gcnt) {   // tiles are folded in their stored order, one after the other
                  const float ts = __shfl_sync(0xffffffffu, my_ts, j + u);
#pragma unroll
                  for (int m = 0; m < CW; ++m) {
                    const float x = (KIND == VOID_KIND_I8) ? __int2float_rn((int)r[u][m]) : __uint_as_float(r[u][m]);
                    acc[q][m] = fmaf(ts, x, acc[q][m]);
                  }
                }
              }
            }
          }
        }
        if (++slot == n_slots) { slot = 0; sphase ^= 1u; }
      }
      if (!alive) break;
      const OutDesc od = out_desc(p);   // read here, not before the loop: registers are what this role is short of
      const int n_base = s.chunk * NP * kPanelN + quad * 32 + lane;
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        if (q < npan) {
          const int n = n_base + q * kPanelN;
          if (n < p.N) {
            if (p.acc_out != nullptr) {
              float* a = reinterpret_cast<float*>(p.acc_out) + ((size_t)s.row * kTile + m_first) * p.N + n;
#pragma unroll
              for (int m = 0; m < CW; ++m) a[(size_t)m * p.N] = acc[q][m];
            }
            const float cs = (p.col_scale != nullptr) ? p.col_scale[n] * p.b_scale : p.b_scale;
            const float bias = (p.bias != nullptr) ? p.bias[n] : 0.0f;
#pragma unroll
            for (int c = 0; c < CW; c += 8) {
              float v[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) v[k] = acc[q][c + k] * cs + bias;
              store8(od, s.row, n, m_first + c, v);
            }
          }
        }
      }
    }
    if (threadIdx.x == 32 * C::EPI0) stamp<TRACE>(p, 6);
  }
  pipeline_teardown<C, TRACE>(p, ctl_s, tmem_base, kTmemCols);
}

// ------------------------------------------------------------------------------------------
// Host side: tensor map, launch shape, argument checks.
// ------------------------------------------------------------------------------------------
// Products the kernel for few columns (skinny.cu) takes: plain launches that ask for nothing else, with N at most 16, or
// with little enough work.  That kernel's time grows with the (tile, 32 columns) pairs, about 0.7 / 0.9 / 1.4 ns each for 8- /
// 16- / 32-bit tiles; the tensor-memory kernel's with the length of a tile row, which one CTA streams through its ring, about
// 0.13 / 0.22 / 0.42 us per tile.  The lines were swept at 16 ... 512 tile rows of 2 ... 64 tiles, N = 1 ... 128; at 4096^2,
// 90 % (13 tiles per row) fp16: N = 8 4.8 us against 9.6, N = 64 6.0 against 5.2; 2048 x 8192, 80 % (51 tiles), N = 64 7.3
// against 10.3; 16384^2, 90 % (51 tiles) INT8: N = 16 12.9 against 23.8, N = 32 21.6 against 13.9.
static bool few_columns(const void_spmm_args* a, int kind, int es, bool drain) {
  if (drain || a->N > kPanelN || a->transposed == 2 || a->segs != nullptr || a->acc_out != nullptr || a->worker_partials != nullptr ||
      a->trace != nullptr || a->n_peers != 0 || a->test_hooks != 0 || a->panels_per_item != 0 || a->stages != 0 || a->grid != 0 ||
      a->tiles_per_stage != 0 || a->cta_shape != 0 || (a->flags & ~4) != 0)
    return false;
  if (a->N <= 16) return true;
  const long long pairs = a->nnz * ((a->N + 31) / 32), rows = a->nbr > 0 ? a->nbr : 1;
  if (kind == VOID_KIND_F8E4M3 && a->tile_terms > 1) return pairs * rows < 150 * (a->nnz - 10 * rows);
  return pairs * rows < (es == 1 ? 180 : 160) * (a->nnz + rows);
}

// Three tenths of the L2's bytes make a pass: its two halves each keep what their SMs read, and A and C go through it too.  One
// pass where B is smaller.
static Passes make_passes(const DeviceInfo& dev, int rows, int n_chunks, long long K, int chunk_bytes) {
  const long long slab = (K > 0 ? K : 1) * chunk_bytes, fit = dev.l2_bytes * 3ll / 10 / slab;
  const int most = fit < 1 ? 1 : (fit < n_chunks ? (int)fit : n_chunks);
  const int passes = (n_chunks + most - 1) / most;
  Passes p;
  p.pass_chunks = (n_chunks + passes - 1) / passes;
  p.pass_items = rows * p.pass_chunks;
  p.n_full = (n_chunks - 1) / p.pass_chunks;
  p.last_chunks = n_chunks - p.n_full * p.pass_chunks;
  p.inverse = (unsigned)(((1ull << 31) + p.pass_chunks - 1) / p.pass_chunks);
  p.last_inverse = (unsigned)(((1ull << 31) + p.last_chunks - 1) / p.last_chunks);
  return p;
}

static int spmm_launch(const void_spmm_args* a, int kind, cudaStream_t stream) {
  if (a == nullptr) return VOID_ERR_BAD_ARG;
  if (a->M < 0 || a->N < 0 || a->K < 0 || a->nbr < 0 || a->nnz < 0) return VOID_ERR_BAD_ARG;
  if (a->M == 0 || a->N == 0) return VOID_OK;
  if (a->out == nullptr || a->row_ptr == nullptr) return VOID_ERR_BAD_ARG;
  if (a->nnz > 0 && (a->tiles == nullptr || a->tile_cols == nullptr || a->b == nullptr)) return VOID_ERR_BAD_ARG;
  if (a->out_dtype < VOID_OUT_F32 || a->out_dtype > VOID_OUT_BF16) return VOID_ERR_BAD_ARG;
  if (a->act < VOID_ACT_NONE || a->act > VOID_ACT_SILU) return VOID_ERR_BAD_ARG;
  if (a->scale_mode != VOID_SCALE_ROW_MEAN && a->scale_mode != VOID_SCALE_PER_TILE) return VOID_ERR_BAD_ARG;
  if (a->scale_mode == VOID_SCALE_PER_TILE && a->nnz > 0 && a->tile_scales == nullptr) return VOID_ERR_BAD_ARG;
  if (a->segs != nullptr && a->partials_bytes > 0 && a->n_peers == 0 && (a->partials == nullptr || a->counters == nullptr))
    return VOID_ERR_BAD_ARG;
  if ((long long)a->nbr * kTile < a->M) return VOID_ERR_SHAPE;
  if (a->transposed < 0 || a->transposed > 2) return VOID_ERR_BAD_ARG;
  const bool tr = a->transposed != 0, tr_b = a->transposed == 1;   // C ([N, M]), and B ([N, K]) with it
  if (a->ldc < (tr ? a->M : a->N)) return VOID_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(a->tiles) & 1023u) != 0) return VOID_ERR_ALIGN;
  if (kind < VOID_KIND_I8 || kind > VOID_KIND_TF32) return VOID_ERR_BAD_ARG;
  const int es = (kind == VOID_KIND_TF32) ? 4 : ((kind == VOID_KIND_F16 || kind == VOID_KIND_BF16) ? 2 : 1);
  const bool floating = es > 1;
  if ((reinterpret_cast<uintptr_t>(a->b) & 15u) != 0 || (a->ldb & 15) != 0 ||
      a->ldb < (long long)(tr_b ? a->K : a->N) * es)
    return VOID_ERR_ALIGN;
  // transposed operands: row-accumulate kernel without a plan or raw-accumulator outputs
  if (tr && (kind == VOID_KIND_F8E4M3 || a->scale_mode != VOID_SCALE_ROW_MEAN || a->segs != nullptr ||
             a->acc_out != nullptr || a->worker_partials != nullptr))
    return VOID_ERR_BAD_ARG;
  if (floating && (a->scale_mode != VOID_SCALE_ROW_MEAN || a->row_scale != nullptr)) return VOID_ERR_BAD_ARG;

  const DeviceInfo dev = device_info();
  if (!dev.ok) return VOID_ERR_CUDA;
  if (dev.cc_major != 10) return VOID_ERR_ARCH;

  const bool drain = (a->scale_mode == VOID_SCALE_PER_TILE);
  if (few_columns(a, kind, es, drain)) {
    SkinnyParams s;
    s.tiles = reinterpret_cast<const uint8_t*>(a->tiles);
    s.tile_cols = a->tile_cols;
    s.row_ptr = a->row_ptr;
    s.row_scale = a->row_scale;
    s.b = reinterpret_cast<const uint8_t*>(a->b);
    s.ldb = a->ldb;
    s.K = a->K; s.N = a->N; s.M = a->M;
    s.col_scale = a->col_scale;
    s.b_scale = a->b_scale;
    s.bias = a->bias;
    s.row_bias = a->row_bias;
    s.out = a->out;
    s.ldc = a->ldc;
    s.out_dtype = a->out_dtype;
    s.act = a->act;
    s.terms = a->tile_terms == 0 ? 1 : a->tile_terms;
    s.a_stable = (a->flags & 4) ? 1 : 0;
    if (s.terms < 1 || s.terms > 3 || (s.terms > 1 && kind != VOID_KIND_F8E4M3)) return VOID_ERR_BAD_ARG;
    return status_of(skinny_launch(s, kind, tr, a->nbr, a->nnz, stream));
  }
  const int total_panels = (a->N + kPanelN - 1) / kPanelN;
  int np = a->panels_per_item;
  if (np != 0 && np != 1 && np != 2 && np != 4) return VOID_ERR_BAD_ARG;
  if (floating && np > 2) return VOID_ERR_BAD_ARG;  // ring stages of wider items do not fit
  // Floating products: one panel per item, and the CTA shape that goes with the length of the tile rows (below); of 16-bit
  // tiles two panels per item where there are twenty items per SM: a tile then comes in once for both and an SM keeps more in
  // flight (9 x 18 KB in mid CTAs, 8 x 18 KB in slim ones, against 11 x 10 KB).  us, one panel in the better shape and two:
  // 16384 rows, N = 2048, 3 / 6 / 13 tiles per row 28.1 24.8, 38.9 36.3, 69.6 61.7; 8192^2, 80 %, N = 2048 117 112; C transposed,
  // 51 tiles 256 231; both transposed, N = 4096, 8192 x 3328 89.4 85.4, 8192 x 6656 156 150.  With B transposed not for rows of
  // up to 16 tiles under forty items per SM (6 tiles 30.9 32.4, 13 tiles 45.2 44.8).
  // An odd number of panels leaves half of the last item's stages unused: two per item from nine panels on, with short rows (slim
  // CTAs) from five.  us, one panel and two: one panel in all, 131072 rows, N = 128, 6 / 13 / 19 tiles 22 30, 39 55, 53 78; three, N = 384
  // 3 / 10 / 13 / 19 tiles 42 44, 75 86, 94 106, 130 148, B transposed 13 tiles 121 154; five, 3 / 10 / 19 tiles 66 61, 120 125, 209 222,
  // B transposed 10 / 19 tiles 163 159, 289 314; seven, 65536 rows 3 / 19 tiles 49.7 46.9, 153 157; nine, 16384 rows, 13 / 19 tiles 38.4
  // 37.9, 52.5 51.0.
  const long long row_panels = (long long)a->nbr * total_panels;
  const bool plain = floating && a->cta_shape == 0 && a->segs == nullptr && a->acc_out == nullptr && a->worker_partials == nullptr;
  const bool large16 = plain && es == 2 && np == 0 && row_panels >= 20ll * dev.sms &&
                       (!tr_b || row_panels >= 40ll * dev.sms || a->nnz > 16ll * a->nbr);
  const bool slim_rows = a->nnz < (tr_b ? 10ll : 5ll) * a->nbr;   // of large 16-bit products
  const bool two_panels = large16 && (total_panels % 2 == 0 || total_panels >= (slim_rows ? 5 : 9));
  if (np == 0 && floating) np = two_panels ? 2 : 1;
  if (np == 0) {
    // two panels per item keep two CTAs on an SM, which measured faster than four panels with one
    np = total_panels >= 2 ? 2 : 1;
    if (a->segs == nullptr) {  // keep enough work items to fill the machine
      while (np > 1 && (long long)a->nbr * ((total_panels + np - 1) / np) < 4ll * dev.sms) np >>= 1;
    }
  }
  const int n_chunks = (total_panels + np - 1) / np;
  // CTA shape: the slim one (four CTAs per SM) for the 8-bit row-accumulate kernel with at most two panels per item and for
  // work plans; the wide one for floating operands without a plan (two CTAs share a ring twice as deep: what a CTA takes
  // for its row is the row's tiles times the ring's round trip, and a slim ring holds two 32-bit tiles or four 16-bit
  // ones; 4096^2, 90 %, N = 512: fp32 15.7 -> 13.1 us, fp16 9.1 -> 8.8; 2048^2, 80 %, N = 256 fp32 12.1 -> 8.1), for the
  // per-tile kernel and for four-panel items (TMEM: 2 x np x 32 columns per row-accumulate CTA, 512 per SM).  Short tile
  // rows are bound by what an item costs besides its stream, which four CTAs hide better where the SM has more than two
  // items.  16-bit tiles, wide and slim, us: 8192 rows, N = 512, 6 / 13 / 20 tiles per row 8.7 7.8, 12.4 12.1, 16.0 16.4; N = 2048
  // 26.4 20.6, 39.2 37.1, 55.6 52.2; B transposed, N = 1024 6 / 9 / 13 / 20 tiles 19.0 18.4, 21.6 20.2, 25.0 24.8, 33.0 33.6; 2048 rows,
  // N = 1024 (512 items) 9 tiles 7.85 8.03.  32-bit tiles with B transposed, N = 1024, 3 / 6 / 9 / 13 tiles: 22.8 22.3, 27.4 25.5,
  // 33.0 31.9, 41.6 40.9; 2048 rows, N = 512 26 tiles 21.7 22.1.
  // Between them the mid shape, slim CTAs three to an SM with rings in between: large 16-bit products of several panels with rows
  // of 5 tiles and more (10 with B transposed; one panel per item, N = 384, wide, slim, mid: 32768 rows of 13 / 19 tiles 30.6 29.0
  // 26.4, 39.0 38.7 36.7, 131072 108 95 94, 143 135 130), and 32-bit ones from six items per SM on.  fp32, 8192 rows, wide, slim, mid: N = 512, 3 /
  // 6 / 13 tiles per row 9.6 9.1 8.4, 12.1 12.4 12.1, 20.6 21.0 20.5; N = 2048 28.9 25.3 24.5, 40.1 37.9 37.6, 73.1 70.9 65.6; 20 tiles
  // 101 to 105 in all; B transposed, N = 2048, 6 / 9 / 13 / 20 tiles 52.4 48.1 50.1, 67.6 60.4 63.2, 86.3 79.7 77.8, 116 104 104.  With 512
  // items it holds one and a half per CTA: 4096^2, 90 %, N = 512 12.1 13.0 13.9.
  int shape = a->cta_shape;
  if (shape < 0 || shape > 6) return VOID_ERR_BAD_ARG;
  if (shape == 6 && (!floating || a->segs != nullptr || a->acc_out != nullptr || a->worker_partials != nullptr)) return VOID_ERR_BAD_ARG;
  if (tr && np > 2) return VOID_ERR_BAD_ARG;
  if (tr && shape == 1 && kind == VOID_KIND_I8) return VOID_ERR_BAD_ARG;  // (8-bit transposed: the slim shape only)
  const long long n_items = (long long)a->nbr * n_chunks;
  long long short_row = 0;   // tiles per row up to which rows are short
  if (n_items > 2ll * dev.sms) {
    if (es == 2) short_row = tr_b ? (n_items > 6ll * dev.sms ? 16 : 6) : (n_items > 20ll * dev.sms ? 14 : 10);
    else if (tr_b) short_row = 10;
  }
  const bool short_rows = a->nnz <= short_row * a->nbr;
  if (large16 && total_panels > 1) shape = slim_rows ? 2 : 6;
  if (plain && np == 1 && es == 4 && n_items > 6ll * dev.sms && !(tr_b && short_rows)) shape = 6;
  if (shape == 0) shape = (!drain && np <= 2) ? ((floating && np == 1 && a->segs == nullptr && !short_rows) ? 1 : 2) : ((drain && np == 1) ? kDefaultDrainShape : 1);
  if (shape == 2 && (np > 2 || (drain && np > 1))) return VOID_ERR_BAD_ARG;
  if (shape >= 3 && shape <= 5 && (!drain || np != 1 || tr)) return VOID_ERR_BAD_ARG;  // shapes of the per-tile kernel
  const bool slim = (shape == 2 || shape == 6);   // seven warps, results of 16 bits staged
  const int producer_warps = (shape == 1) ? Wide::PW : ((shape == 4 || shape == 5) ? 1 : Slim::PW);
  const int ctas_per_sm = (shape == 2 || shape == 5) ? 4 : (shape >= 3 ? 3 : ((np == 4) ? 1 : Wide::CTAS_PER_SM));
  // CTAs that will share an SM: fewer than fit it when there are not enough work items, and each then has more of its
  // shared memory for the ring
  int share = ctas_per_sm;
  if (!drain && a->segs == nullptr && a->grid == 0) {
    const long long per_sm = ((long long)a->nbr * n_chunks + dev.sms - 1) / dev.sms;
    if (per_sm < share) share = per_sm < 1 ? 1 : (int)per_sm;
  }
  // 16-bit outputs of the slim row-accumulate kernel leave through a staging tile (32 x 128 x 2 bytes behind the
  // ring) and a tiled TMA store, when C qualifies as a tensor for the copy engine (16-byte aligned base and pitch)
  // (with a plan, whole-row segments take this route and the pieces of split rows the ordinary one; a sum over one rank, whose
  // rows are all whole or this GPU's, is a product with a plan: fp16 4096^2, 90 %, N = 512 7.6 us, 8.7 with direct stores,
  // 16384 x 4096, N = 1024 24.8 and 27.5)
  const bool one_rank = a->n_peers == 1 && a->peer_slots == 0 && a->peer_out[0] == a->out;
  const bool staged = !drain && !tr && slim && a->acc_out == nullptr && (a->n_peers == 0 || one_rank) &&
                         a->worker_partials == nullptr && (a->flags & 2) == 0 &&
                         (a->out_dtype == VOID_OUT_F16 || a->out_dtype == VOID_OUT_BF16) &&
                         (reinterpret_cast<uintptr_t>(a->out) & 15u) == 0 && ((a->ldc * 2) & 15) == 0;
  // Where every CTA has one item, the staging tile lies in the ring (ten KB at least), whose stages have all been multiplied by
  // then, and the ring has its 8 KB: ten (tile + panel) units of INT8 instead of nine, nine of FP8 tiles of two terms instead of
  // six.  4096^2, N = 512, us: FP8 80 % 10.2 (3 stages x 2) -> 9.3 (3 x 3; 4 x 2 9.6, 2 x 4 9.7), 90 % 7.0 -> 6.3, 70 % 12.7 -> 11.6; INT8 90 %
  // 5.66 (3 x 3) -> 5.54 (2 x 5; 5 x 2 5.9, 2 x 4 5.9), 70 % 9.3 -> 9.2.
  const bool single = staged && a->segs == nullptr && n_items <= (a->grid > 0 ? a->grid : dev.sms * ctas_per_sm);
  int group = a->tiles_per_stage;  // 0 = default
  // What a CTA streams is bounded by the bytes its ring keeps in flight over a stage's round trip, so the defaults fill
  // the shared memory the CTAs of an SM leave each other: nine (tile + panel) units as 3 stages x 3 for one 8-bit panel per
  // item and four CTAs (swept on B200, headline / 70 % / 16384^2: 2 x 4 units 7.02 / 11.06 / 69.9 us, 3 x 3: 6.76 / 10.21 /
  // 65.1, 4 x 2: 6.96 / 10.87 / 69.4, 9 x 1: 8.64 / 16.2 / 111); stages of one or two tiles pay the fixed cost of a stage
  // too often.  With fewer CTAs on the SM longer stages pay (1024 x 8192, 70 %, N = 256, one CTA per SM: INT8 3 x 3 12.4
  // us, 7 x 6 10.4; FP8 of two terms 17.4 -> 13.3; fp16 21.5 -> 13.4 with 6 x 3; fp32 41.2 -> 25.3 with 8 x 1).
  const bool longer = single && a->stages == 0;   // (a number of stages that is asked for is one of the ordinary length)
  if (group == 0) {
    if (floating) group = (es == 2 && np == 1) ? ((tr_b && share > 1) || slim ? 2 : 3) : 1;
    // (a tile stored as several terms is that much longer: 3 stages x 2 at four CTAs, headline 7.66 us, 2 x 3: 7.93)
    else if (a->tile_terms > 1) group = np == 1 ? (share == 1 ? 6 : (share == 2 ? 3 : (longer && a->tile_terms == 2 ? 3 : 2))) : 1;
    else group = np == 1 ? (share == 1 ? 6 : (share == 2 ? 4 : (longer ? 5 : 3))) : 2;
  }
  if (group < 1 || group > 8) return VOID_ERR_BAD_ARG;
  if (drain && np == 1 && shape != 1 && a->tiles_per_stage == 0) group = 2;
  int drain_tmem = 32;   // the largest power of two that lets ctas_per_sm CTAs share the SM's 512 columns
  while (drain_tmem * 2 * ctas_per_sm <= 512) drain_tmem *= 2;
  if (drain && group * np * 32 * 2 > drain_tmem) return VOID_ERR_BAD_ARG;  // two slot groups of products in TMEM
  int terms = a->tile_terms == 0 ? 1 : a->tile_terms;
  if (terms < 1 || terms > 3) return VOID_ERR_BAD_ARG;
  if (terms > 1 && (kind != VOID_KIND_F8E4M3 || drain || tr)) return VOID_ERR_BAD_ARG;  // FP8 row-accumulate only
  const int stage_bytes = group * (np * kPanelBytes + kTileBytes * terms) * es;
  const int staging_bytes = staged && !single ? kTile * kPanelN * 2 : 0;
  int stages = a->stages;
  if (stages == 0) {
    // dynamic shared memory a CTA may use so that its share of them fits an SM: the SM's bytes less the kilobyte
    // the system keeps per CTA and the kernel's static variables, less this kernel's 1 KB of slack for alignment
    // and the staging tile
    const int budget = dev.smem_per_sm / share - 1024 - 640 - 1024 - staging_bytes;
    stages = budget / stage_bytes;
    if (stages > 8) stages = 8;
  }
  // The shared memory the full stages leave over becomes a shorter last stage (row-accumulate kernel, ring sized
  // here) when it adds at least a fifth to the tiles in flight: 2 + 2 + 1 tiles of two 8-bit panels each take 63.8 us
  // at 16384^2 and 64.0 on an eight-rank shard of 65536^2 against 68.9 and 70.8 with 2 + 2; a seventh tile behind
  // 3 x 2 FP8 tiles of two terms costs more in stage turns than it brings (7.49 against 7.44 us, 13.54 against 13.25)
  int last_group = group;
  if (a->stages == 0 && !drain) {
    const int budget = dev.smem_per_sm / share - 1024 - 640 - 1024 - staging_bytes;
    const int left = (budget - stages * stage_bytes) / (stage_bytes / group);
    if (left >= 1 && 5 * left >= stages * group && stages < kMaxStages) {
      last_group = left < group ? left : group;
      stages += 1;
    }
  }
  // A producer warp may run up to (producer warps - 1) groups ahead of the consumer's order; the
  // parity of a ring barrier only tells two consecutive uses of a stage apart, so the ring must
  // hold at least one stage per producer warp.
  if (stages < producer_warps || stages > kMaxStages) return VOID_ERR_BAD_ARG;
  const int smem_bytes = ((stages - 1) * group + last_group) * (stage_bytes / group) + 1024 + staging_bytes;
  if (smem_bytes > dev.max_smem) return VOID_ERR_SHAPE;

  SpmmParams p;
  p.tiles = a->nnz > 0 ? reinterpret_cast<const uint8_t*>(a->tiles) : nullptr;  // null: no tensor map either
  p.tile_cols = a->tile_cols;
  p.tile_scales = a->tile_scales;
  p.row_ptr = a->row_ptr;
  p.row_order = a->segs == nullptr ? a->row_order : nullptr;
  p.row_scale = a->row_scale;
  p.nbr = a->nbr;
  p.nbc = a->nbc;
  p.nnz = a->nnz;
  p.n_chunks = n_chunks;
  p.N = a->N;
  p.M = a->M;
  p.col_scale = a->col_scale;
  p.b_scale = a->b_scale;
  p.bias = a->bias;
  p.row_bias = a->row_bias;
  p.out = a->out;
  p.ldc = a->ldc;
  p.out_dtype = a->out_dtype;
  p.act = a->act;
  p.acc_out = a->acc_out;
  p.segs = a->segs;
  p.cta_seg_ptr = a->cta_seg_ptr;
  p.partials = reinterpret_cast<int32_t*>(a->partials);
  p.counters = a->counters;
  p.worker_partials = reinterpret_cast<int32_t*>(a->worker_partials);
  p.status = a->status;
  p.n_peers = a->n_peers;
  p.peer_slots = a->peer_slots ? 1 : 0;
  if (a->n_peers < 0 || a->n_peers > 8) return VOID_ERR_BAD_ARG;
  PeerParams peers;
  if (a->peer_slots != 0 && (a->n_peers == 0 || kind != VOID_KIND_I8)) return VOID_ERR_BAD_ARG;
  if (a->n_peers > 0) {
    // reduction across GPUs: a plan whose segments name the owner of their tile row; INT8 / floating row-accumulate
    if (a->segs == nullptr || drain || tr || a->acc_out != nullptr || a->worker_partials != nullptr) return VOID_ERR_BAD_ARG;
    for (int r = 0; r < a->n_peers; ++r) {
      if (a->peer_partials[r] == nullptr) return VOID_ERR_BAD_ARG;
      if (!a->peer_slots && (a->peer_counters[r] == nullptr || a->peer_out[r] == nullptr)) return VOID_ERR_BAD_ARG;
      peers.partials[r] = reinterpret_cast<int32_t*>(a->peer_partials[r]);
      peers.counters[r] = a->peer_counters[r];
      peers.out[r] = a->peer_out[r];
    }
    if (one_rank) {
      p.partials = peers.partials[0];
      p.counters = peers.counters[0];
    }
  }
  p.trace = reinterpret_cast<unsigned long long*>(a->trace);
  p.np = np;
  p.terms = terms;
  p.group = group;
  p.stages = stages;
  p.last_group = last_group;
  p.part_off = single ? 0 : smem_bytes - 1024 - staging_bytes;
  p.use3d = (!tr_b && a->N % (kPanelN / es) == 0) ? 1 : 0;
  p.tmem_cols = drain_tmem;
  p.n_items = a->nbr * n_chunks;
  p.passes = make_passes(dev, a->nbr, n_chunks, a->K, np * kPanelN * es);
  p.a_stable = (a->flags & 4) ? 1 : 0;
  // room of the split-row scratch, in rows: the kernel refuses segments whose counter index lies beyond it
  p.ctr_limit = 0;
  if (a->segs != nullptr && ((a->partials != nullptr && a->counters != nullptr) || a->n_peers > 0) && a->partials_bytes > 0) {
    const long long per_row = (long long)np * kPanelN * kTile * (long long)sizeof(int32_t) * (a->peer_slots ? a->n_peers : 1);
    const long long rows = a->partials_bytes / per_row;
    p.ctr_limit = rows > 0x7fffffffll ? 0x7fffffff : (int)rows;
  }
  // test hooks (args->test_hooks): bits 0..15 = limit of every device-side wait in milliseconds (0: the
  // default), bit 16 = the producers never deliver the first group of tiles of each CTA
  p.wait_limit_ms = (a->test_hooks & 0xffff) ? (a->test_hooks & 0xffff) : kDefaultWaitLimitMs;
  p.drop_group = (a->test_hooks >> 16) & 1;
  if (a->trace != nullptr && !((kind == VOID_KIND_I8 && !drain && slim && !tr) ||
                               (kind == VOID_KIND_F8E4M3 && drain && np == 1 && shape >= 2)))
    return VOID_ERR_BAD_ARG;   // time stamps exist in the diagnostic instantiations only

  // Operand descriptors.  Packed tile (instruction operand B, K-major, no swizzle): 8x16-byte core
  // matrices, 128 bytes between the two k-halves (leading offset), 256 bytes between 8-row groups
  // (stride offset).  B panel (operand A, MN-major, 128-byte swizzle): one swizzle atom along n,
  // four 8-row groups along k, 1024 bytes apart.
  p.desc_hi_b = smem_desc_hi(128, 256, kLayoutNone);
  // Wider elements: the tile's row groups are 256 * es bytes apart; the panel is es swizzle atoms wide
  // along n, 4096 bytes apart (leading offset), its 8-row k groups stay 1024 bytes apart.
  // 32-bit elements in an MN-major operand need the swizzle that permutes 32-byte pieces of a 128-byte
  // row (pattern of 4 rows, so k groups of 4 rows, 512 bytes apart); the copy engine writes the same
  // pattern with its 32-byte-atom mode.
  if (floating) {
    p.desc_hi_b = smem_desc_hi(128, 256 * es, kLayoutNone);
    p.desc_hi_a = (es == 4) ? smem_desc_hi(4096, 512, kLayoutSw128Base32) : smem_desc_hi(4096, 1024, kLayoutSw128);
  } else {
    p.desc_hi_a = smem_desc_hi(1024, 1024, kLayoutSw128);
  }
  // Transposed B ([N, K], k contiguous) is a K-major operand: rows of 32 * es bytes (one swizzle span of 32,
  // 64 or 128 bytes), groups of 8 rows 256 * es bytes apart.
  const uint32_t a_mn = tr_b ? 0u : 1u;
  if (tr_b) p.desc_hi_a = smem_desc_hi(16, 256 * es, es == 4 ? kLayoutSw128 : (es == 2 ? kLayoutSw64 : kLayoutSw32));
  if (kind == VOID_KIND_I8) p.idesc = instr_desc(/*c s32*/ 2, /*a s8*/ 1, /*b s8*/ 1, a_mn, /*b K*/ 0, 128, 32);
  else if (kind == VOID_KIND_F8E4M3) p.idesc = instr_desc(/*c f32*/ 1, /*a e4m3*/ 0, /*b e4m3*/ 0, a_mn, 0, 128, 32);
  else if (kind == VOID_KIND_F16) p.idesc = instr_desc(1, /*a f16*/ 0, /*b f16*/ 0, a_mn, 0, 128, 32);
  else if (kind == VOID_KIND_BF16) p.idesc = instr_desc(1, /*a bf16*/ 1, /*b bf16*/ 1, a_mn, 0, 128, 32);
  else p.idesc = instr_desc(1, /*a tf32*/ 2, /*b tf32*/ 2, a_mn, 0, 128, 32);

  int grid;
  if (a->segs != nullptr) {
    if (a->cta_seg_ptr == nullptr || a->n_cta <= 0 || a->panels_per_item == 0) return VOID_ERR_BAD_ARG;
    if (drain || kind == VOID_KIND_F8E4M3) return VOID_ERR_BAD_ARG;  // split rows: row-accumulate kernel only
    grid = a->n_cta;
  } else {
    grid = a->grid > 0 ? a->grid : dev.sms * ctas_per_sm;
    if (grid > p.n_items) grid = p.n_items;
    if (grid < 1) grid = 1;
  }

  CUtensorMap tmap;
  memset(&tmap, 0, sizeof(tmap));
  if (a->nnz > 0) {
    bool whole = p.use3d != 0;
    const bool ok = tr_b ? panel_map_transposed(&tmap, a->b, a->ldb, a->K, a->N, es) : panel_map(&tmap, a->b, a->ldb, a->K, a->N, es, np, &whole);
    if (!ok) return VOID_ERR_TENSOR_MAP;
    p.use3d = whole ? 1 : 0;
  }

  CUtensorMap tmap_c;
  if (staged && !store_map(&tmap_c, a->out, a->ldc, a->M, a->N)) return VOID_ERR_TENSOR_MAP;

#define VB_LAUNCH(KERNEL, SHAPE)                                                               \
  do {                                                                                        \
    if (ensure_smem((const void*)KERNEL, smem_bytes)) return VOID_ERR_CUDA;                   \
    return status_of(launch_pdl(KERNEL, grid, SHAPE::THREADS, smem_bytes, stream, tmap, p));  \
  } while (0)
  const bool traced = a->trace != nullptr;
  if (!drain) {
    const bool split = a->segs != nullptr || a->acc_out != nullptr || a->worker_partials != nullptr;
    const bool active = split || traced || a->act != VOID_ACT_NONE || a->row_bias != nullptr;
    const int epilogue = (staged ? kStaged : 0) | (split ? kSplit : 0) | (active ? kActive : 0) | (traced ? kTraced : 0);
    const RowaccLaunch l = {shape, a->transposed, epilogue, grid, smem_bytes, stream, tmap, tmap_c, peers, p};
    return kind == VOID_KIND_I8       ? launch_rowacc<VOID_KIND_I8>(l)
           : kind == VOID_KIND_F8E4M3 ? launch_rowacc<VOID_KIND_F8E4M3>(l)
           : kind == VOID_KIND_TF32   ? launch_rowacc<VOID_KIND_TF32>(l)
                                      : launch_rowacc<VOID_KIND_F16>(l);   // fp16 and bf16 differ in the descriptor only
  } else if (kind == VOID_KIND_I8) {
    if (np == 1 && shape == 2) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_I8, 1, Slim>), Slim);
    else if (np == 1 && shape == 3) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_I8, 1, Slim3>), Slim3);
    else if (np == 1 && shape == 4) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_I8, 1, Drain8>), Drain8);
    else if (np == 1 && shape == 5) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_I8, 1, Slim1>), Slim1);
    else if (np == 1) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_I8, 1, Wide>), Wide);
    else if (np == 2) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_I8, 2, Wide>), Wide);
    else VB_LAUNCH((spmm_drain_kernel<VOID_KIND_I8, 4, Wide>), Wide);
  } else {
    if (np == 1 && shape == 2 && traced) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 1, Slim, true>), Slim);
    else if (np == 1 && shape == 3 && traced) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 1, Slim3, true>), Slim3);
    else if (np == 1 && shape == 4 && traced) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 1, Drain8, true>), Drain8);
    else if (np == 1 && shape == 5 && traced) return VOID_ERR_BAD_ARG;
    else if (np == 1 && shape == 2) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 1, Slim>), Slim);
    else if (np == 1 && shape == 3) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 1, Slim3>), Slim3);
    else if (np == 1 && shape == 4) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 1, Drain8>), Drain8);
    else if (np == 1 && shape == 5) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 1, Slim1>), Slim1);
    else if (np == 1) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 1, Wide>), Wide);
    else if (np == 2) VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 2, Wide>), Wide);
    else VB_LAUNCH((spmm_drain_kernel<VOID_KIND_F8E4M3, 4, Wide>), Wide);
  }
#undef VB_LAUNCH
}

// ------------------------------------------------------------------------------------------
// Built-in scratch for callers that cannot allocate device memory.
// ------------------------------------------------------------------------------------------
// int32 accumulators of split tile rows followed by their arrival counters.  The array lives in the
// library's device image: every GPU that loads the library holds these bytes until the process
// exits.
constexpr size_t kStaticPartialsBytes = 8u << 20;    // 8 MiB of int32 row accumulators
constexpr int kStaticCounters = 4096;                // arrival counters (16 KiB)
static __device__ __align__(256) unsigned char g_static_scratch[kStaticPartialsBytes + kStaticCounters * 4];

// Device address of g_static_scratch on the current device.  In host code the array's name is only
// a handle for the runtime, not an address a kernel could use; the address has to be asked for,
// once per device, with that device current.
static int static_scratch_ptr(unsigned char** out) {
  static unsigned char* ptrs[64] = {nullptr};
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return VOID_ERR_CUDA;
  std::lock_guard<std::mutex> lock(mu);
  if (ptrs[dev] == nullptr) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_static_scratch) != cudaSuccess || ptr == nullptr) return VOID_ERR_CUDA;
    ptrs[dev] = static_cast<unsigned char*>(ptr);
  }
  *out = ptrs[dev];
  return VOID_OK;
}

static int spmm_i8_static_scratch(const void_spmm_args* a, int32_t n_split_rows, cudaStream_t stream) {
  if (a == nullptr || n_split_rows < 0) return VOID_ERR_BAD_ARG;
  if (a->segs == nullptr || a->panels_per_item == 0) return VOID_ERR_BAD_ARG;  // a split-row plan is the point
  const size_t acc_bytes = (size_t)a->panels_per_item * kPanelN * kTile * sizeof(int32_t);  // one split row
  if ((size_t)n_split_rows * acc_bytes > kStaticPartialsBytes || n_split_rows > kStaticCounters) return VOID_ERR_TOO_LARGE;
  unsigned char* base = nullptr;
  const int st = static_scratch_ptr(&base);
  if (st != VOID_OK) return st;
  void_spmm_args b = *a;
  b.partials = base;
  // the room the kernel may use is what this call clears: a segment of the plan whose counter index is
  // n_split_rows or more is skipped and reported through the status word instead of touching the rest
  b.partials_bytes = (int64_t)((size_t)n_split_rows * acc_bytes);
  b.counters = reinterpret_cast<int32_t*>(base + kStaticPartialsBytes);
  // The array keeps whatever the previous call left.  Row accumulators and counters must start at
  // zero (a launch that ran to the end leaves them so, a launch that gave up may not), so the part
  // this call uses is cleared in stream order before the launch.
  if (n_split_rows > 0) {
    if (cudaMemsetAsync(b.partials, 0, (size_t)n_split_rows * acc_bytes, stream) != cudaSuccess) return VOID_ERR_CUDA;
    if (cudaMemsetAsync(b.counters, 0, (size_t)n_split_rows * sizeof(int32_t), stream) != cudaSuccess)
      return VOID_ERR_CUDA;
  }
  return spmm_launch(&b, VOID_KIND_I8, stream);
}

// A kernel that does nothing but take part in programmatic dependent launch the way the SpMM kernels do.
__global__ void floor_kernel() {
  grid_dependency_wait();
  grid_launch_dependents();
}

}  // namespace vb

extern "C" {

int void_launch_floor(int32_t grid, int32_t threads, int32_t smem_bytes, void_stream_t stream) {
  if (grid < 1 || threads < 32 || threads > 1024 || smem_bytes < 0) return VOID_ERR_BAD_ARG;
  if (vb::ensure_smem((const void*)vb::floor_kernel, smem_bytes)) return VOID_ERR_CUDA;
  return vb::status_of(vb::launch_pdl(vb::floor_kernel, grid, threads, smem_bytes, reinterpret_cast<cudaStream_t>(stream)));
}

int void_spmm_i8_static_scratch(const void_spmm_args* args, int32_t n_split_rows, void_stream_t stream) {
  return vb::spmm_i8_static_scratch(args, n_split_rows, reinterpret_cast<cudaStream_t>(stream));
}

int void_spmm_i8(const void_spmm_args* args, void_stream_t stream) {
  return vb::spmm_launch(args, VOID_KIND_I8, reinterpret_cast<cudaStream_t>(stream));
}
int void_spmm_f8(const void_spmm_args* args, void_stream_t stream) {
  return vb::spmm_launch(args, VOID_KIND_F8E4M3, reinterpret_cast<cudaStream_t>(stream));
}
int void_spmm_fp(const void_spmm_args* args, int32_t kind, void_stream_t stream) {
  if (kind != VOID_KIND_F16 && kind != VOID_KIND_BF16 && kind != VOID_KIND_TF32) return VOID_ERR_BAD_ARG;
  return vb::spmm_launch(args, kind, reinterpret_cast<cudaStream_t>(stream));
}
int void_device_sm_count(void) {
  const vb::DeviceInfo d = vb::device_info();
  return d.ok ? d.sms : 0;
}

}  // extern "C"
