// The row-accumulate kernel (pipeline.cuh): one accumulator per (tile row, column chunk).
#pragma once
#include <type_traits>

#include "pipeline.cuh"

namespace vb {

// All COLS accumulator columns of one epilogue warp, requested together (no wait).
template <int COLS>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[COLS]) {
#pragma unroll
  for (int c = 0; c < COLS; c += 16) tmem_ld_32x16p(taddr + (uint32_t)c, &r[c]);
}

// The accumulator of a split row's panel q, [32 m][128 n]; with peers the owner's.
template <typename X>
__device__ __forceinline__ int32_t* row_sums(const SpmmParams& p, const X& x, int seg_words, bool peers, int q) {
  int32_t* base = p.partials;
  if constexpr (std::is_same<X, PeerParams>::value)
    if (peers) base = x.partials[word_of(seg_words, 5)];
  return base + ((size_t)word_of(seg_words, 7) * p.np + q) * (kTile * kPanelN);
}

// What a kernel is given besides B and the common parameters: C as a tensor, the peers of a sum over ranks, or nothing.  (A
// launch takes longer by about a nanosecond for every four bytes of parameters.)
struct Nothing {};
template <int EPI>
using ExtraOf = std::conditional_t<(EPI & kStaged) != 0, CUtensorMap, std::conditional_t<(EPI & kSplit) != 0, PeerParams, Nothing>>;

// TR: 1 = B and C transposed ([N, K] and [N, M]), 2 = C alone.  EPI: what the epilogue is asked for (kStaged ...).  What is not run
// costs a little too, in spilled registers and in instructions fetched around it: INT8 4096^2, 90 %, N = 512, fp16 results 6.10 us,
// through the kernel that also splits rows and activates 6.20; with GELU 6.57, through that kernel 6.60.
template <int KIND, class C, int TR, int EPI>
__global__ void __launch_bounds__(C::THREADS, C::CTAS_PER_SM) spmm_rowacc_kernel(const __grid_constant__ CUtensorMap tmap_b,
                                                                                 const __grid_constant__ ExtraOf<EPI> x,
                                                                                 const __grid_constant__ SpmmParams p) {
  constexpr bool STAGED = (EPI & kStaged) != 0, SPLIT = (EPI & kSplit) != 0, ACT = (EPI & kActive) != 0, TRACE = (EPI & kTraced) != 0;
  static_assert(!TR || (!STAGED && !SPLIT), "transposed results are stored directly, of whole rows");
  static_assert(!STAGED || C::COLS == kTile, "an epilogue warp stages whole columns of a tile row");
  extern __shared__ uint8_t smem_raw[];
  __shared__ PipeBars bars;
  __shared__ uint32_t tmem_base_s;
  __shared__ int ctl_s[2];   // abort flag, wait limit in ms
  __shared__ int last_s;
  __shared__ int ok_s[2];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t ring_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  constexpr int ES = Elem<KIND>::ES;
  const uint32_t unit_smem = (uint32_t)((p.np * kPanelBytes + kTileBytes * p.terms) * ES);
  const uint32_t stage_bytes = (uint32_t)p.group * unit_smem;   // the last stage may be shorter (p.last_group tiles)
  const uint32_t acc_cols = (uint32_t)p.np * 32u;  // TMEM columns of one accumulator buffer
  uint32_t tmem_cols = 32;
  while (tmem_cols < 2u * acc_cols) tmem_cols <<= 1;
  volatile int* ctl = ctl_s;

  if (threadIdx.x == 0) last_s = 0;
  pipeline_setup<C, ES, TRACE>(p, &tmap_b, bars, &tmem_base_s, ctl_s, 2, tmem_cols);
  const uint32_t tmem_base = tmem_base_s;

  if (warp < C::PW) {
    producer_loop<C, ES, TR, SPLIT, TRACE>(p, &tmap_b, &bars, ring_base, stage_bytes, ctl, lane, warp);
    if (warp == 0 && lane == 0) stamp<TRACE>(p, 2);
  } else if (warp == C::MMA) {
    {
      // The whole warp walks the loop and waits on the barriers together; one elected lane issues the MMAs and
      // the commits.  The control flow stays convergent, so the addresses, descriptors and counters are the
      // same in every lane and the compiler may keep them in the warp's uniform registers, where the
      // instruction operands have to be: a loop run by a single lane computes them per thread and moves them
      // over before every MMA.
      // The warp reads the index of A and the plan only; everything else reaches it through the ring.
      const bool leader = elect_one();
      if (!p.a_stable) grid_dependency_wait();
      const uint32_t idesc = p.idesc;
      const uint64_t hi_a = p.desc_hi_a, hi_b = p.desc_hi_b;
      const int S = p.stages, np = p.np, terms = p.terms;
      constexpr uint64_t kPanelStep = (kPanelBytes * ES) >> 4, kTileStep = (kTileBytes * ES) >> 4;
      // one MMA covers 32 bytes of k: 32 / ES k-rows of the panel (8-row groups 1024 bytes apart) and two
      // 16-byte k-chunks of the packed tile (128 bytes apart)
      // (transposed B: the panel is K-major, 32 bytes of k lie inside one row of its swizzle atom)
      constexpr uint64_t kPanelKStep = TR == 1 ? 2 : ((kPanelBytes / ES) >> 4), kTileKStep = 256 >> 4;
      int begin, end, step;
      seg_range<SPLIT>(p, begin, end, step);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t sbase = ring_base;
      uint32_t it = 0;
      bool ok = true;
      Seg seg_next = {};  // the next segment's descriptor is fetched one item ahead
      if (begin < end) seg_next = load_seg<SPLIT>(p, begin);
      for (int i = begin; i < end && ok; i += step, ++it) {
        const Seg s = seg_next;
        if (i + step < end) seg_next = load_seg<SPLIT>(p, i + step);
        const int npan = panels_in_chunk(p, s.chunk);
        const uint32_t buf = it & 1u, aph = (it >> 1) & 1u;
        ok = mbar_wait_warp(smem_u32(&bars.acc_empty[buf]), aph ^ 1u, ctl);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d0 = tmem_base + buf * acc_cols;
        uint32_t acc = 0u;
        int gidx = 0;
        for (int t = s.t0; t < s.t1; ++gidx) {
          const int cap = stage_cap(p, stage);
          const int gcnt = (s.t1 - t) < cap ? (s.t1 - t) : cap;
          t += gcnt;
          if (TRACE && leader && i == begin && gidx < 8) stamp<TRACE>(p, 48 + gidx);
          ok = mbar_wait_warp(smem_u32(&bars.full[stage]), phase, ctl);
          if (!ok) break;
          if (TRACE && leader && i == begin && gidx < 12) stamp<TRACE>(p, 16 + gidx);   // slots 28 .. 31: last arriver of a split row
          tc_fence_after();
          uint64_t ad = smem_desc(hi_a, sbase);
          uint64_t bd = smem_desc(hi_b, sbase + tile_off<ES>(p, cap, 0));
          for (int j = 0; j < gcnt; ++j) {
            auto panel = [&](uint64_t a, uint32_t d) {
#pragma unroll
              for (int kk = 0; kk < ES; ++kk) issue_mma<KIND>(leader, d, a + kk * kPanelKStep, bd + kk * kTileKStep, idesc, kk == 0 ? acc : 1u);
              // a tile stored as a sum of terms: every further term multiplies the same panel
              if (KIND == VOID_KIND_F8E4M3) {
                if (terms > 1) issue_mma<KIND>(leader, d, a, bd + kTileStep, idesc, 1u);
                if (terms > 2) issue_mma<KIND>(leader, d, a, bd + 2 * kTileStep, idesc, 1u);
              }
            };
            panel(ad, d0);
            if (npan > 1) panel(ad + kPanelStep, d0 + 32u);
            for (int q = 2; q < npan; ++q) panel(ad + kPanelStep * (uint64_t)q, d0 + 32u * (uint32_t)q);
            ad += kPanelStep * (uint64_t)np;
            bd += kTileStep * (uint64_t)terms;
            acc = 1u;
          }
          if (leader) tc_commit(smem_u32(&bars.empty[stage]));
          sbase += stage_bytes;
          if (++stage == S) { stage = 0; phase ^= 1u; sbase = ring_base; }
        }
        if (!ok) break;
        if (leader) {
          if (s.t1 > s.t0) tc_commit(smem_u32(&bars.acc_full[buf]));
          else mbar_arrive(smem_u32(&bars.acc_full[buf]));
          if (i == begin) stamp<TRACE>(p, 3);
        }
      }
      if (leader) stamp<TRACE>(p, 4);
    }
    __syncwarp();
  } else {
    // epilogue warps: TMEM lane quadrant = warp id mod 4; the two warps of a quadrant split the
    // 32 accumulator columns (tile rows m) in halves
    const int quad = warp & 3;
    const int half = (warp - C::EPI0) >> 2;
    const int epi_tid = (int)threadIdx.x - 32 * C::EPI0;
    const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
    const int m_first = half * C::COLS;
    const OutDesc od = out_desc(p);
    // this warp's part of the staging tile
    const uint32_t part = ring_base + (uint32_t)p.part_off + (uint32_t)(warp - C::EPI0) * (32u * kTile * 2u);
    bool store_pending = false;
    // the column scales and biases this role reads and the C it writes may be the previous kernel's; the index
    // of A may be read ahead of it when the caller vouches for A
    if (!p.a_stable) grid_dependency_wait();
    int begin, end, step;
    seg_range<SPLIT>(p, begin, end, step);
    uint32_t it = 0;
    int seg_next = 0;  // the next segment's descriptor is fetched one item ahead, a word per lane
    if (begin < end) seg_next = load_seg_word<SPLIT>(p, begin, lane);
    if (p.a_stable) grid_dependency_wait();
    if (epi_tid == 0) stamp<TRACE>(p, 0);
    for (int i = begin; i < end; i += step, ++it) {
      const int seg = seg_next;
      if (i + step < end) seg_next = load_seg_word<SPLIT>(p, i + step, lane);
      const int row = word_of(seg, 0), chunk = word_of(seg, 1), nseg = SPLIT ? word_of(seg, 4) : 1;
      const int npan = panels_in_chunk(p, chunk);
      const uint32_t buf = it & 1u, aph = (it >> 1) & 1u;
      const bool has = word_of(seg, 3) > word_of(seg, 2);
      // an empty tile row is zeros (+ bias): nothing to scale, no scales to wait for
      const float rs = (p.row_scale != nullptr && (has || nseg > 1)) ? p.row_scale[row] : 1.0f;
      const int n_base = chunk * p.np * kPanelN + quad * 32 + lane;
      // per-column scale and bias of the first panel are fetched before the accumulator is ready
      float cs = p.b_scale, bias = 0.0f;
      if (n_base < p.N) {
        if (p.col_scale != nullptr && (has || nseg > 1)) cs = p.col_scale[n_base] * p.b_scale;
        if (p.bias != nullptr) bias = p.bias[n_base];
      }
      // one warp waits, the named barrier hands its verdict to all epilogue warps, so that they
      // leave the loop together if the wait gave up (a warp that went on alone would wait at the next
      // named barrier for ever)
      if (epi_tid < 32) {
        const bool in = mbar_wait_warp(smem_u32(&bars.acc_full[buf]), aph, ctl);
        if (epi_tid == 0) ok_s[it & 1u] = in ? 1 : 0;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
      if (!ok_s[it & 1u]) break;
      if (epi_tid == 0 && i == begin) stamp<TRACE>(p, 5);
      if (epi_tid == 0) stamp<TRACE>(p, 8);
      tc_fence_after();
      // Everything but whole rows into C alone goes through here first: raw accumulators for the caller, pieces of split rows.
      const bool whole = !SPLIT || (nseg == 1 && (STAGED || (od.acc_out == nullptr && p.worker_partials == nullptr)));
      const bool peers = SPLIT && !STAGED && p.n_peers > 0 && nseg > 1;
      if (!whole) {
        const int owner = word_of(seg, 5), ctr = word_of(seg, 7);
        // a split row whose scratch index lies outside what the caller provided is skipped and reported
        const bool bad_split = nseg > 1 && (ctr < 0 || ctr >= p.ctr_limit || (p.n_peers > 0 && (unsigned)owner >= (unsigned)p.n_peers));
        int32_t *split_partials = p.partials, *counter = p.counters + ctr;
        if constexpr (SPLIT && !STAGED)
          if (peers && !bad_split) {
            split_partials = x.partials[owner];
            counter = x.counters[owner] + ctr;
          }
        if (bad_split && epi_tid == 0 && p.status != nullptr) atomicCAS(p.status, 0, kStatusBadPlan);
#pragma unroll 1
        for (int q = 0; q < npan; ++q) {
          const int n = n_base + q * kPanelN;
          float csq = p.b_scale, biasq = 0.0f;
          if (!STAGED && n < p.N) {
            if (p.col_scale != nullptr) csq = p.col_scale[n] * p.b_scale;
            if (p.bias != nullptr) biasq = p.bias[n];
          }
          // all columns of the panel with one wait, then the accumulator buffer goes back to the MMA warp
          uint32_t ra[C::COLS];
          if (has) {
            tmem_ld_cols<C::COLS>(tmem_base + lane_sel + buf * acc_cols + (uint32_t)(q * 32 + m_first), ra);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int k = 0; k < C::COLS; ++k) ra[k] = 0u;
          }
          if (q == npan - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars.acc_empty[buf]));
          }
#pragma unroll
          for (int c = 0; c < C::COLS; c += 8) {
            const int m0 = m_first + c;
            uint32_t r[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) r[k] = ra[c + k];
            if (!STAGED && p.worker_partials != nullptr && n < p.N) {
              uint32_t* w = reinterpret_cast<uint32_t*>(p.worker_partials) + ((size_t)i * kTile + m0) * p.N + n;
#pragma unroll
              for (int k = 0; k < 8; ++k) w[(size_t)k * p.N] = r[k];
            }
            if (!STAGED && nseg == 1) {
              finish8<KIND>(od, row, n, m0, r, rs, csq, biasq);
            } else if (!bad_split && has) {
              // partial sum of a split row: added into the row's int32 accumulator in global memory
              // (integer adds commute, so the total does not depend on which CTA - or which GPU - comes first)
              int32_t* dst = split_partials + ((size_t)ctr * p.np + q) * (kTile * kPanelN) + (size_t)m0 * kPanelN +
                             (quad * 32 + lane);
              if (peers && p.peer_slots) {
                // this rank's own slot of the row: nothing else writes it, plain stores (NVLink writes for a remote owner)
                int32_t* slot = split_partials + (((size_t)ctr * p.n_peers + word_of(seg, 6)) * p.np + q) * (kTile * kPanelN) +
                                (size_t)m0 * kPanelN + (quad * 32 + lane);
#pragma unroll
                for (int k = 0; k < 8; ++k) slot[k * kPanelN] = (int32_t)r[k];
              } else if (!STAGED && p.n_peers > 0) {   // the accumulator may be another GPU's: system-wide adds over NVLink
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                  if (KIND == VOID_KIND_I8) atomicAdd_system(dst + k * kPanelN, (int32_t)r[k]);
                  else atomicAdd_system(reinterpret_cast<float*>(dst) + k * kPanelN, __uint_as_float(r[k]));
                }
              } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                  if (KIND == VOID_KIND_I8) red_add_s32(dst + k * kPanelN, (int32_t)r[k]);
                  else red_add_f32(reinterpret_cast<float*>(dst) + k * kPanelN, __uint_as_float(r[k]));
                }
              }
            }
          }
        }
        if (nseg == 1 || bad_split || (peers && p.peer_slots)) continue;
        // the CTA that arrives last reads the completed sums back and finishes the row
        if (epi_tid == 0) stamp<TRACE>(p, 12);
        // The arrival is one release-acquire add by one thread after a barrier of the epilogue warps: the barrier
        // orders every warp's additions before it, the release makes them visible before the count, and the
        // acquire lets the last arriver - after the second barrier - read what the other CTAs added.
        if (peers) __threadfence_system();
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
        if (epi_tid == 0) stamp<TRACE>(p, 13);
        if (epi_tid == 0) {
          const int old = peers ? atomicAdd_system(counter, 1) : atom_add_acq_rel(counter, 1);
          const int last = (old == nseg - 1) ? 1 : 0;
          if (last) *counter = 0;  // left clean for the next launch
          last_s = last;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
        const int last = last_s;
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
        if (epi_tid == 0) stamp<TRACE>(p, 14);
        if (TRACE && epi_tid == 0 && p.trace != nullptr) p.trace[(size_t)blockIdx.x * 64 + 15] = (unsigned long long)last;
        if (!last) continue;
        if (peers) __threadfence_system();
        if (epi_tid == 0) stamp<TRACE>(p, 28);
      }
      // Finished values, panel by panel: of a whole row from tensor memory, of a split row from its sums.  The values of a
      // panel are requested at once and awaited once; an accumulator buffer goes back to the MMA warp as soon as they sit in
      // registers, a row's sums in global memory are cleared for the next launch.
#pragma unroll 1
      for (int q = 0; q < npan; ++q) {
        const int n = n_base + q * kPanelN;
        const uint32_t acc_addr = tmem_base + lane_sel + buf * acc_cols + (uint32_t)(q * 32 + m_first);
        float csq = cs, biasq = bias;   // the first panel's were read before the accumulator was ready
        if (q > 0) {
          csq = p.b_scale; biasq = 0.0f;
          if (n < p.N) {
            if (p.col_scale != nullptr) csq = p.col_scale[n] * p.b_scale;
            if (p.bias != nullptr) biasq = p.bias[n];
          }
        }
        if constexpr (STAGED) {
          // 16-bit outputs: every epilogue warp puts its part of the result tile (32 columns of the tile row) together in its own
          // piece of shared memory and sends it off itself - no barrier between the warps.  The copy engine clips at the
          // edges of C; the part is free again once the previous store has read it.
          uint32_t lo[16], hi[16];
          if (!whole) {
            const int32_t* from = row_sums(p, x, seg, peers, q) + quad * 32 + 2 * (lane & 3) * kPanelN + (lane >> 2);
#pragma unroll
            for (int k = 0; k < 16; ++k) {   // rows 8 (k / 4) + k % 2 further, columns 8 (k / 2 % 2), and 16 more
              lo[k] = (uint32_t)__ldcg(from + (8 * (k >> 2) + (k & 1)) * kPanelN + 8 * ((k >> 1) & 1));
              hi[k] = (uint32_t)__ldcg(from + (8 * (k >> 2) + (k & 1)) * kPanelN + 8 * ((k >> 1) & 1) + 16);
            }
          } else if (has) {
            tmem_ld_fragments(acc_addr, lo, hi);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int k = 0; k < 16; ++k) lo[k] = hi[k] = 0u;
          }
          if (epi_tid == 0 && q == 0) stamp<TRACE>(p, 9);
          if (whole && q == npan - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars.acc_empty[buf]));
          }
          if (store_pending) {
            if (lane == 0) bulk_wait_read();
            __syncwarp();
          }
          if (whole && !has && p.bias == nullptr && p.row_bias == nullptr) {
            // an empty tile row without bias is zeros under every activation: no conversions
            uint4* z = reinterpret_cast<uint4*>(smem_raw + (part - smem_u32(smem_raw))) + lane;
#pragma unroll
            for (int k = 0; k < 4; ++k) z[k * 32] = make_uint4(0u, 0u, 0u, 0u);
          } else {
            finish_fragments<KIND, ACT>(od, row * kTile, lo, hi, rs, csq, biasq, p.bias != nullptr, part, lane);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&x, part, (chunk * p.np + q) * kPanelN + quad * 32, row * kTile);
            bulk_commit();
          }
          store_pending = true;
          // (after the store has been issued: the fence in front of it would wait for these writes)
          if (!whole) {
            int32_t* sums = row_sums(p, x, seg, peers, q) + m_first * kPanelN + quad * 32;
#pragma unroll
            for (int k = 0; k < 8; ++k) reinterpret_cast<int4*>(sums)[(lane >> 3) * 32 + k * 128 + (lane & 7)] = make_int4(0, 0, 0, 0);
          }
        } else {
          uint32_t r[C::COLS];
          OutDesc to = od;
          if (!whole) {
            int32_t* sums = row_sums(p, x, seg, peers, q) + m_first * kPanelN + quad * 32;
#pragma unroll
            for (int k = 0; k < C::COLS; ++k) r[k] = (uint32_t)(peers ? __ldcv(sums + k * kPanelN + lane) : __ldcg(sums + k * kPanelN + lane));
#pragma unroll
            for (int k = 0; k < C::COLS; ++k) sums[k * kPanelN + lane] = 0;
            if (od.acc_out != nullptr && n < od.N) {
              uint32_t* a = reinterpret_cast<uint32_t*>(od.acc_out) + ((size_t)row * kTile + m_first) * od.N + n;
#pragma unroll
              for (int k = 0; k < C::COLS; ++k) a[(size_t)k * od.N] = r[k];
            }
            if constexpr (SPLIT && !STAGED)
              if (peers) to.out = x.out[word_of(seg, 5)];   // the owner's rows of C
          } else if (has) {
            tmem_ld_cols<C::COLS>(acc_addr, r);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int k = 0; k < C::COLS; ++k) r[k] = 0u;
          }
          if (whole && q == npan - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars.acc_empty[buf]));
          }
#pragma unroll
          for (int c = 0; c < C::COLS; c += 16) {
            if (TR) finish16_tr<KIND, ACT>(to, row, n, m_first + c, &r[c], rs, csq, biasq);
            else finish16<KIND, ACT>(to, row, n, m_first + c, &r[c], rs, csq, biasq);
          }
        }
        if (epi_tid == 0 && q == 0) stamp<TRACE>(p, 10);
      }
    }
    // a part must have been read before shared memory is given back; the writes themselves
    // complete with the kernel
    if (store_pending && lane == 0) bulk_wait_read();
    if (epi_tid == 0) stamp<TRACE>(p, 6);
  }
  pipeline_teardown<C, TRACE>(p, ctl_s, tmem_base, tmem_cols);
}

template <int KIND, class C, int TR, int EPI>
int launch_rowacc(const RowaccLaunch& l) {
  auto kernel = spmm_rowacc_kernel<KIND, C, TR, EPI>;
  if (ensure_smem((const void*)kernel, l.smem_bytes)) return VOID_ERR_CUDA;
  if constexpr ((EPI & kStaged) != 0) return status_of(launch_pdl(kernel, l.grid, C::THREADS, l.smem_bytes, l.stream, l.b, l.c, l.p));
  else if constexpr ((EPI & kSplit) != 0) return status_of(launch_pdl(kernel, l.grid, C::THREADS, l.smem_bytes, l.stream, l.b, l.peers, l.p));
  else return status_of(launch_pdl(kernel, l.grid, C::THREADS, l.smem_bytes, l.stream, l.b, Nothing{}, l.p));
}
template <int KIND, class C>
int launch_rowacc(const RowaccLaunch& l) {
  if constexpr (KIND != VOID_KIND_F8E4M3 && (KIND != VOID_KIND_I8 || C::COLS == kTile)) {
    if (l.transposed)
      return l.transposed == 1
                 ? (l.epilogue & kActive ? launch_rowacc<KIND, C, 1, kActive>(l) : launch_rowacc<KIND, C, 1, 0>(l))
                 : (l.epilogue & kActive ? launch_rowacc<KIND, C, 2, kActive>(l) : launch_rowacc<KIND, C, 2, 0>(l));
  }
  switch (l.epilogue) {
    case 0: return launch_rowacc<KIND, C, 0, 0>(l);
    case kActive: return launch_rowacc<KIND, C, 0, kActive>(l);
    default: break;
  }
  if constexpr (C::COLS == kTile) {   // slim and mid
    if (l.epilogue == kStaged) return launch_rowacc<KIND, C, 0, kStaged>(l);
    if (l.epilogue == (kStaged | kActive)) return launch_rowacc<KIND, C, 0, kStaged | kActive>(l);
  }
  if constexpr (C::CTAS_PER_SM != Mid::CTAS_PER_SM) {
    if (l.epilogue == (kSplit | kActive)) return launch_rowacc<KIND, C, 0, kSplit | kActive>(l);
    if constexpr (KIND != VOID_KIND_F8E4M3 && C::COLS == kTile)
      if (l.epilogue == (kStaged | kSplit | kActive)) return launch_rowacc<KIND, C, 0, kStaged | kSplit | kActive>(l);
  }
  if constexpr (KIND == VOID_KIND_I8 && C::COLS == kTile) {
    constexpr int T = kTraced | kActive;
    switch (l.epilogue) {
      case T: return launch_rowacc<KIND, C, 0, T>(l);
      case T | kStaged: return launch_rowacc<KIND, C, 0, T | kStaged>(l);
      case T | kSplit: return launch_rowacc<KIND, C, 0, T | kSplit>(l);
      case T | kStaged | kSplit: return launch_rowacc<KIND, C, 0, T | kStaged | kSplit>(l);
    }
  }
  return VOID_ERR_BAD_ARG;
}
template <int KIND>
int launch_rowacc(const RowaccLaunch& l) {
  if constexpr (KIND == VOID_KIND_F16 || KIND == VOID_KIND_TF32)
    if (l.shape == 6) return launch_rowacc<KIND, Mid>(l);
  return l.shape == 2 ? launch_rowacc<KIND, Slim>(l) : launch_rowacc<KIND, Wide>(l);
}

}  // namespace vb
