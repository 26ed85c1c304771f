// The row-accumulate kernel (pipeline.cuh): one accumulator per (tile row, column chunk).
#pragma once
#include "pipeline.cuh"

namespace vb {

// All COLS accumulator columns of one epilogue warp, requested together (no wait).
template <int COLS>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[COLS]) {
#pragma unroll
  for (int c = 0; c < COLS; c += 16) tmem_ld_32x16p(taddr + (uint32_t)c, &r[c]);
}

// TR: 1 = B and C transposed ([N, K] and [N, M]), 2 = C alone
template <int KIND, class C, int TR = 0, bool TRACE = false>
__global__ void __launch_bounds__(C::THREADS, C::CTAS_PER_SM) spmm_rowacc_kernel(const __grid_constant__ CUtensorMap tmap_b,
                                                               const __grid_constant__ CUtensorMap tmap_c,
                                                               const __grid_constant__ SpmmParams p) {
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
  const uint32_t ring_bytes = (uint32_t)((p.stages - 1) * p.group + p.last_group) * unit_smem;
  const uint32_t acc_cols = (uint32_t)p.np * 32u;  // TMEM columns of one accumulator buffer
  uint32_t tmem_cols = 32;
  while (tmem_cols < 2u * acc_cols) tmem_cols <<= 1;
  volatile int* ctl = ctl_s;

  if (threadIdx.x == 0) last_s = 0;
  pipeline_setup<C, ES, TRACE>(p, &tmap_b, bars, &tmem_base_s, ctl_s, 2, tmem_cols);
  const uint32_t tmem_base = tmem_base_s;

  if (warp < C::PW) {
    producer_loop<C, ES, TR, TRACE>(p, &tmap_b, &bars, ring_base, stage_bytes, ctl, lane, warp);
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
      seg_range(p, begin, end, step);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t sbase = ring_base;
      uint32_t it = 0;
      bool ok = true;
      Seg seg_next = {};  // the next segment's descriptor is fetched one item ahead
      if (begin < end) seg_next = load_seg(p, begin);
      for (int i = begin; i < end && ok; i += step, ++it) {
        const Seg s = seg_next;
        if (i + step < end) seg_next = load_seg(p, i + step);
        const int npan = panels_in_chunk(p, s.chunk);
        const uint32_t buf = it & 1u, aph = (it >> 1) & 1u;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.acc_empty[buf]), aph ^ 1u, ctl));
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
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.full[stage]), phase, ctl));
          if (!ok) break;
          if (TRACE && leader && i == begin && gidx < 12) stamp<TRACE>(p, 16 + gidx);   // slots 28 .. 31: last arriver of a split row
          tc_fence_after();
          uint64_t ad = smem_desc(hi_a, sbase);
          uint64_t bd = smem_desc(hi_b, sbase + tile_off<ES>(p, cap, 0));
          for (int j = 0; j < gcnt; ++j) {
            uint64_t adq = ad;
            uint32_t d = d0;
            for (int q = 0; q < npan; ++q) {
              if (leader) issue_mma<KIND>(d, adq, bd, idesc, acc);
#pragma unroll
              for (int kk = 1; kk < ES; ++kk)
                if (leader) issue_mma<KIND>(d, adq + kk * kPanelKStep, bd + kk * kTileKStep, idesc, 1u);
              // a tile stored as a sum of terms: every further term multiplies the same panel
              if (KIND == VOID_KIND_F8E4M3)
                for (int v = 1; v < terms; ++v)
                  if (leader) issue_mma<KIND>(d, adq, bd + (uint64_t)v * kTileStep, idesc, 1u);
              adq += kPanelStep;
              d += 32u;
            }
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
    // staging tile of the TMA-store epilogue: behind the ring
    const uint32_t stage_u32 = ring_base + ring_bytes;
    uint16_t* stage_tile = reinterpret_cast<uint16_t*>(smem_raw + (stage_u32 - smem_u32(smem_raw)));
    bool store_pending = false;
    // the column scales and biases this role reads and the C it writes may be the previous kernel's; the index
    // of A may be read ahead of it when the caller vouches for A
    if (!p.a_stable) grid_dependency_wait();
    int begin, end, step;
    seg_range(p, begin, end, step);
    uint32_t it = 0;
    Seg seg_next = {};  // the next segment's descriptor is fetched one item ahead
    if (begin < end) seg_next = load_seg(p, begin);
    if (p.a_stable) grid_dependency_wait();
    if (epi_tid == 0) stamp<TRACE>(p, 0);
    for (int i = begin; i < end; i += step, ++it) {
      const Seg s = seg_next;
      if (i + step < end) seg_next = load_seg(p, i + step);
      const int npan = panels_in_chunk(p, s.chunk);
      const uint32_t buf = it & 1u, aph = (it >> 1) & 1u;
      const bool has = s.t1 > s.t0;
      // an empty tile row is zeros (+ bias): nothing to scale, no scales to wait for
      const float rs = (p.row_scale != nullptr && (has || s.nseg > 1)) ? __ldg(p.row_scale + s.row) : 1.0f;
      const int n_base = s.chunk * p.np * kPanelN + quad * 32 + lane;
      // per-column scale and bias of the first panel are fetched before the accumulator is ready
      float cs = p.b_scale, bias = 0.0f;
      if (n_base < p.N) {
        if (p.col_scale != nullptr && (has || s.nseg > 1)) cs = __ldg(p.col_scale + n_base) * p.b_scale;
        if (p.bias != nullptr) bias = __ldg(p.bias + n_base);
      }
      // a split row whose scratch index lies outside what the caller provided is skipped and reported
      const bool peers = p.n_peers > 0 && s.nseg > 1;
      const bool bad_split = s.nseg > 1 && (s.ctr < 0 || s.ctr >= p.ctr_limit || (peers && (unsigned)s.slot0 >= (unsigned)p.n_peers));
      int32_t* split_partials = p.partials;
      int32_t* split_counters = p.counters;
      if (peers && !bad_split) {
        split_partials = p.peer_partials[s.slot0];
        split_counters = p.peer_counters[s.slot0];
      }
      if (bad_split && epi_tid == 0 && p.status != nullptr) atomicCAS(p.status, 0, kStatusBadPlan);
      // one thread waits, the named barrier hands its verdict to all epilogue warps, so that they
      // leave the loop together if the wait gave up (a warp that went on alone would wait at the next
      // named barrier for ever)
      if (epi_tid == 0) ok_s[it & 1u] = mbar_wait(smem_u32(&bars.acc_full[buf]), aph, ctl) ? 1 : 0;
      asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
      if (!ok_s[it & 1u]) break;
      if (epi_tid == 0 && i == begin) stamp<TRACE>(p, 5);
      if (epi_tid == 0) stamp<TRACE>(p, 8);
      tc_fence_after();
      const bool fast = s.nseg == 1 && od.acc_out == nullptr && p.worker_partials == nullptr;
#pragma unroll 1
      for (int q = 0; q < npan; ++q) {
        const int n = n_base + q * kPanelN;
        const uint32_t acc_addr = tmem_base + lane_sel + buf * acc_cols + (uint32_t)(q * 32 + m_first);
        if (fast) {
          // All of this warp's columns of the panel are requested at once and awaited once; the
          // accumulator buffer goes back to the MMA warp as soon as the values sit in registers.
          float csq = cs, biasq = bias;
          if (q > 0) {
            csq = p.b_scale; biasq = 0.0f;
            if (n < p.N) {
              if (p.col_scale != nullptr) csq = __ldg(p.col_scale + n) * p.b_scale;
              if (p.bias != nullptr) biasq = __ldg(p.bias + n);
            }
          }
          uint32_t r[C::COLS];
          if (has) {
            tmem_ld_cols<C::COLS>(acc_addr, r);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int k = 0; k < C::COLS; ++k) r[k] = 0u;
          }
          if (epi_tid == 0 && q == 0) stamp<TRACE>(p, 9);
          if (q == npan - 1) {  // this warp is done with the accumulator buffer
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars.acc_empty[buf]));
          }
          if (!TR && p.tma_store == 2) {
            // 16-bit outputs, one store per epilogue warp: the warp puts its 32 x 32 part of the result tile
            // together in its own 2 KB of shared memory and sends it off itself - no barrier between the warps.
            // The copy engine clips at the edges of C; the part is free again once the previous store has read it.
            if (store_pending) {
              if (lane == 0) bulk_wait_read();
              __syncwarp();
            }
            uint16_t* part = stage_tile + quad * (32 * 32);
            if (!has && p.bias == nullptr && p.row_bias == nullptr) {
              // an empty tile row without bias is zeros under every activation: 2 KB of zero words, no conversions
              uint4* z = reinterpret_cast<uint4*>(part) + lane;
#pragma unroll
              for (int k = 0; k < 4; ++k) z[k * 32] = make_uint4(0u, 0u, 0u, 0u);
            } else {
#pragma unroll
              for (int c = 0; c < C::COLS; c += 16)
                finish16_stage<KIND, 32>(od, s.row, n, m_first + c, &r[c], rs, csq, biasq, part + lane);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&tmap_c, stage_u32 + (uint32_t)quad * (32 * 32 * 2), (s.chunk * p.np + q) * kPanelN + quad * 32,
                           s.row * kTile);
              bulk_commit();
            }
            store_pending = true;
          } else if (!TR && p.tma_store) {
            // 16-bit outputs: the 32 x 128 result tile is put together in shared memory and leaves in one
            // tiled store; the copy engine clips it at the edges of C.  The staging tile is free again once
            // the previous store has read it.
            if (store_pending) {
              if (epi_tid == 0) bulk_wait_read();
              asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
            }
#pragma unroll
            for (int c = 0; c < C::COLS; c += 16)
              finish16_stage<KIND, kPanelN>(od, s.row, n, m_first + c, &r[c], rs, csq, biasq, stage_tile + quad * 32 + lane);
            fence_proxy_async_smem();
            asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
            if (epi_tid == 0) {
              tma_store_2d(&tmap_c, stage_u32, (s.chunk * p.np + q) * kPanelN, s.row * kTile);
              bulk_commit();
            }
            store_pending = true;
          } else {
#pragma unroll
            for (int c = 0; c < C::COLS; c += 16) {
              if (TR) finish16_tr<KIND>(od, s.row, n, m_first + c, &r[c], rs, csq, biasq);
              else finish16<KIND>(od, s.row, n, m_first + c, &r[c], rs, csq, biasq);
            }
          }
          if (epi_tid == 0 && q == 0) stamp<TRACE>(p, 10);
          continue;
        }
        float csq = p.b_scale, biasq = 0.0f;
        if (n < p.N) {
          if (p.col_scale != nullptr) csq = __ldg(p.col_scale + n) * p.b_scale;
          if (p.bias != nullptr) biasq = __ldg(p.bias + n);
        }
        // (raw accumulators wanted, or a piece of a split row) all columns of the panel with one wait, then the
        // accumulator buffer goes back to the MMA warp
        uint32_t ra[C::COLS];
        if (has) {
          tmem_ld_cols<C::COLS>(acc_addr, ra);
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
          if (p.worker_partials != nullptr && n < p.N) {
            uint32_t* w = reinterpret_cast<uint32_t*>(p.worker_partials) + ((size_t)i * kTile + m0) * p.N + n;
#pragma unroll
            for (int k = 0; k < 8; ++k) w[(size_t)k * p.N] = r[k];
          }
          if (s.nseg == 1) {
            finish8<KIND>(od, s.row, n, m0, r, rs, csq, biasq);
          } else if (!bad_split && has) {
            // partial sum of a split row: added into the row's int32 accumulator in global memory
            // (integer adds commute, so the total does not depend on which CTA - or which GPU - comes first)
            int32_t* dst = split_partials + ((size_t)s.ctr * p.np + q) * (kTile * kPanelN) + (size_t)m0 * kPanelN +
                           (quad * 32 + lane);
            if (peers && p.peer_slots) {
              // this rank's own slot of the row: nothing else writes it, plain stores (NVLink writes for a remote owner)
              int32_t* slot = split_partials + (((size_t)s.ctr * p.n_peers + s.my_idx) * p.np + q) * (kTile * kPanelN) +
                              (size_t)m0 * kPanelN + (quad * 32 + lane);
#pragma unroll
              for (int k = 0; k < 8; ++k) slot[k * kPanelN] = (int32_t)r[k];
            } else if (p.n_peers > 0) {   // the accumulator may be another GPU's: system-wide adds over NVLink
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
      if (s.nseg > 1 && !bad_split && !(peers && p.peer_slots)) {
        // the CTA that arrives last reads the completed sums back and finishes the row
        if (epi_tid == 0) stamp<TRACE>(p, 12);
        // The arrival is one release-acquire add by one thread after a barrier of the epilogue warps: the barrier
        // orders every warp's additions before it, the release makes them visible before the count, and the
        // acquire lets the last arriver - after the second barrier - read what the other CTAs added.
        if (peers) __threadfence_system();
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
        if (epi_tid == 0) stamp<TRACE>(p, 13);
        if (epi_tid == 0) {
          const int old = peers ? atomicAdd_system(split_counters + s.ctr, 1) : atom_add_acq_rel(split_counters + s.ctr, 1);
          const int last = (old == s.nseg - 1) ? 1 : 0;
          if (last) split_counters[s.ctr] = 0;  // left clean for the next launch
          last_s = last;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
        const int last = last_s;
        asm volatile("bar.sync 1, %0;" ::"n"(C::EPI_THREADS) : "memory");
        if (epi_tid == 0) stamp<TRACE>(p, 14);
        if (TRACE && epi_tid == 0 && p.trace != nullptr) p.trace[(size_t)blockIdx.x * 64 + 15] = (unsigned long long)last;
        if (last) {
          if (peers) __threadfence_system();
          if (epi_tid == 0) stamp<TRACE>(p, 28);
          OutDesc od2 = od;
          od2.acc_out = nullptr;
          if (peers) od2.out = p.peer_out[s.slot0];   // the owner's rows of C
#pragma unroll 1
          for (int q = 0; q < npan; ++q) {
            const int n = n_base + q * kPanelN;
            float csq = cs, biasq = bias;   // the first panel's were read before the accumulator was ready
            if (q > 0) {
              csq = p.b_scale; biasq = 0.0f;
              if (n < p.N) {
                if (p.col_scale != nullptr) csq = __ldg(p.col_scale + n) * p.b_scale;
                if (p.bias != nullptr) biasq = __ldg(p.bias + n);
              }
            }
            // all of this warp's sums of the panel are requested at once (one L2 round trip), then
            // the accumulator is cleared for the next launch
            int32_t* src = split_partials + ((size_t)s.ctr * p.np + q) * (kTile * kPanelN) + (size_t)m_first * kPanelN +
                           (quad * 32 + lane);
            uint32_t rl[C::COLS];
            if (TRACE && epi_tid == 0 && q == 0) { asm volatile("" ::"f"(csq), "f"(biasq) : "memory"); stamp<TRACE>(p, 29); }
#pragma unroll
            for (int k = 0; k < C::COLS; ++k)
              rl[k] = (uint32_t)(peers ? __ldcv(src + k * kPanelN) : __ldcg(src + k * kPanelN));
            if (TRACE && epi_tid == 0 && q == 0) { asm volatile("" ::"r"(rl[0]), "r"(rl[C::COLS - 1]) : "memory"); stamp<TRACE>(p, 30); }
            if (epi_tid == 0 && q == 0) stamp<TRACE>(p, 31);
            if (!TR && p.tma_store == 2 && !peers && od.acc_out == nullptr) {
              // 16-bit outputs leave as in the unsplit case: the warp's 32 x 32 part through shared memory and one tiled store
              if (store_pending) {
                if (lane == 0) bulk_wait_read();
                __syncwarp();
              }
              uint16_t* part = stage_tile + quad * (32 * 32);
#pragma unroll
              for (int c = 0; c < C::COLS; c += 16)
                finish16_stage<KIND, 32>(od, s.row, n, m_first + c, &rl[c], rs, csq, biasq, part + lane);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                tma_store_2d(&tmap_c, stage_u32 + (uint32_t)quad * (32 * 32 * 2), (s.chunk * p.np + q) * kPanelN + quad * 32,
                             s.row * kTile);
                bulk_commit();
              }
              store_pending = true;
              // (cleared after the store has been issued: the fence in front of it would wait for these writes)
#pragma unroll
              for (int k = 0; k < C::COLS; ++k) src[k * kPanelN] = 0;
              continue;
            }
#pragma unroll
            for (int k = 0; k < C::COLS; ++k) src[k * kPanelN] = 0;
#pragma unroll
            for (int c = 0; c < C::COLS; c += 16) {
              if (od.acc_out != nullptr && n < od.N) {
                uint32_t* a = reinterpret_cast<uint32_t*>(od.acc_out) + ((size_t)s.row * kTile + m_first + c) * od.N + n;
#pragma unroll
                for (int k = 0; k < 16; ++k) a[(size_t)k * od.N] = rl[c + k];
              }
              finish16<KIND>(od2, s.row, n, m_first + c, &rl[c], rs, csq, biasq);
            }
          }
        }
      }
    }
    // the staging tile must have been read before shared memory is given back; the writes themselves
    // complete with the kernel
    if (store_pending && (p.tma_store == 2 ? lane == 0 : epi_tid == 0)) bulk_wait_read();
    if (epi_tid == 0) stamp<TRACE>(p, 6);
  }
  pipeline_teardown<C, TRACE>(p, ctl_s, tmem_base, tmem_cols);
}

template <class C, typename Kernel>
int launch_rowacc(Kernel kernel, const RowaccLaunch& l, const CUtensorMap& b, const CUtensorMap& c, const SpmmParams& p) {
  if (ensure_smem((const void*)kernel, l.smem_bytes)) return VOID_ERR_CUDA;
  launch_pdl(kernel, l.grid, C::THREADS, l.smem_bytes, l.stream, b, c, p);
  return VOID_OK;
}
template <int KIND, int TR>
int launch_rowacc_tr(const RowaccLaunch& l, const CUtensorMap& b, const CUtensorMap& c, const SpmmParams& p) {
  if constexpr (KIND != VOID_KIND_I8)
    if (!l.slim) return launch_rowacc<Wide>(spmm_rowacc_kernel<KIND, Wide, TR>, l, b, c, p);
  return launch_rowacc<Slim>(spmm_rowacc_kernel<KIND, Slim, TR>, l, b, c, p);
}
template <int KIND>
int launch_rowacc(const RowaccLaunch& l, const CUtensorMap& b, const CUtensorMap& c, const SpmmParams& p) {
  if constexpr (KIND != VOID_KIND_F8E4M3) {
    if (l.transposed == 1) return launch_rowacc_tr<KIND, 1>(l, b, c, p);
    if (l.transposed == 2) return launch_rowacc_tr<KIND, 2>(l, b, c, p);
  }
  if constexpr (KIND == VOID_KIND_I8)
    if (l.slim && l.traced) return launch_rowacc<Slim>(spmm_rowacc_kernel<KIND, Slim, 0, true>, l, b, c, p);
  return l.slim ? launch_rowacc<Slim>(spmm_rowacc_kernel<KIND, Slim>, l, b, c, p) : launch_rowacc<Wide>(spmm_rowacc_kernel<KIND, Wide>, l, b, c, p);
}

}  // namespace vb
