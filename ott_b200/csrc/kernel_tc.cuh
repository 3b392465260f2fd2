// Persistent Sinkhorn kernel on the tensor-core (tcgen05, BF16 split-3)
// engine. One CTA per SM (its shared memory exceeds half an SM), so the
// 512-column TMEM allocation never waits on another CTA.
//
// A sweep's work units run pipelined across units and roles: the dealer
// warp takes the units (round-robin or from the sweep's atomic queue) and
// publishes each as a descriptor in a ring of four slots in shared memory;
// the producer and MMA warps consume the descriptors in order, so they load
// the next unit's A tile and B tiles and issue its MMAs while the epilogue
// warps still reduce the current unit's last tiles; the finalizer warp
// merges, combines and applies each unit's row results while the epilogue
// warps reduce the next one (a CTA's last unit: four epilogue warps, a row a
// lane). Only the sweep's end, a grid barrier, joins all warps.
#pragma once

#include "engine_tc.cuh"
#include "persistent.cuh"

namespace ottb {

__device__ __forceinline__ TcOperands make_tc_operands(const ProbDev& P, int kind,
                                                       int parity) {
  const TcMaps* maps = reinterpret_cast<const TcMaps*>(P.maps);
  TcOperands op;
  if (kind == kSweepG) {
    op.mapA = &maps->y; op.padA = (int32_t)P.m_pad; op.rows = P.m;
    op.mapB = &maps->x; op.padB = (int32_t)P.n_pad; op.cols = P.n;
    // symmetric problem: the columns' potential is the current g, whose
    // shift rows the g-updates write into y's buffers (y's points are x's)
    op.mapBext = P.symmetric ? &maps->exty : &maps->extx;
    op.extRow0 = P.symmetric ? (int32_t)(parity * P.m_pad) : 0;
  } else {
    op.mapA = &maps->x; op.padA = (int32_t)P.n_pad; op.rows = P.n;
    op.mapB = &maps->y; op.padB = (int32_t)P.m_pad; op.cols = P.m;
    op.mapBext = &maps->exty; op.extRow0 = (int32_t)(parity * P.m_pad);
  }
  return op;
}

// Whether this problem's units of the sweep use the bounded row shift, and
// the bound: D = the largest change of a column shift since the rows' last
// sweep (0 when no potential changed), usable while the spread of those
// changes stays within kMaxShiftSpread.
__device__ __forceinline__ bool shift_bound(const ProbDev& P, const SweepParams& sp, float& dmax) {
  dmax = 0.f;
  if (!sp.fast || P.symmetric || !P.lprev || !P.dkey) return false;
  const int* slot = P.dkey + ((sp.kind * 2 + sp.rslot) * 2);
  const int kmax = __ldcg(slot), kmin = __ldcg(slot + 1);
  float spread = 0.f;
  if (kmax != kDkeyEmptyMax) {
    if (kmin == kDkeyEmptyMin) return false;
    dmax = fkey_value(kmax);
    spread = dmax - fkey_value(kmin);
  }
  return spread <= kMaxShiftSpread && isfinite(dmax);
}

__device__ __forceinline__ RowShift row_shift_of(const ProbDev& P, const SweepParams& sp, bool on,
                                                 float dmax) {
  if (!on) return RowShift{nullptr, 0.f, 0, false};
  return RowShift{P.lprev + (sp.kind == kSweepG ? P.n_pad : 0), dmax,
                  sp.kind == kSweepG ? P.m : P.n, true};
}

// The problem of unit u in a sweep's unit list: the last q with
// prefix[q] <= u (prefix[count] = total > u), by a 32-way search over the
// warp's lanes (two rounds for up to 1024 problems).
__device__ __forceinline__ int warp_find_problem(const int* prefix, int count, int u) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = count;
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) >> 5;
    const int idx = lo + lane * step;
    const bool le = idx < hi && __ldcg(prefix + idx) <= u;
    const unsigned bal = __ballot_sync(0xffffffffu, le);  // lane 0 (idx = lo) is set
    lo += (31 - __clz(bal)) * step;
    hi = min(hi, lo + step);
  }
  return lo;
}

// One sweep on the tensor cores (see the file comment). Returns false,
// uniformly over the CTA, if any wait timed out.
template <int DK, int TN>
__device__ bool tc_sweep(const KernelArgs& A, const SweepParams& sp, unsigned sweep_idx,
                         TcSmem<DK, TN>& sm, TcPipe& pp) {
  constexpr int CG = TcCfg<DK, TN>::kColGroups;
  constexpr uint32_t NSLOT = TcCfg<DK, TN>::kDescSlots;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const volatile int* err = &sm.err;
  const uint64_t tmo = A.timeout_ns;
  // every problem's record is in shared memory, or none
  auto prob = [&](int p) -> const ProbDev& {
    return A.num_problems <= TcCfg<DK, TN>::kProbSlots ? sm.probs[p] : A.probs[p];
  };

  int tail_at = -1;  // one warp: its CTA's last unit, if any
  if (warp == 2) {
    // dealer: every unit of this CTA, then the end marker
    const int* ids = sp.final_eval ? A.eval_ids : A.active_ids;
    const int* pre = sp.final_eval ? A.eval_prefix
                                   : (A.prefix + (sp.kind == kSweepG ? 0 : A.num_problems + 1));
    // A call of one problem needs no look at the unit list (a chain of four
    // trips to L2 before the sweep's first unit): problem 0, its splits.
    const bool one = A.num_problems == 1;
    const int count = one ? 1 : sp.final_eval ? ld_sched(&A.sched->num_eval)
                                              : ld_sched(&A.sched->num_active);
    const int one_split = one ? split_of(A.state[0], sp.kind) : 0;
    const int total = one ? (sp.kind == kSweepG      ? prob(0).rb_g
                             : prob(0).symmetric ? 0  // f = g
                                                 : prob(0).rb_f) * one_split
                      : sp.final_eval ? ld_sched(&A.sched->eval_units)
                                      : ld_sched(&A.sched->total_units[sp.kind == kSweepG ? 0 : 1]);
    const bool dynamic = ld_sched(&A.sched->dynamic_units) != 0;
    // Split 0 (one problem): no units of a split, but the sweep's tiles, row
    // block after row block, dealt to the CTAs in equal runs. A run's part
    // of a row block is a unit; S is the number of CTAs whose runs meet it.
    const bool runs = one && one_split == 0;
    unsigned tiles = 0, row_tiles = 1, pos = 0, run_end = 0;
    if (runs) {
      const ProbDev& P = prob(0);
      row_tiles = (unsigned)(((sp.kind == kSweepG ? P.n : P.m) + TN - 1) / TN);
      tiles = row_tiles * (unsigned)(sp.kind == kSweepG ? P.rb_g : P.symmetric ? 0 : P.rb_f);
      // the host takes runs only where tiles * gridDim.x is below 2^31
      const unsigned v = tiles * (blockIdx.x + (lane & 1)) / gridDim.x;
      pos = __shfl_sync(0xffffffffu, v, 0);
      run_end = __shfl_sync(0xffffffffu, v, 1);
    }
    // the bounded row shift of the one problem: its keys' loads are in flight
    // with the others
    float dmax = 0.f;
    bool on = one && shift_bound(prob(0), sp, dmax);
    unsigned* ctr = &A.gl->unit_ctr[sweep_idx % 3];
    if (blockIdx.x == 0 && lane == 0) A.gl->unit_ctr[(sweep_idx + 1) % 3] = 0u;
    int rr = blockIdx.x;
    bool ended = false;
    while (!ended) {
      const uint32_t w = pp.wdesc++;
      const uint32_t slot = w % NSLOT;
      bool ok = w < NSLOT || tc::mbar_wait(&sm.unit_empty[slot], ((w - NSLOT) / NSLOT) & 1, tmo);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicExch(&sm.err, 1);
        break;
      }
      TcUnit& u = sm.units[slot];
      int ui = 0;
      if (lane == 0) ui = runs ? 0 : dynamic ? (int)atomicAdd(ctr, 1u) : rr;
      ui = __shfl_sync(0xffffffffu, ui, 0);
      rr += gridDim.x;
      // after an error the end marker lets the other roles unwind at once
      if ((runs ? pos >= run_end : ui >= total) || __any_sync(0xffffffffu, *err != 0)) {
        ended = true;
        if (lane == 0) u.end = 1;
      } else {
        const int q = one ? 0 : warp_find_problem(pre, count, ui);
        unsigned rb = 0, first = 0, last = 0, end = 0;
        if (runs) {
          rb = pos / row_tiles;
          end = (rb + 1) * row_tiles;  // of the row block
          // the CTA of tile t: the last one whose run starts at t or before
          const unsigned t = (lane & 1) ? end - 1 : end - row_tiles;
          const unsigned c = ((t + 1) * gridDim.x - 1) / tiles;
          first = __shfl_sync(0xffffffffu, c, 0);
          last = __shfl_sync(0xffffffffu, c, 1);
        }
        if (lane == 0) {
          const int p = one ? 0 : __ldcg(ids + q);
          const ProbDev& P = prob(p);
          u.end = 0;
          u.p = p;
          u.parity = sp.final_eval ? __ldcg(&A.state[p].final_parity) : sp.parity;
          if (runs) {
            u.S = (int)(last - first) + 1;
            u.rb = (int)rb;
            u.sidx = (int)(blockIdx.x - first);
            u.t0 = (int)(pos - (end - row_tiles));
            u.t1 = (int)(min(end, run_end) - (end - row_tiles));
          } else {
            const int local = one ? ui : ui - __ldcg(pre + q);
            const int S = one ? one_split : split_of(A.state[p], sp.kind);
            u.S = S;
            u.rb = (int)((unsigned)local / (unsigned)S);
            u.sidx = local - u.rb * S;
            // at most 2^24 tiles and 32 splits: 32-bit products and divisions
            const int64_t cols = sp.kind == kSweepG ? P.n : P.m;
            const unsigned ntiles = (unsigned)((cols + TN - 1) / TN);
            u.t0 = (int)(ntiles * (unsigned)u.sidx / (unsigned)S);
            u.t1 = (int)(ntiles * (unsigned)(u.sidx + 1) / (unsigned)S);
          }
          // The x layout carries the exponent scale of the target epsilon; a
          // sweep at another epsilon scales the accumulator by ws / ws_t.
          u.r = sp.mult == 1.0f ? 1.0f : sweep_wscale(P, sp.mult) / P.ws_t;
          u.op = make_tc_operands(P, sp.kind, u.parity);
          if (!one) on = shift_bound(P, sp, dmax);
          u.rs = row_shift_of(P, sp, on, dmax);
        }
        pos = min(end, run_end);
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sm.unit_full[slot]);
    }
  } else if (warp == 3) {
    // finalizer: per unit, merge the column groups' (shift, sum) of each row
    // (lane l: rows l + 32 k), combine the column splits of a row block
    // (the CTA that completes its last split finishes it, as sweep_units)
    // and update the rows' potentials. Where the unit is the CTA's last of
    // the sweep, nothing hides the merge and the update, and the epilogue
    // warps have nothing left to do: four of them take a row a lane (tail
    // below).
    bool handed = false;
    while (true) {
      const uint32_t d = pp.desc++;
      const uint32_t slot = d % NSLOT;
      bool ok = tc::mbar_wait(&sm.unit_full[slot], (d / NSLOT) & 1, tmo);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicExch(&sm.err, 1);
        break;
      }
      const TcUnit& u = sm.units[slot];
      const bool stop = u.end != 0 || __any_sync(0xffffffffu, *err != 0);
      if (!stop) {
        const uint32_t pb = pp.unit & 1;
        const ProbDev& P = prob(u.p);
        // what the update reads besides the sums, while they are computed
        RowInputs<4> in;
        load_row_inputs(P, sp, u.parity, (int64_t)u.rb * kBM, sm.log2t, in);
        ok = __all_sync(0xffffffffu, tc::mbar_wait(&sm.epi_done[pb], (pp.unit >> 1) & 1, tmo));
        ++pp.unit;
        if (!ok) {
          if (lane == 0) atomicExch(&sm.err, 1);
          break;
        }
        float mv[4], lv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = lane + 32 * k;
          mv[k] = sm.part_m[pb][0][r];
          lv[k] = sm.part_l[pb][0][r];
#pragma unroll
          for (int c = 1; c < CG; ++c) lse_merge(mv[k], lv[k], sm.part_m[pb][c][r], sm.part_l[pb][c][r]);
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&sm.part_free[pb]);
        const int64_t R = sp.kind == kSweepG ? P.m : P.n;
        const int64_t rbase = (int64_t)u.rb * kBM;
        bool do_final = true;
        if (u.S > 1) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int64_t row = rbase + lane + 32 * k;
            if (row < R) {
              P.part_m[(int64_t)u.sidx * R + row] = mv[k];
              P.part_l[(int64_t)u.sidx * R + row] = lv[k];
            }
          }
          // the warp's partials, released by lane 0's arrival; the last
          // arrival acquires the other splits' (a fence on either side of a
          // relaxed add took ~1500 cycles more)
          __syncwarp();
          int last = 0;
          if (lane == 0) {
            int prev;
            asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;"
                         : "=r"(prev)
                         : "l"(P.arrive + u.rb)
                         : "memory");
            last = prev == u.S - 1;
            if (last) atomicExch(&P.arrive[u.rb], 0);
          }
          do_final = __shfl_sync(0xffffffffu, last, 0) != 0;
        }
        if (do_final) {
          // the next descriptor has long been dealt
          const uint32_t d1 = pp.desc, s1 = d1 % NSLOT;
          ok = __all_sync(0xffffffffu, tc::mbar_wait(&sm.unit_full[s1], (d1 / NSLOT) & 1, tmo));
          if (!ok) {
            if (lane == 0) atomicExch(&sm.err, 1);
            break;
          }
          if (sm.units[s1].end) {
            handed = true;
            if (lane == 0) {
              sm.tail = 1;
              tc::mbar_arrive(&sm.tail_full);
            }
          } else {
            if (u.S > 1) {
              // two splits of the four rows at a time: 16 loads in flight (one
              // split of one row after the other took S x 4 trips to L2; four
              // splits at a time spill)
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                mv[k] = kNegSentinel;
                lv[k] = 0.f;
              }
              for (int j0 = 0; j0 < u.S; j0 += 2) {
                float m2[2][4], l2[2][4];
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                  for (int k = 0; k < 4; ++k) {
                    const int64_t row = rbase + lane + 32 * k;
                    const bool in_range = j0 + j < u.S && row < R;
                    const int64_t at = (int64_t)(j0 + j) * R + row;
                    m2[j][k] = in_range ? __ldcg(P.part_m + at) : kNegSentinel;
                    l2[j][k] = in_range ? __ldcg(P.part_l + at) : 0.f;
                  }
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                  for (int k = 0; k < 4; ++k)
                    if (j0 + j < u.S) lse_merge(mv[k], lv[k], m2[j][k], l2[j][k]);
              }
            }
            double err_sum, msum;
            finalize_rows_warp(P, sp, u.parity, rbase, mv, lv, A.cfg.norm_error, sm.log2t, in,
                               err_sum, msum);
            if (sp.eval && lane == 0) {
              P.err_part[u.rb] = err_sum;
              P.msum_part[u.rb] = msum;
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sm.unit_empty[slot]);
      if (stop) break;
    }
    if (!handed && lane == 0) {
      sm.tail = 0;
      tc::mbar_arrive(&sm.tail_full);
    }
  } else if (warp < 2) {
    // producer (warp 0) and MMA issuer (warp 1)
    // the column shifts, which other CTAs wrote with plain stores in the last
    // sweep, before this one's TMA loads of them
    if (warp == 0) tc::fence_proxy_async_global();
    while (true) {
      const uint32_t d = pp.desc++;
      const uint32_t slot = d % NSLOT;
      bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&sm.unit_full[slot], (d / NSLOT) & 1, tmo));
      if (!ok) {
        if (lane == 0) atomicExch(&sm.err, 1);
        break;
      }
      // read in place: the dealer rewrites this slot only after this warp,
      // the other control warp and the finalizer have arrived on unit_empty
      const TcUnit& u = sm.units[slot];
      const bool stop = u.end != 0 || __any_sync(0xffffffffu, *err != 0);
      if (!stop) {
        const bool r = warp == 0 ? tc_produce<DK, TN>(sm, pp, u, tmo)
                                 : tc_mma<DK, TN>(sm, pp, u, tmo);
        ok = __all_sync(0xffffffffu, r);
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sm.unit_empty[slot]);
      if (stop || !ok) break;
    }
  } else {
    // epilogue warps, each on its own: reduce every unit's tiles into the
    // part buffers
    int at = -1;  // the last unit's slot, which the dealer leaves alone until the next sweep
    bool ended = false;
    while (true) {
      const uint32_t d = pp.desc++;
      const uint32_t slot = d % NSLOT;
      bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&sm.unit_full[slot], (d / NSLOT) & 1, tmo));
      if (!ok) {
        if (lane == 0) atomicExch(&sm.err, 1);
        break;
      }
      const TcUnit& u = sm.units[slot];
      if (u.end != 0 || __any_sync(0xffffffffu, *err != 0)) {
        ended = true;
        break;
      }
      if (!__all_sync(0xffffffffu, tc_epilogue<DK, TN>(sm, pp, u, tmo))) break;
      at = (int)slot;
    }
    // The sweep's tail: the last unit's row block, 32 rows a warp, a row a
    // lane. By the finalizer warp alone, four rows a lane, the splits' merge
    // and the update took 7.2k of the 41k cycles of a sweep at n = m = 4096
    // (d = 64: 1.74 -> 1.59 ms; 96 ragged problems, d = 32: 8.9 -> 8.4).
    const int q = warp - TcCfg<DK, TN>::kEpiWarp0;
    if (q < 4 && ended && at >= 0) {
      const TcUnit& u = sm.units[at];
      const ProbDev& P = prob(u.p);
      const int64_t row0 = (int64_t)u.rb * kBM + 32 * q;
      RowInputs<1> in;
      load_row_inputs(P, sp, u.parity, row0, sm.log2t, in);
      if (!__all_sync(0xffffffffu, tc::mbar_wait(&sm.tail_full, pp.sweeps & 1, tmo))) {
        if (lane == 0) atomicExch(&sm.err, 1);
      } else if (sm.tail) {
        float mv[1] = {kNegSentinel}, lv[1] = {0.f};
        if (u.S > 1) {
          const int64_t R = sp.kind == kSweepG ? P.m : P.n;
          const int64_t row = row0 + lane;
          constexpr int U = 8;  // splits in flight
          for (int j0 = 0; j0 < u.S; j0 += U) {
            float m2[U], l2[U];
#pragma unroll
            for (int j = 0; j < U; ++j) {
              const bool in_range = j0 + j < u.S && row < R;
              const int64_t a = (int64_t)(j0 + j) * R + row;
              m2[j] = in_range ? __ldcg(P.part_m + a) : kNegSentinel;
              l2[j] = in_range ? __ldcg(P.part_l + a) : 0.f;
            }
#pragma unroll
            for (int j = 0; j < U; ++j)
              if (j0 + j < u.S) lse_merge(mv[0], lv[0], m2[j], l2[j]);
          }
        } else {
          const uint32_t pb = (pp.unit - 1) & 1;
          const int r = 32 * q + lane;
          mv[0] = sm.part_m[pb][0][r];
          lv[0] = sm.part_l[pb][0][r];
#pragma unroll
          for (int c = 1; c < CG; ++c)
            lse_merge(mv[0], lv[0], sm.part_m[pb][c][r], sm.part_l[pb][c][r]);
        }
        double err_sum, msum;
        finalize_rows_warp(P, sp, u.parity, row0, mv, lv, A.cfg.norm_error, sm.log2t, in,
                           err_sum, msum);
        if (lane == 0) {
          sm.tail_red[q][0] = err_sum;
          sm.tail_red[q][1] = msum;
        }
      }
    }
    tail_at = q == 0 && ended ? at : -1;
  }
  ++pp.sweeps;
  __syncthreads();
  if (tail_at >= 0 && lane == 0 && sp.eval && sm.tail && *err == 0) {
    const TcUnit& u = sm.units[tail_at];
    const ProbDev& P = prob(u.p);
    double e = 0.0, t = 0.0;
    for (int k = 0; k < 4; ++k) {
      e += sm.tail_red[k][0];
      t += sm.tail_red[k][1];
    }
    P.err_part[u.rb] = e;
    P.msum_part[u.rb] = t;
  }
  return *err == 0;
}

template <int DK, int TN>
__global__ void __launch_bounds__(TcCfg<DK, TN>::kThreads, 1)
sinkhorn_tc_kernel(KernelArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // The 128-byte swizzled operand tiles need 1024-byte alignment.
  const uint32_t base = tc::smem_u32(smem_raw);
  unsigned char* aligned = smem_raw + ((1024u - (base & 1023u)) & 1023u);
  TcSmem<DK, TN>& sm = *reinterpret_cast<TcSmem<DK, TN>*>(aligned);
  constexpr int NS = TcCfg<DK, TN>::kStages;
  constexpr int NB = TcCfg<DK, TN>::kTmemBufs;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    constexpr int NE = TcCfg<DK, TN>::kEpiWarps;
    for (int i = 0; i < NS; ++i) {
      tc::mbar_init(&sm.full[i], 1);   // producer arrival + TMA bytes
      tc::mbar_init(&sm.empty[i], 1);  // MMA commit
    }
    for (int i = 0; i < NB; ++i) {
      tc::mbar_init(&sm.tfull[i], 1);
      tc::mbar_init(&sm.tempty[i], NE);
    }
    tc::mbar_init(&sm.a_full, 1);
    tc::mbar_init(&sm.a_empty, 1);
    tc::mbar_init(&sm.drain, 1);
    for (int i = 0; i < TcCfg<DK, TN>::kDescSlots; ++i) {
      tc::mbar_init(&sm.unit_full[i], 1);   // the dealer
      tc::mbar_init(&sm.unit_empty[i], 3);  // producer, MMA and finalizer warps
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&sm.epi_done[i], NE);   // one arrival per epilogue warp
      tc::mbar_init(&sm.part_free[i], 1);   // the finalizer
    }
    tc::mbar_init(&sm.tail_full, 1);        // the finalizer
    sm.err = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(&sm.tmem_base, TcCfg<DK, TN>::kTmemCols);
    tc::tmem_relinquish();
  }
  log2_table_fill(sm.log2t);
  if (A.num_problems <= TcCfg<DK, TN>::kProbSlots) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(A.probs);
    uint32_t* dst = reinterpret_cast<uint32_t*>(sm.probs);
    for (int i = threadIdx.x; i < A.num_problems * (int)(sizeof(ProbDev) / 4); i += blockDim.x)
      dst[i] = src[i];
  }
  // Extension blocks: zero everywhere; A's first 3 K columns are ones.
  {
    uint32_t* a32 = reinterpret_cast<uint32_t*>(sm.Aext);
    for (int i = threadIdx.x; i < TcCfg<DK, TN>::kAExtBytes / 4; i += blockDim.x) a32[i] = 0u;
    for (int st = 0; st < NS; ++st) {
      uint32_t* b32 = reinterpret_cast<uint32_t*>(sm.Bext[st]);
      for (int i = threadIdx.x; i < TcCfg<DK, TN>::kBExtBytes / 4; i += blockDim.x) b32[i] = 0u;
    }
    __syncthreads();
    if (threadIdx.x < kBM) {
      const __nv_bfloat16 one = __float2bfloat16_rn(1.f);
      for (int k = 0; k < 3; ++k)
        reinterpret_cast<__nv_bfloat16*>(sm.Aext + threadIdx.x * 16)[k] = one;
    }
    tc::fence_proxy_async_smem();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();

  TcPipe pp{0u, 0u, 0u, 0u, 0u, 0, 0u, 0u, 0u};
  auto sweep = [&](const SweepParams& sp, unsigned idx) -> bool {
    return tc_sweep<DK, TN>(A, sp, idx, sm, pp);
  };
  persistent_main(A, sweep);

  // Teardown. After a timeout, wait (bounded) for this CTA's own MMAs and
  // TMA loads still in flight before the TMEM and shared memory go away.
  __syncthreads();
  if (sm.err) {
    const uint64_t limit = 1000000000ull;  // 1 s
    if (warp == 1 && lane == 0) {
      tc::mma_commit(&sm.drain);
      tc::mbar_wait(&sm.drain, 0, limit);
    }
    if (warp == 0 && lane == 0 && pp.issued)
      tc::mbar_wait(&sm.full[pp.last_full_stage], pp.last_full_parity, limit);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 1) tc::tmem_dealloc(sm.tmem_base, TcCfg<DK, TN>::kTmemCols);
}

}  // namespace ottb
