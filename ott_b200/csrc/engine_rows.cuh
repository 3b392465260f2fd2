// FP32 row-owner engine: the whole fixed-point loop of a problem run by a
// team of CTAs, each of which owns whole rows of both sweeps.
//
// A CTA that owns a row reduces it over every column, so a sweep has no
// partial results that travel between CTAs and one barrier: new potentials
// out, barrier, next sweep. (The tiled engine of engine_simt.cuh splits a
// row block over CTAs, and at n = m = 2048 spent 4/5 of a sweep dealing
// units, merging splits and waiting for the CTA that merges.)
//
// Teams. A small problem is solved by one CTA or one thread-block cluster:
// both point sets, their norms and every potential stay in shared memory, a
// new potential is written straight into the shared memory of every CTA of
// the cluster, and the barrier is the cluster's. Clusters take problems from
// a queue and never wait for one another, so a batch has no sweep-wide
// barriers. A larger problem is solved by the whole grid: potentials go
// through global memory, the barrier is grid_barrier. Both point sets stay in
// shared memory where they fit; where only one fits they take turns in one
// buffer: the points never change, so the next sweep's are on their way (bulk
// copies by one thread) during the row updates and the barrier. Larger sets
// are streamed from L2 in chunks (cp.async, double-buffered), whose waits and
// part-filled tiles cost a sweep of n = 3000, m = 4100, d = 10 51.7k cycles
// against 39.2k in turns.
//
// Inside a CTA each warp takes 1/W of the columns for all of the CTA's
// rows. Rows are covered by tiles of 4 RS rows (RS = 1 ... 32): lane =
// (phase, slot), slot's 4 consecutive rows stay in registers with their
// running (shift, sum), the 32 / RS phases take alternate groups of 4
// columns, read from shared memory as 16-byte broadcasts. So a row's sum is
// thread-local until the end of the tile: no shared-memory product tile, no
// barrier inside a sweep's columns. Per entry D + 1 FMA (packed pairs of
// columns), the subtraction of the shift, ex2, and sums in
// chunks of 8 with TwoSum, as in the tiled engine. The shift is a running
// maximum or, once a sweep of the kind has run, the tensor-core engine's
// bound (engine_tc.cuh): row log-sum-exp of the last sweep + largest change
// of a column shift, which takes the maxima and the branch out of the loop.
//
// What bounds it, and what it measured (B200, solve to 1e-3; the tiled
// engine before): a sweep's chain of latencies for small problems (n = 120,
// m = 96, d = 3: 1.18 -> 0.59 ms; n = m = 2048, d = 2: 1.53 -> 0.78), the
// FMA pipe, the MUFU and the issue slots about equally for large ones (n =
// 7013, m = 5001, d = 3: 11.3 -> 5.5 ms), the FMA pipe for d > 4 (n = 3000,
// m = 4100, d = 10: 1.52 -> 0.84). 256 problems of 1024 x 1024, d = 2, in
// one call: 47 -> 29 ms.
#pragma once

#include "common.cuh"
#include "driver.cuh"
#include "rows.h"
#include "tc_ptx.cuh"

namespace ottb {

__device__ __forceinline__ void word_store(unsigned long long* p, float v, unsigned seq) {
  const unsigned long long w = ((unsigned long long)seq << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long word_load(const unsigned long long* p) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}

// Cover of Q quads of rows by tiles of RS = 1 << b quads: nfull tiles of
// 1 << big, then one tile per set bit of rest (highest first).
struct RowsCover {
  int big, nfull, rest;
};

// The cover of Q quads for column segments of gseg groups (taken NG at a
// time) with the fewest iterations: full tiles of the best size, the rest
// by one tile that holds it or by its binary digits.
__device__ inline RowsCover rows_cover(int Q, int gseg, int NG) {
  // iterations of a tile with 2^b slots (each: 4 NG columns of 4 rows a
  // lane), and about one and a half for its row loads and lane merges
  const int ng = NG == 2 ? 1 : 0;
  auto cost = [&](int b) {
    const int per = ng + 5 - b;  // log2 of the groups of one iteration
    return 4 * ((gseg + (1 << per) - 1) >> per) + 6 + (5 - b);
  };
  RowsCover best{5, 0, 0};
  int bc = 0x7fffffff;
  for (int b = 5; b >= 0; --b) {
    const int nf = Q >> b, rem = Q - (nf << b);
    int c = nf * cost(b), rest = rem;
    if (rem) {
      int bin = 0;
      for (int k = 0; k < 5; ++k)
        if (rem >> k & 1) bin += cost(k);
      const int up = rem > 1 ? 32 - __clz(rem - 1) : 0;
      const int one = cost(up);
      if (one <= bin) rest = 1 << up;
      c += one < bin ? one : bin;
    }
    if (c < bc) {
      bc = c;
      best = RowsCover{b, nf, rest};
    }
  }
  return best;
}

// The CTA's dynamic shared memory. File scope, and offsets instead of
// pointers below: a pointer that crosses a call would be a generic one, and
// its loads generic loads (in the inner loop, half the kernel's time).
extern __shared__ __align__(16) float rows_mem[];

// Iterations of a cover.
__device__ inline int rows_iters(RowsCover c, int gseg, int NG) {
  auto iters = [&](int b) {
    const int per = (NG == 2 ? 1 : 0) + 5 - b;
    return (gseg + (1 << per) - 1) >> per;
  };
  int n = c.nfull * iters(c.big);
  for (int b = 0; b <= 5; ++b)
    if (c.rest >> b & 1) n += iters(b);
  return n;
}

// The bounded shift of a row: every exponent of the row is at most this. A
// row without a finite log-sum-exp has no finite term either; one at -inf
// gets the running maximum's mark of a row without a term, by which
// update_row knows it (exp2_poly2 turns its terms into 2^-126, not 0).
__device__ __forceinline__ float row_sigma(float lprev, float dmax) {
  return isfinite(lprev) ? lprev + dmax : lprev == -INFINITY ? kNegSentinel : 0.f;
}

// One warp's share of a sweep over the columns in shared memory: rows
// [arow, arow + 4 Q) of A against column groups [g0, g1) of 4 columns
// (points [D][stride] at pts, shifts at w, group gpad of them -inf). A is
// in shared memory at aoff, or in global memory at ag where that is not
// null. The rows' base-2 (shift, sum) go to pm / pl (this warp's slice),
// merged with what is there unless first. Offsets are into rows_mem.
//
// BOUND: every exponent of row r is at most its shift sigma_r = (row r's
// log-sum-exp of its last sweep, at lp) + dmax (RowsShared::dmax): no
// maxima, no rescaling and no branch in the loop, only sums (pm unused).
template <int D, bool BOUND>
__device__ __noinline__ void rows_warp(int pts, int stride, int w, int g0, int g1, int gpad,
                                       int aoff, const float* ag, int64_t a_stride, int64_t arow,
                                       int64_t a_last, int Q, RowsCover cov, float s, int pm,
                                       int pl, bool first, int lp, float dmax) {
  constexpr int NG = rows_groups(D);   // column groups per iteration
  constexpr int NP = 2 * NG;           // column pairs per iteration
  const int lane = threadIdx.x & 31;
  const f32x2 s2 = pack2(s, s);
  int q0 = 0, nf = cov.nfull, rest = cov.rest;
  while ((nf > 0 || rest) && q0 < Q) {
    int b = cov.big;
    if (nf > 0) {
      --nf;
    } else {
      b = 31 - __clz(rest);
      rest &= ~(1 << b);
    }
    const int slot = lane & ((1 << b) - 1), ph = lane >> b, P = 32 >> b;
    float a[4][D];
    {
      int64_t row = arow + 4 * (int64_t)(q0 + slot);
      if (row > a_last) row = a_last;  // tile rows past the CTA's: any readable quad
#pragma unroll
      for (int k = 0; k < D; ++k) {
        const float4 v = ag ? *reinterpret_cast<const float4*>(ag + k * a_stride + row)
                            : *reinterpret_cast<const float4*>(rows_mem + aoff + k * (int)a_stride + (int)row);
        a[0][k] = v.x; a[1][k] = v.y; a[2][k] = v.z; a[3][k] = v.w;
      }
    }
    float m[4];
    f32x2 l[2], lc[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) m[i] = kNegSentinel;
    if constexpr (BOUND) {
      // a tile's slots past the CTA's rows: any kept values
      const float4 v = *reinterpret_cast<const float4*>(rows_mem + lp + 4 * min(q0 + slot, Q - 1));
      m[0] = row_sigma(v.x, dmax); m[1] = row_sigma(v.y, dmax);
      m[2] = row_sigma(v.z, dmax); m[3] = row_sigma(v.w, dmax);
    }
    l[0] = l[1] = lc[0] = lc[1] = pack2(0.f, 0.f);

    for (int g = g0 + ph; g < g1; g += NG * P) {
      f32x2 t[4][NP];
      f32x2 wp[NP];
      int gg[NG];
#pragma unroll
      for (int h = 0; h < NG; ++h) {
        gg[h] = g + h * P;
        int gw = gg[h];
        if (h > 0 && gg[h] >= g1) {
          gg[h] = g;
          gw = gpad;
        }
        const float4 v = *reinterpret_cast<const float4*>(rows_mem + w + 4 * gw);
        wp[2 * h] = pack2(v.x, v.y);
        wp[2 * h + 1] = pack2(v.z, v.w);
      }
      // t = s <a, b> + w: the inner product first, one rounding for the
      // scale and the shift (seeding the chain with w would round every
      // step at |w|)
#pragma unroll
      for (int k = 0; k < D; ++k) {
        f32x2 bp[NP];
#pragma unroll
        for (int h = 0; h < NG; ++h) {
          const float4 v = *reinterpret_cast<const float4*>(rows_mem + pts + k * stride + 4 * gg[h]);
          bp[2 * h] = pack2(v.x, v.y);
          bp[2 * h + 1] = pack2(v.z, v.w);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const f32x2 ad = pack2(a[i][k], a[i][k]);
#pragma unroll
          for (int j = 0; j < NP; ++j)
            t[i][j] = k == 0 ? mul2(ad, bp[j]) : fma2(ad, bp[j], t[i][j]);
        }
      }
      if constexpr (BOUND) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < NP; ++j) t[i][j] = fma2(t[i][j], s2, wp[j]);
      } else {
        float cm[4];
        bool up = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float v[2 * NP];
#pragma unroll
          for (int j = 0; j < NP; ++j) {
            t[i][j] = fma2(t[i][j], s2, wp[j]);
            unpack2(t[i][j], v[2 * j], v[2 * j + 1]);
          }
          cm[i] = fmaxf(fmax3(v[0], v[1], v[2]), v[3]);
          if constexpr (NG == 2) cm[i] = fmax3(fmax3(cm[i], v[4], v[5]), v[6], v[7]);
          up |= cm[i] > m[i] + kTau;
        }
        if (up) {
          float sc[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            sc[i] = 1.f;
            if (cm[i] > m[i] + kTau) {
              sc[i] = ex2_approx(m[i] - cm[i]);
              m[i] = cm[i];
            }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const f32x2 sp = pack2(sc[2 * h], sc[2 * h + 1]);
            l[h] = mul2(l[h], sp);
            lc[h] = mul2(lc[h], sp);
          }
        }
      }
      float sum[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const f32x2 nm = pack2(-m[i], -m[i]);
        f32x2 e[NP];
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          const f32x2 x = add2(t[i][j], nm);
          // where the MUFU binds, a part of the exponentials on the FMA pipe
          if (j == NP - 1 && i < rows_poly_pairs(D)) {
            e[j] = exp2_poly2(x);
          } else {
            float x0, x1;
            unpack2(x, x0, x1);
            e[j] = pack2(ex2_approx(x0), ex2_approx(x1));
          }
        }
        f32x2 es = add2(e[0], e[1]);
        if constexpr (NG == 2) es = add2(es, add2(e[2], e[3]));
        float e0, e1;
        unpack2(es, e0, e1);
        sum[i] = e0 + e1;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // two_sum_acc on a pair of rows
        const f32x2 x = pack2(sum[2 * h], sum[2 * h + 1]);
        const f32x2 tt = add2(l[h], x);
        const f32x2 bb = sub2(tt, l[h]);
        const f32x2 err = add2(sub2(l[h], sub2(tt, bb)), sub2(x, bb));
        l[h] = tt;
        lc[h] = add2(lc[h], err);
      }
    }

    // merge the phases of each row, then store (or merge into) the slice
    float lv[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) unpack2(add2(l[h], lc[h]), lv[2 * h], lv[2 * h + 1]);
    if (b < 5) {
      if constexpr (!BOUND) {
        float mx[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) mx[i] = m[i];
        for (int off = 1 << b; off < 32; off <<= 1)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], off));
#pragma unroll
        for (int i = 0; i < 4; ++i) lv[i] *= ex2_approx(m[i] - mx[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) m[i] = mx[i];
      }
      for (int off = 1 << b; off < 32; off <<= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i) lv[i] += __shfl_xor_sync(0xffffffffu, lv[i], off);
    }
    if (ph == 0 && q0 + slot < Q) {
      float4* dm = reinterpret_cast<float4*>(rows_mem + pm + 4 * (q0 + slot));
      float4* dl = reinterpret_cast<float4*>(rows_mem + pl + 4 * (q0 + slot));
      if (!first) {
        const float4 ol = *dl;
        if constexpr (BOUND) {
          lv[0] += ol.x; lv[1] += ol.y; lv[2] += ol.z; lv[3] += ol.w;
        } else {
          const float4 om = *dm;
          lse_merge(m[0], lv[0], om.x, ol.x);
          lse_merge(m[1], lv[1], om.y, ol.y);
          lse_merge(m[2], lv[2], om.z, ol.z);
          lse_merge(m[3], lv[3], om.w, ol.w);
        }
      }
      if constexpr (!BOUND) *dm = make_float4(m[0], m[1], m[2], m[3]);
      *dl = make_float4(lv[0], lv[1], lv[2], lv[3]);
    }
    q0 += 1 << b;
  }
}

// ---------------------------------------------------------------- cluster
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Barrier over the cluster's threads (the CTA's for a cluster of one),
// ordering their shared-memory and global accesses.
__device__ __forceinline__ void cluster_barrier(int size) {
  if (size == 1) {
    __syncthreads();
    return;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of a shared-memory variable in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, unsigned rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t addr, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Remote store that signals its bytes on the receiving CTA's mbarrier.
__device__ __forceinline__ void cluster_store_async(uint32_t addr, float v, uint32_t bar) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
      "r"(__float_as_uint(v)), "r"(bar)
      : "memory");
}
// Waits (bounded) for the phase of a barrier that cluster_store_async signals.
__device__ __forceinline__ bool cluster_wait(uint64_t* bar, uint32_t parity, uint64_t timeout_ns) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(bar);
  auto done = [&]() {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0;
  };
  if (done()) return true;
  const uint64_t t0 = global_timer_ns();
  while (!done())
    if (global_timer_ns() - t0 > timeout_ns) return false;
  return true;
}

// What a sweep needs, written by one thread for the whole CTA: the sweep's
// code then keeps nothing in registers over rows_warp, which uses them all
// (spilled state was reloaded through an L1 that every acquire empties).
struct RowsCmd {
  int kind, eval, write, fin, parity, done;
  int colx;       // the columns' values: x's (1) or g buffer `parity` (0)
  int arrive;     // cluster: wait for them on sh.bar[colx ? 0 : 1 + parity]
  unsigned phase; // ... its phase parity
  unsigned want;  // grid: number of the sweep that wrote them (0: the initial ones)
  unsigned seq;   // this sweep's number
  int change;     // 1: the columns' values changed since the kind's last sweep; 0: they did not;
                  // -1: not known (no last sweep at this multiplier)
  float mult, ws, s;
  double eps, epsln2;
};

// The loop's state between sweeps.
struct RowsState {
  int next, it, commits, fpar;
  int fused, may_continue, need_err;
  unsigned seq, seq_of[3];  // sweep that last wrote x's values, g buffer 0's and 1's
  unsigned last[2];         // per sweep kind: its last sweep, if at multiplier 1 (else 0)
  unsigned pending, phases; // cluster, bit k of sh.bar[k]: written and not yet awaited; phase parity
};

struct RowsShared {
  RowsArgs A;
  ProbDev P;
  RowsLayout L;
  GridBarrier bar_grid;
  int rank, size;  // this CTA in its team
  Log2Table log2t;
  RowsCmd cmd[2];
  RowsState st;
  RowsCover cover[2];    // per sweep kind
  int iters[2];          // ... and its iterations per warp
  int row0[2], row1[2];  // this CTA's rows, per sweep kind
  unsigned owners[2];    // cluster, per sweep kind: bit q, CTA q owns rows of it
  unsigned awaits;       // cluster, bit k of bar[k]: this CTA is sent those values
  int partial;           // a CTA of the team owns no rows of one sweep kind
  int resync;            // see sums
  double red[2][kRowsWarps];
  double slot[2][kRowsMaxCluster];  // cluster: each CTA's error and marginal sums
  double err, msum;
  double eps;       // update_epsilon at multiplier 1
  uint64_t bar[3];  // cluster: the values of x and of both g buffers have arrived; in turns,
                    // bar[0]: the points of pts_side have
  int pts_side;     // in turns: 0 x, 1 y, -1 neither
  unsigned pts_loads;  // ... loads so far
  int q;
  int fail;  // a wait ran out
  int key[2][2];  // resident: largest and smallest change of a column shift, by sweep parity
  float dmax[2];  // per sweep kind: the bound of the last sweep's shifts
  int bound[2];   // ... and whether it was in use
};

// File scope: the functions below reach them without a pointer in registers
// (or, over calls, in local memory).
static __shared__ RowsShared rows_sh;

// The loop of one problem by this CTA's team; every member takes the same
// decisions from the same values.
template <int D, bool GRID>
struct RowsSolver {
  enum { kInitF, kBlock, kG, kF, kFinal, kDone };

  static __device__ __forceinline__ bool resident() { return !GRID || rows_sh.A.resident; }
  static __device__ __forceinline__ bool turns() { return GRID && rows_sh.A.turns; }
  // the epsilon multiplier is 1 throughout: the team exchanges column shifts
  // instead of potentials
  static __device__ __forceinline__ bool constant() {
    return rows_sh.A.cfg.eps_decay == 1.0f && rows_sh.A.cfg.eps_init <= 1.0f;
  }
  // the thread that runs the loop's control: not one of the few that update
  // rows in small problems
  static __device__ __forceinline__ bool control() { return threadIdx.x == blockDim.x - 1; }

  // Whether this CTA owns rows of a sweep of `kind`. One that owns none (a
  // side with fewer quads of rows than the team has CTAs) reads none of that
  // sweep's values and is sent none: whoever reads a sweep's values publishes
  // in that sweep, on which the exchange without barriers rests (rows.h).
  static __device__ __forceinline__ bool has_rows(int kind) {
    return rows_sh.row1[kind] > rows_sh.row0[kind];
  }

  static __device__ __noinline__ void begin() {
    const ProbDev& P = rows_sh.P;
    const int W = blockDim.x >> 5, wsh = 31 - __clz(W);
    const bool res = resident();
    if (threadIdx.x == 0) {
      rows_sh.L = rows_layout(P.n, P.m, D, rows_sh.size, W, !GRID, res, turns());
      rows_sh.eps = update_epsilon(P.ws_t);
    }
    if (threadIdx.x < 2) {
      const int64_t rows = threadIdx.x == kSweepG ? P.m : P.n;
      rows_sh.row0[threadIdx.x] = (int)rows_begin(rows, rows_sh.rank, rows_sh.size);
      rows_sh.row1[threadIdx.x] = (int)rows_begin(rows, rows_sh.rank + 1, rows_sh.size);
    }
    __syncthreads();
    const RowsLayout& L = rows_sh.L;
    if (threadIdx.x < 2) {
      const int kind = threadIdx.x;
      const int cols = kind == kSweepG ? L.n4 : L.m4;
      const int G = (res ? cols : chunk_cols(cols)) / 4;
      rows_sh.cover[kind] = rows_cover((min(rows_sh.row1[kind] - rows_sh.row0[kind], L.rp) + 3) / 4,
                                  (G + W - 1) >> wsh, rows_groups(D));
      rows_sh.iters[kind] = rows_iters(rows_sh.cover[kind], (G + W - 1) >> wsh, rows_groups(D));
    }
    if (threadIdx.x < 2) rows_sh.bound[threadIdx.x] = 0;
    // A side with fewer quads of rows than the team has CTAs leaves some
    // without rows.
    const bool partial = (min(P.n, P.m) + 3) / 4 < rows_sh.size;
    if (threadIdx.x == 0) {
      rows_sh.partial = partial;
      rows_sh.resync = partial || (P.symmetric && rows_sh.A.cfg.inner_iterations == 1);
      // x's values are read by g-sweeps, y's by f-sweeps (in a symmetric
      // problem, where every CTA owns the same rows of both, by g-sweeps)
      rows_sh.awaits =
          rows_sh.size == 1 ? 0u : (has_rows(kSweepG) ? 1u : 0u) | (has_rows(kSweepF) ? 6u : 0u);
    }
    // (by a loop: a ballot here, executed or not, cost the sweeps of 256
    // problems of 1024 points 2 %)
    if (!GRID && partial && threadIdx.x < 2) {
      const int64_t rows = threadIdx.x == kSweepG ? P.m : P.n;
      unsigned mask = 0;
      for (int q = 0; q < rows_sh.size; ++q)
        if (rows_begin(rows, q, rows_sh.size) < rows_begin(rows, q + 1, rows_sh.size)) mask |= 1u << q;
      rows_sh.owners[threadIdx.x] = mask;
    }
    const int x0 = rows_sh.row0[kSweepF], x1 = rows_sh.row1[kSweepF];
    const int y0 = rows_sh.row0[kSweepG], y1 = rows_sh.row1[kSweepG];
    const int t = threadIdx.x, nt = blockDim.x;
    auto fill = [&](int dst, const float* src, int64_t pad, int c4, int rows) {
      for (int k = 0; k < rows; ++k)
        for (int i = t; i < c4 / 4; i += nt)
          reinterpret_cast<float4*>(rows_mem + dst + (size_t)k * c4)[i] =
              reinterpret_cast<const float4*>(src + k * pad)[i];
    };
    if (res && !turns()) {
      fill(L.cx, P.xt, P.n_pad, L.n4, D);
      fill(L.cy, P.yt, P.m_pad, L.m4, D);
      if (!GRID) {
        fill(L.nx, P.nx, 0, L.n4, 1);
        fill(L.ny, P.ny, 0, L.m4, 1);
      }
    }
    if (GRID && L.own) {
      for (int i = t; i < x1 - x0; i += nt) rows_mem[L.anx + i] = P.nx[x0 + i];
      for (int i = t; i < y1 - y0; i += nt) rows_mem[L.any + i] = P.ny[y0 + i];
    }
    if ((!res || turns()) && L.own) {
      // whole quads: the last own quad may reach into the padding
      if (x1 > x0) {
        for (int k = 0; k < D; ++k)
          for (int i = t; i < (x1 - x0 + 3) / 4; i += nt)
            reinterpret_cast<float4*>(rows_mem + L.ax + k * L.rf)[i] =
                reinterpret_cast<const float4*>(P.xt + k * P.n_pad + x0)[i];
      }
      if (y1 > y0) {
        for (int k = 0; k < D; ++k)
          for (int i = t; i < (y1 - y0 + 3) / 4; i += nt)
            reinterpret_cast<float4*>(rows_mem + L.ay + k * L.rg)[i] =
                reinterpret_cast<const float4*>(P.yt + k * P.m_pad + y0)[i];
      }
    }
    // the column shifts' padding (rows_warp's gpad group too)
    const float ninf = -INFINITY;
    if (GRID && !res && t < 8) rows_mem[L.w + (t >> 2) * L.wstride + rows_chunk(D) + (t & 3)] = ninf;
    if (!GRID) {
      const bool cw = constant();
      for (int i = t; i < L.n4 + 4; i += nt)
        rows_mem[L.vx + i] = i < (int)P.n ? (cw ? (P.f[i] - P.nx[i]) * P.ws_t : P.f[i]) : ninf;
      for (int i = t; i < L.m4 + 4; i += nt) {
        rows_mem[L.vy + i] =
            i < (int)P.m ? (cw ? (P.gbuf[0][i] - P.ny[i]) * P.ws_t : P.gbuf[0][i]) : ninf;
        rows_mem[L.vy + L.m4 + 4 + i] = ninf;
      }
    }
    if (L.own) {
      for (int i = t; i < x1 - x0; i += nt) rows_mem[L.px + i] = P.f[x0 + i];
      for (int i = t; i < y1 - y0; i += nt) rows_mem[L.py + i] = P.gbuf[0][y0 + i];
      double* lg = reinterpret_cast<double*>(rows_mem + L.logm);
      for (int i = t; i < x1 - x0; i += nt) lg[i] = log((double)P.a[x0 + i]);
      for (int i = t; i < y1 - y0; i += nt) lg[L.rf + i] = log((double)P.b[y0 + i]);
    }
    // what another layout kept in the points' buffer is behind its first load
    if (turns()) tc::fence_proxy_async_smem();
    __syncthreads();
  }

  // In turns: brings the points of the columns of a sweep of `kind` into the
  // buffer, unless they are there (or on their way). By one thread, once no
  // thread reads the buffer; sweeps wait for it in points_arrived.
  static __device__ __noinline__ void load_points(int kind) {
    const ProbDev& P = rows_sh.P;
    const bool isG = kind == kSweepG;
    if (rows_sh.pts_side == (isG ? 0 : 1)) return;
    rows_sh.pts_side = isG ? 0 : 1;
    ++rows_sh.pts_loads;
    const int c4 = isG ? rows_sh.L.n4 : rows_sh.L.m4;
    const float* src = isG ? P.xt : P.yt;
    const int64_t pad = isG ? P.n_pad : P.m_pad;
    tc::mbar_arrive_expect_tx(&rows_sh.bar[0], 4u * (unsigned)(D * c4));
    // each CTA starts at another coordinate (see columns)
    int k = rows_sh.rank % D;
    for (int i = 0; i < D; ++i) {
      tc::bulk_load(rows_mem + rows_sh.L.cx + k * c4, src + k * pad, 4u * (unsigned)c4,
                    &rows_sh.bar[0]);
      k = k + 1 < D ? k + 1 : 0;
    }
  }
  // Waits for the last load's points (also when nobody reads them: a CTA
  // does not leave while one is in flight).
  static __device__ __forceinline__ void points_arrived() {
    const unsigned loads = rows_sh.pts_loads;
    if (loads == 0) return;
    if (!tc::mbar_wait(&rows_sh.bar[0], (loads - 1) & 1, rows_sh.A.timeout_ns)) {
      grid_abort(rows_sh.A.gl, &rows_sh.A.sched->status);
      rows_sh.fail = 1;
    }
  }

  // persistent_main's loop (fixed_point_loop.py:23-93) as a step between
  // sweeps: from the sweep that just ran (an evaluating one's sums in err,
  // msum) to the next one's command. One thread runs it, beside the others'
  // row updates where the sweep evaluates nothing.
  static __device__ __noinline__ void advance(int slot, bool start, double err, double msum) {
    RowsCmd& cmd = rows_sh.cmd[slot];
    const ottb_solver_cfg& c = rows_sh.A.cfg;
    const ProbDev& P = rows_sh.P;
    RowsState& S = rows_sh.st;
    const int inner = c.inner_iterations;
    const bool force_scan = c.min_iterations == c.max_iterations;
    const int scan_end = force_scan ? (c.max_iterations / inner) * inner : c.max_iterations;
    // the top of an iteration: the block test first where one is due
    auto top = [&]() {
      S.fused = 0;
      if (S.it > 0 && S.it % inner == 0) {
        const int last = S.it - 1;
        S.need_err = (last == c.max_iterations - 1) || (last >= c.min_iterations);
        S.may_continue = S.it < scan_end;
        S.fused = S.need_err && S.may_continue && eps_mult(c, S.it) == 1.0f;
        return (int)kBlock;
      }
      return (int)(S.it == 0 && scan_end == 0 ? kFinal : kG);
    };
    auto after_g = [&]() {
      ++S.commits;
      if (!P.symmetric) return (int)kF;
      ++S.it;
      return top();
    };
    auto block = [&](double e) {
      if (S.need_err) {
        if (c.norm_error != 1) e = pow(e, 1.0 / (double)c.norm_error);
        // parallel updates: the error of both marginals, equal here
        if (P.symmetric) e *= 2.0;
      }
      const float errf = (float)e;
      if (rows_sh.rank == 0) P.errors[(S.it - 1) / inner] = errf;
      bool cont;
      if (force_scan) {
        cont = S.may_continue;
      } else {
        // sinkhorn.py:940-953 inside fixed_point_loop.py:63-70
        const bool converged = errf < c.threshold;
        const bool diverged = !isfinite(errf);
        cont = S.may_continue && ((S.it < c.min_iterations) || (!diverged && !converged));
      }
      if (cont) return S.fused ? after_g() : (int)kG;
      S.fpar = S.commits & 1;
      // a state without a marginal sum gets one: reg_ot_cost needs it
      return (int)(S.need_err ? kDone : kFinal);
    };
    int next;
    if (start) {
      const unsigned phases = S.phases;
      S = RowsState{};
      S.phases = phases;
      rows_sh.pts_side = -1;
      next = c.init_f_from_g && scan_end > 0 && !P.symmetric ? (int)kInitF : top();
    } else if (S.next == kBlock) {
      next = block(err);
    } else if (S.next == kG) {
      next = after_g();
    } else if (S.next == kF) {
      ++S.it;
      next = top();
    } else if (S.next == kInitF) {
      next = top();
    } else {
      next = kDone;
    }
    // a block whose error is not asked for needs no sweep
    while (next == kBlock && !S.need_err) next = block(INFINITY);
    S.next = next;
    rows_sh.msum = msum;
    cmd.done = next == kDone;
    if (next == kDone) return;
    const bool eval = next == kBlock || next == kFinal;
    const bool isf = next == kF || next == kInitF;
    const float mult = eval ? 1.0f : eps_mult(c, S.it);  // a fused block's is 1
    cmd.kind = isf ? kSweepF : kSweepG;
    cmd.eval = eval;
    cmd.write = next == kBlock ? S.fused : !eval;
    cmd.fin = next == kFinal;
    cmd.parity = next == kInitF ? 0 : next == kFinal ? S.fpar : S.commits & 1;
    cmd.colx = !isf && !P.symmetric;
    const int k = cmd.colx ? 0 : 1 + cmd.parity;
    cmd.want = S.seq_of[k];
    cmd.arrive = S.pending >> k & 1;
    cmd.phase = S.phases >> k & 1;
    if (cmd.arrive) {
      S.pending ^= 1u << k;
      S.phases ^= 1u << k;
    }
    cmd.seq = ++S.seq;
    // In a symmetric problem the kind's last sweep has itself written the
    // columns of this one (want == last).
    cmd.change = mult != 1.0f || S.last[cmd.kind] == 0 ? -1 : cmd.want >= S.last[cmd.kind] ? 1 : 0;
    S.last[cmd.kind] = mult == 1.0f ? cmd.seq : 0;
    rows_sh.key[cmd.seq & 1][0] = kDkeyEmptyMax;
    rows_sh.key[cmd.seq & 1][1] = kDkeyEmptyMin;
    if (GRID && P.dkey && rows_sh.rank == 0) {
      // the next sweep's keys (the first one's are clear from the start): its
      // writers come behind the barrier that ends this sweep, before which
      // this is written. They were the keys of the sweep three before this
      // one, whose readers, in the sweep after it, have passed a barrier
      // since.
      P.dkey[2 * ((cmd.seq + 1) & 3)] = kDkeyEmptyMax;
      P.dkey[2 * ((cmd.seq + 1) & 3) + 1] = kDkeyEmptyMin;
    }
    if (cmd.write) {
      const int to = isf ? 0 : 1 + (cmd.parity ^ 1);
      S.seq_of[to] = cmd.seq;
      if (!GRID) S.pending |= 1u << to & rows_sh.awaits;
    }
    cmd.mult = mult;
    cmd.ws = mult == 1.0f ? P.ws_t : sweep_wscale(P, mult);
    cmd.s = 2.0f * P.inv_scale * cmd.ws;
    cmd.eps = mult == 1.0f ? rows_sh.eps : update_epsilon(cmd.ws);
    cmd.epsln2 = cmd.eps * kLn2;
    if (turns()) load_points(cmd.kind);
  }

  // ------------------------------------------------------------- columns
  // Cluster: waits for the values on rows_sh.bar[k]. After a wait ran out
  // (reported in the results) the loop goes on without waits: the CTAs stay
  // in step, so none leaves while another still writes into its shared
  // memory.
  static __device__ __forceinline__ void arrived(int k, unsigned phase) {
    if (threadIdx.x == 0)
      tc::mbar_arrive_expect_tx(&rows_sh.bar[k], 4u * (unsigned)(k == 0 ? rows_sh.P.n : rows_sh.P.m));
    if (!*(volatile int*)&rows_sh.fail && !cluster_wait(&rows_sh.bar[k], phase, rows_sh.A.timeout_ns)) {
      atomicExch(&rows_sh.A.sched->status, (int)OTTB_ERR_TIMEOUT);
      rows_sh.fail = 1;
    }
  }

  // Polls a word until its sweep number is `want`; after the time limit it
  // gives up (rows_sh.fail, and the grid's barrier is poisoned).
  static __device__ __noinline__ unsigned long long await(const unsigned long long* p, unsigned want) {
    unsigned long long w = word_load(p);
    const uint64_t t0 = global_timer_ns();
    for (int spin = 1; (unsigned)(w >> 32) != want; ++spin) {
      if ((spin & 63) == 0) {
        if (global_timer_ns() - t0 > rows_sh.A.timeout_ns) {
          grid_abort(rows_sh.A.gl, &rows_sh.A.sched->status);
          rows_sh.fail = 1;
          break;
        }
        if (*(volatile int*)&rows_sh.A.sched->status == OTTB_ERR_TIMEOUT) {
          rows_sh.fail = 1;
          break;
        }
      }
      w = word_load(p);
    }
    return w;
  }

  // The shifts of the U columns c[u] < C (grid team): from the initial
  // potentials, or from what the sweep `want` published, which is a shift or
  // a potential (constant()), as a word or, behind the barrier, a plain
  // value. Every load is in flight before the first is looked at.
  template <int U>
  static __device__ __forceinline__ void shifts(int slot, const int64_t (&c)[U], int64_t C,
                                                float (&v)[U]) {
    const RowsCmd& cmd = rows_sh.cmd[slot];
    const ProbDev& P = rows_sh.P;
    const float* nb = cmd.kind == kSweepG ? P.nx : P.ny;
    const int64_t off = cmd.colx ? 0 : P.n + cmd.parity * P.m;
    const bool own = cmd.want != 0 && P.words;
    if (own && rows_sh.A.seqwords) {
      unsigned long long w[U];
#pragma unroll
      for (int u = 0; u < U; ++u) w[u] = c[u] < C ? word_load(P.words + off + c[u]) : 0ull;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (c[u] < C && (unsigned)(w[u] >> 32) != cmd.want)
          w[u] = await(P.words + off + c[u], cmd.want);
        v[u] = __uint_as_float((unsigned)w[u]);
      }
    } else {
      const float* p = own ? reinterpret_cast<const float*>(P.words) + off
                           : cmd.colx ? P.f : P.gbuf[cmd.parity];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = c[u] < C ? __ldcg(p + c[u]) : 0.f;
    }
    if (own && constant()) return;
    float b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) b[u] = c[u] < C ? nb[c[u]] : 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = (v[u] - b[u]) * cmd.ws;
  }

  // Changes of column shifts, folded into [mx, mn].
  static __device__ __forceinline__ void fold_change(float now, float was, float& mx, float& mn) {
    if (isfinite(now) && isfinite(was)) {
      mx = fmaxf(mx, now - was);
      mn = fminf(mn, now - was);
    } else if (isfinite(now) != isfinite(was)) {
      // a value became or stopped being -inf: no bound
      mx = INFINITY;
      mn = -INFINITY;
    }
  }
  static __device__ __forceinline__ void publish_change(int* key, float mx, float mn) {
    const int kx = __reduce_max_sync(0xffffffffu, fkey(mx));
    const int kn = __reduce_min_sync(0xffffffffu, fkey(mn));
    if ((threadIdx.x & 31) == 0) {
      if (kx > kDkeyEmptyMax) atomicMax(key, kx);
      if (kn < kDkeyEmptyMin) atomicMin(key + 1, kn);
    }
  }
  // Whether this sweep's shifts are bounded, from the changes' keys: as the
  // tensor-core engine's bounded_row_shift.
  static __device__ __forceinline__ bool bounded(int change, int kmax, int kmin, float& dmax) {
    dmax = 0.f;
    if (change < 0) return false;
    if (change == 0 || kmax == kDkeyEmptyMax) return true;
    if (kmin == kDkeyEmptyMin) return false;
    dmax = fkey_value(kmax);
    return dmax - fkey_value(kmin) <= kMaxShiftSpread && isfinite(dmax);
  }
  // Resident sweeps with this much work per warp pay for the pass that
  // finds the bound.
  static __device__ __forceinline__ bool wants_bound(int kind) {
    if (!rows_sh.L.lx) return false;
    return GRID || rows_sh.iters[kind] >= 6;
  }

  // Resident columns: waits for their values and, where the cluster
  // exchanges potentials, the grid words, or a bound is wanted, turns them
  // into the side's shifts.
  static __device__ __noinline__ void columns(int slot) {
    const RowsCmd& cmd = rows_sh.cmd[slot];
    const RowsLayout& L = rows_sh.L;
    if (!GRID && cmd.arrive) arrived(cmd.colx ? 0 : 1 + cmd.parity, cmd.phase);
    const bool isG = cmd.kind == kSweepG, cw = constant();
    const bool find = wants_bound(cmd.kind);
    if (!GRID && cw && !find) return;
    const int C = (int)(isG ? rows_sh.P.n : rows_sh.P.m), c4 = isG ? L.n4 : L.m4;
    const float* nb = rows_mem + (isG ? L.nx : L.ny);
    const float* v = rows_mem + (cmd.colx ? L.vx : L.vy + cmd.parity * (L.m4 + 4));
    float* w = rows_mem + (isG ? L.wx : L.wy);
    const bool changes = find && cmd.change > 0;
    float mx = -INFINITY, mn = INFINITY;
    // Every CTA of the grid reads every value: each starts at another place,
    // so that they do not all ask one L2 slice at a time.
    const int total = c4 + 4;
    const int rot = GRID ? (rows_sh.rank * 64) % total & ~31 : 0;
    constexpr int U = 8;  // loads in flight per thread
    for (int b0 = threadIdx.x; b0 < total; b0 += U * blockDim.x) {
      float x[U];
      int64_t c[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        int i = b0 + u * blockDim.x;
        c[u] = i < total ? (i + rot < total ? i + rot : i + rot - total) : total;
      }
      if (GRID) {
        shifts<U>(slot, c, C, x);
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
          x[u] = c[u] < C ? (cw ? v[c[u]] : (v[c[u]] - nb[c[u]]) * cmd.ws) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (c[u] < total) {
          const float now = c[u] < C ? x[u] : -INFINITY;
          if (changes) fold_change(now, w[c[u]], mx, mn);
          w[c[u]] = now;
        }
      }
    }
    int* key = rows_sh.key[cmd.seq & 1];
    if (changes) publish_change(key, mx, mn);
    if (turns()) points_arrived();
    __syncthreads();
    if (threadIdx.x == 0) {
      float dmax = 0.f;
      rows_sh.bound[cmd.kind] = find && bounded(cmd.change, key[0], key[1], dmax);
      rows_sh.dmax[cmd.kind] = dmax;
    }
    __syncthreads();
  }

  static __device__ __forceinline__ void reduce_resident(int slot, int p0, int nrows) {
    const RowsCmd& cmd = rows_sh.cmd[slot];
    const RowsLayout& L = rows_sh.L;
    const bool isG = cmd.kind == kSweepG;
    const int wsh = 31 - __clz(blockDim.x >> 5), warp = threadIdx.x >> 5;
    const int c4 = isG ? L.n4 : L.m4, a4 = isG ? L.m4 : L.n4, G = c4 / 4;
    const int w = GRID || !constant() || wants_bound(cmd.kind)
                      ? (isG ? L.wx : L.wy)
                      : cmd.colx ? L.vx : L.vy + cmd.parity * (L.m4 + 4);
    const int lp = (isG ? L.ly : L.lx) + p0 - rows_sh.row0[cmd.kind];
    const bool tn = turns();
    const int as = tn ? (isG ? L.rg : L.rf) : a4;
    const int ax = tn ? (isG ? L.ay : L.ax) : isG ? L.cy : L.cx;
    const auto run = [&](auto warp_fn) {
      warp_fn(isG ? L.cx : L.cy, c4, w, (G * warp) >> wsh, (G * (warp + 1)) >> wsh, G,
              ax, nullptr, as, tn ? p0 - rows_sh.row0[cmd.kind] : p0, as - 4, (nrows + 3) / 4,
              rows_sh.cover[cmd.kind], cmd.s, L.pm + warp * L.rp, L.pl + warp * L.rp, true, lp,
              rows_sh.dmax[cmd.kind]);
    };
    if (rows_sh.bound[cmd.kind]) run(rows_warp<D, true>);
    else run(rows_warp<D, false>);
  }

  // Streamed columns: chunks by cp.async, double-buffered, each chunk's
  // shifts computed a chunk ahead.
  static constexpr int kChunk = rows_chunk(D);
  static constexpr int kPer = kChunk / kRowsThreads;  // columns per thread and chunk

  // Columns of a chunk: C in the fewest chunks of about equal width.
  static __device__ __forceinline__ int chunks(int C) { return (C + kChunk - 1) / kChunk; }
  static __device__ __forceinline__ int chunk_cols(int C) {
    const int n = chunks(C);
    return ((C + n - 1) / n + 127) & ~127;
  }

  // Chunk ch into buffer buf.
  static __device__ __noinline__ void stage(int slot, int ch, int buf) {
    const RowsCmd& cmd = rows_sh.cmd[slot];
    const ProbDev& P = rows_sh.P;
    const RowsLayout& L = rows_sh.L;
    const bool isG = cmd.kind == kSweepG;
    const float* Bt = isG ? P.xt : P.yt;
    const int64_t bp = isG ? P.n_pad : P.m_pad;
    const int C = (int)(isG ? P.n : P.m);
    const int wide = chunk_cols(C);
    const int64_t c0 = (int64_t)ch * wide;
    const int cols = (int)min((int64_t)wide, bp - c0);  // a multiple of 128
    float* dst = rows_mem + L.cx + (size_t)buf * D * kChunk;
    for (int k = 0; k < D; ++k)
      for (int i = threadIdx.x; i < cols / 4; i += blockDim.x)
        rows_cp16(dst + k * kChunk + 4 * i, Bt + k * bp + c0 + 4 * i);
    asm volatile("cp.async.commit_group;\n" ::);
    float x[kPer];
    int64_t c[kPer];
    const int64_t end = min((int64_t)C, c0 + wide);
#pragma unroll
    for (int j = 0; j < kPer; ++j) c[j] = c0 + threadIdx.x + j * kRowsThreads;
    shifts<kPer>(slot, c, end, x);
    float* w = rows_mem + L.w + buf * L.wstride + threadIdx.x;
#pragma unroll
    for (int j = 0; j < kPer; ++j) w[j * kRowsThreads] = c[j] < end ? x[j] : -INFINITY;
  }

  static __device__ __forceinline__ void reduce_chunk(int slot, int ch, int buf, bool first, int p0,
                                                      int nrows) {
    const RowsCmd& cmd = rows_sh.cmd[slot];
    const ProbDev& P = rows_sh.P;
    const RowsLayout& L = rows_sh.L;
    const bool isG = cmd.kind == kSweepG;
    const int wsh = 31 - __clz(blockDim.x >> 5), warp = threadIdx.x >> 5;
    const int C = (int)(isG ? P.n : P.m);
    const int wide = chunk_cols(C);
    const int G = (max(0, min(wide, C - ch * wide)) + 3) / 4;
    const float* ag = L.own ? nullptr : (isG ? P.yt : P.xt);
    const int64_t as = L.own ? (isG ? L.rg : L.rf) : (isG ? P.m_pad : P.n_pad);
    const int lp = (isG ? L.ly : L.lx) + p0 - rows_sh.row0[cmd.kind];
    const auto run = [&](auto warp_fn) {
      warp_fn(L.cx + buf * D * kChunk, kChunk, L.w + buf * L.wstride,
              (G * warp) >> wsh, (G * (warp + 1)) >> wsh, kChunk / 4, isG ? L.ay : L.ax, ag, as,
              L.own ? p0 - rows_sh.row0[cmd.kind] : p0, as - 4, (nrows + 3) / 4,
              rows_sh.cover[cmd.kind], cmd.s, L.pm + warp * L.rp, L.pl + warp * L.rp, first, lp,
              rows_sh.dmax[cmd.kind]);
    };
    if (rows_sh.bound[cmd.kind]) run(rows_warp<D, true>);
    else run(rows_warp<D, false>);
  }

  // ------------------------------------------------------------- rows
  // One row's update (finalize_row's) from its merged base-2 (shift, sum).
  // `lead` stores; lane k of [lane0, lane0 + lanes) sends to the CTAs k, k +
  // lanes, ... of the cluster. An evaluating sweep adds the row's error and
  // marginal terms.
  static __device__ __forceinline__ void update_row(int slot, int row, float mx, float lv, bool lead,
                                                    int k, int lanes, double& err, double& msum,
                                                    float& kx, float& kn) {
    const RowsCmd& cmd = rows_sh.cmd[slot];
    const ProbDev& P = rows_sh.P;
    const RowsLayout& L = rows_sh.L;
    const bool isG = cmd.kind == kSweepG;
    const int parity = cmd.parity, own = row - rows_sh.row0[cmd.kind];
    const float old = L.own ? rows_mem[(isG ? L.py + parity * L.rg : L.px) + own]
                            : __ldcg((isG ? P.gbuf[parity] : P.f) + row);
    const float nrmf = !GRID   ? rows_mem[(isG ? L.ny : L.nx) + row]
                       : L.own ? rows_mem[(isG ? L.any : L.anx) + own]
                                  : (isG ? P.ny : P.nx)[row];
    const double nrm = (double)nrmf;
    const double lm = L.own ? reinterpret_cast<const double*>(rows_mem + L.logm)[(isG ? L.rf : 0) + own]
                            : log((double)(isG ? P.b : P.a)[row]);
    if (mx == kNegSentinel && lv < 1.f) lv = 0.f;  // every column at -inf
    double lse2;
    if (log2_table_ok(lv)) lse2 = (double)mx + log2_table(rows_sh.log2t, lv);
    else lse2 = lv > 0.f ? (double)mx + log2((double)lv)
                         : (lv == 0.f ? -INFINITY : (double)NAN);
    const double app = cmd.epsln2 * lse2 - nrm;
    if (lead && L.lx) rows_mem[(isG ? L.ly : L.lx) + own] = (float)lse2;
    if (cmd.write) {
      const bool keep = isfinite(old) && isfinite(app);
      double newp = cmd.eps * lm - (keep ? app : 0.0);
      // symmetric problem: Momentum(value=0.5) on the parallel update
      if (P.symmetric) newp = 0.5 * (isfinite(old) ? (double)old : 0.0) + 0.5 * newp;
      const float nf = (float)newp;
      if (GRID) {
        if (!resident()) fold_change(nf * P.ws_t, old * P.ws_t, kx, kn);
        if (lead) {
          if (P.words) {
            const int64_t at = (isG ? P.n + (parity ^ 1) * P.m : 0) + row;
            const float x = constant() ? (nf - nrmf) * P.ws_t : nf;
            if (rows_sh.A.seqwords) word_store(P.words + at, x, cmd.seq);
            else reinterpret_cast<float*>(P.words)[at] = x;
          }
          (isG ? P.gbuf[parity ^ 1] : P.f)[row] = nf;
        }
      } else {
        const float x = constant() ? (nf - nrmf) * P.ws_t : nf;
        float* dst = rows_mem + (isG ? L.vy + (parity ^ 1) * (L.m4 + 4) : L.vx) + row;
        if (rows_sh.size == 1) {
          if (lead) *dst = x;
        } else {
          const uint64_t* b = &rows_sh.bar[isG ? 1 + (parity ^ 1) : 0];
          // only to the CTAs that own rows of the sweep that reads them
          if (!rows_sh.partial) {
            for (int q = k; q < rows_sh.size; q += lanes)
              cluster_store_async(cluster_addr(dst, q), x, cluster_addr(b, q));
          } else {
            const unsigned readers = rows_sh.owners[isG ? kSweepF : kSweepG];
            for (int q = k; q < rows_sh.size; q += lanes)
              if (readers >> q & 1) cluster_store_async(cluster_addr(dst, q), x, cluster_addr(b, q));
          }
        }
      }
      if (lead && L.own) rows_mem[(isG ? L.py + (parity ^ 1) * L.rg : L.px) + own] = nf;
    }
    if (cmd.eval && lead) {
      const double mg = (double)(isG ? P.b : P.a)[row];
      double bh = 0.0;
      if (!(old == -INFINITY)) bh = exp2(lse2 + ((double)old - nrm) * (double)cmd.ws);
      const double dv = fabs(bh - mg);
      err += (rows_sh.A.cfg.norm_error == 1) ? dv : pow(dv, (double)rows_sh.A.cfg.norm_error);
      msum += bh;
      if (cmd.fin && P.marg_out) P.marg_out[row] = (float)bh;
      if (cmd.fin && P.lse_out) P.lse_out[row] = (float)app;
    }
  }

  // Rows [p0, p0 + nrows): merge the warps' slices and update. Few rows: 16
  // lanes a row, one slice each, merged by shuffles, and the same lanes send
  // the new value to the CTAs of a cluster (a thread a row, its 32 loads and
  // its stores to 16 CTAs in turn took ~2500 of the ~6900 cycles of a small
  // problem's sweep); many rows: a thread a row.
  static __device__ __forceinline__ void update(int slot, int p0, int nrows, double& err,
                                                double& msum) {
    const RowsLayout& L = rows_sh.L;
    const int W = blockDim.x >> 5;
    const int kind = rows_sh.cmd[slot].kind;
    const bool bound = rows_sh.bound[kind] != 0;
    const float dmax = rows_sh.dmax[kind];
    const int lp = (kind == kSweepG ? L.ly : L.lx) + p0 - rows_sh.row0[kind];
    float kx = -INFINITY, kn = INFINITY;
    if (nrows <= 4 * W) {
      const int k = threadIdx.x & 15, half = (threadIdx.x >> 4) & 1;
      for (int r2 = (threadIdx.x >> 5) * 2; r2 < nrows; r2 += 2 * W) {
        const int r = min(r2 + half, nrows - 1);  // an odd last row twice
        float lk = k < W ? rows_mem[L.pl + k * L.rp + r] : 0.f;
        float mx;
        if (bound) {
          mx = row_sigma(rows_mem[lp + r], dmax);
        } else {
          const float mk = k < W ? rows_mem[L.pm + k * L.rp + r] : kNegSentinel;
          mx = mk;
#pragma unroll
          for (int off = 8; off > 0; off >>= 1)
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
          lk *= ex2_approx(mk - mx);
        }
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) lk += __shfl_xor_sync(0xffffffffu, lk, off);
        if (r2 + half < nrows) update_row(slot, p0 + r, mx, lk, k == 0, k, 16, err, msum, kx, kn);
        __syncwarp();
      }
    } else {
      for (int r = threadIdx.x; r < nrows; r += blockDim.x) {
        float mx = kNegSentinel, lv = 0.f;
        if (bound) {
          mx = row_sigma(rows_mem[lp + r], dmax);
#pragma unroll
          for (int k = 0; k < kRowsWarps; ++k) lv += k < W ? rows_mem[L.pl + k * L.rp + r] : 0.f;
        } else {
          float mk[kRowsWarps];
#pragma unroll
          for (int k = 0; k < kRowsWarps; ++k) {
            mk[k] = k < W ? rows_mem[L.pm + k * L.rp + r] : kNegSentinel;
            mx = fmaxf(mx, mk[k]);
          }
#pragma unroll
          for (int k = 0; k < kRowsWarps; ++k)
            lv += (k < W ? rows_mem[L.pl + k * L.rp + r] : 0.f) * ex2_approx(mk[k] - mx);
        }
        update_row(slot, p0 + r, mx, lv, true, 0, 1, err, msum, kx, kn);
      }
      __syncwarp();
    }
    if (GRID && !resident() && rows_sh.P.dkey && rows_sh.cmd[slot].write)
      publish_change(rows_sh.P.dkey + 2 * (rows_sh.cmd[slot].seq & 3), kx, kn);
  }

  // Grid team: the CTAs' error (0) and marginal (1) sums, in the workspace's
  // per-row-block slots or, for more CTAs than row blocks, in the region of
  // the tiled engines' split partials (the host checks that they fit).
  static __device__ __forceinline__ double* part(int which) {
    const ProbDev& P = rows_sh.P;
    if (rows_sh.size <= P.rb_g) return which ? P.msum_part : P.err_part;
    return reinterpret_cast<double*>(P.part_m) + (which ? rows_sh.size : 0);
  }

  // The team's error and marginal sums, in a fixed order (lanes, warps,
  // CTAs), into rows_sh.err and rows_sh.msum of every CTA. False after a timeout.
  // A CTA overwrites its sums in the next evaluating sweep, which must not
  // begin while another still reads these. Most often the values exchanged in
  // between see to that. They do not where a CTA without rows waits for
  // nobody's, nor where every sweep evaluates (blocks of one iteration of a
  // symmetric problem: the values are out before the sums are read). Such
  // teams meet once more behind the reading (resync).
  static __device__ __noinline__ bool sums(double err, double msum) {
    const int W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int off = 16; off > 0; off >>= 1) {
      err += __shfl_xor_sync(0xffffffffu, err, off);
      msum += __shfl_xor_sync(0xffffffffu, msum, off);
    }
    if (lane == 0) {
      rows_sh.red[0][warp] = err;
      rows_sh.red[1][warp] = msum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      err = msum = 0.0;
      for (int k = 0; k < W; ++k) {
        err += rows_sh.red[0][k];
        msum += rows_sh.red[1][k];
      }
      if (GRID) {
        part(0)[rows_sh.rank] = err;
        part(1)[rows_sh.rank] = msum;
      } else {
        for (int q = 0; q < rows_sh.size; ++q) {
          cluster_store(cluster_addr(&rows_sh.slot[0][rows_sh.rank], q), err);
          cluster_store(cluster_addr(&rows_sh.slot[1][rows_sh.rank], q), msum);
        }
      }
    }
    if (!barrier()) return false;
    if (warp == 0) {
      double e = 0.0, u = 0.0;
      for (int i = lane; i < rows_sh.size; i += 32) {
        e += GRID ? __ldcg(part(0) + i) : rows_sh.slot[0][i];
        u += GRID ? __ldcg(part(1) + i) : rows_sh.slot[1][i];
      }
      for (int off = 16; off > 0; off >>= 1) {
        e += __shfl_xor_sync(0xffffffffu, e, off);
        u += __shfl_xor_sync(0xffffffffu, u, off);
      }
      if (lane == 0) {
        rows_sh.err = e;
        rows_sh.msum = u;
      }
    }
    if (rows_sh.resync) return barrier();
    __syncthreads();
    return true;
  }

  static __device__ __forceinline__ bool barrier() {
    if (GRID) return grid_barrier(rows_sh.A.gl, rows_sh.A.expected, rows_sh.A.timeout_ns, &rows_sh.A.sched->status, rows_sh.bar_grid);
    cluster_barrier(rows_sh.size);
    return true;
  }

  // ------------------------------------------------------------- loop
  // False after a wait of the grid team ran out.
  static __device__ __forceinline__ bool solve(int p) {
    begin();
    if (!GRID) cluster_barrier(rows_sh.size);
    if (control()) advance(0, true, 0.0, 0.0);
    __syncthreads();
    int cur = 0;
    for (; !rows_sh.cmd[cur].done; cur ^= 1) {
      const RowsCmd& cmd = rows_sh.cmd[cur];
      double err = 0.0, msum = 0.0;
      int p0 = rows_sh.row0[cmd.kind];
      while (true) {
        const int nrows = min(rows_sh.row1[cmd.kind] - p0, rows_sh.L.rp);
        if (resident()) {
          if (nrows > 0) {
            if (p0 == rows_sh.row0[cmd.kind]) columns(cur);
            reduce_resident(cur, p0, nrows);
          } else if (turns()) {
            points_arrived();  // before the next load into the buffer
          }
        } else {
          const int C = (int)(cmd.kind == kSweepG ? rows_sh.P.n : rows_sh.P.m);
          const int nch = chunks(C);
          // each CTA starts at another chunk (see columns)
          int ch = rows_sh.rank % nch;
          stage(cur, ch, 0);
          if (threadIdx.x == 0) {
            // the last write's keys: this sweep's columns
            float dmax = 0.f;
            const int* key = rows_sh.P.dkey + 2 * (cmd.want & 3);
            rows_sh.bound[cmd.kind] =
                rows_sh.P.dkey && rows_sh.L.lx &&
                bounded(cmd.change, cmd.change > 0 ? __ldcg(key) : kDkeyEmptyMax,
                        cmd.change > 0 ? __ldcg(key + 1) : kDkeyEmptyMin, dmax);
            rows_sh.dmax[cmd.kind] = dmax;
          }
          for (int k = 0; k < nch; ++k) {
            const int after = ch + 1 < nch ? ch + 1 : 0;
            if (k + 1 < nch) {
              stage(cur, after, (k + 1) & 1);
              asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            } else {
              asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            }
            __syncthreads();
            if (nrows > 0) reduce_chunk(cur, ch, k & 1, k == 0, p0, nrows);
            __syncthreads();
            ch = after;
          }
        }
        __syncthreads();
        if (GRID && *(volatile int*)&rows_sh.fail) return false;
        const bool last = p0 + rows_sh.L.rp >= rows_sh.row1[cmd.kind];
        if (last && !cmd.eval && control()) advance(cur ^ 1, false, 0.0, 0.0);
        // an evaluating sweep that already writes is most often followed by
        // the other side's
        if (turns() && last && cmd.eval && cmd.write && control())
          load_points(rows_sh.P.symmetric ? kSweepG : kSweepF);
        update(cur, p0, nrows, err, msum);
        if (last) break;
        p0 += rows_sh.L.rp;
        __syncthreads();  // the slices are free for the next pass
      }
      if (cmd.eval) {
        if (!sums(err, msum)) return false;
        if (control()) advance(cur ^ 1, false, rows_sh.err, rows_sh.msum);
      } else if (GRID && !rows_sh.A.seqwords) {
        // (otherwise the values themselves order the sweeps)
        if (!barrier()) return false;
      }
      __syncthreads();
    }
    const RowsState& S = rows_sh.st;
    int fpar = S.fpar;
    if (!GRID) {
      // values of a sweep whose state was dropped still come in
      for (int k = 0; k < 3; ++k)
        if (S.pending >> k & 1) arrived(k, S.phases >> k & 1);
      const ProbDev& P = rows_sh.P;
      const RowsLayout& L = rows_sh.L;
      const int x0 = rows_sh.row0[kSweepF], x1 = rows_sh.row1[kSweepF];
      const int y0 = rows_sh.row0[kSweepG], y1 = rows_sh.row1[kSweepG];
      for (int i = x0 + threadIdx.x; i < x1; i += blockDim.x) P.f[i] = rows_mem[L.px + i - x0];
      for (int i = y0 + threadIdx.x; i < y1; i += blockDim.x)
        P.gbuf[0][i] = rows_mem[L.py + fpar * L.rg + i - y0];
      fpar = 0;
    }
    if (rows_sh.rank == 0 && threadIdx.x == 0) {
      ProbState& out = rows_sh.A.state[p];
      out.active = 0;
      out.final_parity = fpar;
      out.stop_it = S.it;
      out.msum = rows_sh.msum;
      out.msum_valid = 1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      rows_sh.st.phases ^= rows_sh.st.pending;
      rows_sh.st.pending = 0;
    }
    return true;
  }

  static __device__ __forceinline__ void rows_cp16(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
  }
};

// GRID: every problem of the list in turn by the whole (co-resident) grid.
// Otherwise: clusters of any size take problems from the queue.
template <int D, bool GRID>
__global__ void __launch_bounds__(kRowsThreads, 1) sinkhorn_rows_kernel(RowsArgs args) {
  using Solver = RowsSolver<D, GRID>;
  if (threadIdx.x == 0) {
    rows_sh.A = args;
    rows_sh.rank = GRID ? (int)blockIdx.x : (int)cluster_rank();
    rows_sh.size = GRID ? (int)gridDim.x : (int)cluster_size();
    rows_sh.bar_grid.phase = 0;
    rows_sh.st.phases = 0;
    rows_sh.fail = 0;
    rows_sh.pts_loads = 0;
    for (int k = 0; k < 3; ++k) tc::mbar_init(&rows_sh.bar[k], 1);
    tc::fence_barrier_init();
  }
  log2_table_fill(rows_sh.log2t);
  __syncthreads();
  // clusters have no grid barrier: a call that asks for phantom arrivals
  // ends here with its timeout
  if (!GRID && args.expected && !grid_barrier(args.gl, args.expected, args.timeout_ns,
                                              &args.sched->status, rows_sh.bar_grid))
    return;
  for (int k = 0;; ++k) {
    int q = k;
    if (!GRID) {
      // one draw per cluster; the barrier before it also ends the last
      // problem's use of the CTAs' shared memory
      cluster_barrier(rows_sh.size);
      if (rows_sh.rank == 0 && threadIdx.x == 0) {
        const int next = (int)atomicAdd(&args.gl->unit_ctr[0], 1u);
        for (int i = 0; i < rows_sh.size; ++i) cluster_store(cluster_addr(&rows_sh.q, i), next);
      }
      cluster_barrier(rows_sh.size);
      q = rows_sh.q;
    }
    if (q >= args.count) break;
    const int p = args.ids[q];
    __syncthreads();
    {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(args.probs + p);
      uint32_t* dst = reinterpret_cast<uint32_t*>(&rows_sh.P);
      for (int i = threadIdx.x; i < (int)(sizeof(ProbDev) / 4); i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    const bool ok = Solver::solve(p);
    if (Solver::turns()) Solver::points_arrived();
    if (!ok) return;
  }
}

}  // namespace ottb
