// The FP32 row-owner engine (engine_rows.cuh) as the solve's host side sees
// it: launch arguments, the split of rows over a team, the shared-memory
// layout and the kernel table.
#pragma once

#include "common.cuh"

namespace ottb {

constexpr int kRowsMaxDim = 16;
constexpr int kRowsThreads = 512;    // most threads of a CTA
constexpr int kRowsWarps = kRowsThreads / 32;
constexpr int kRowsMaxCluster = 16;
constexpr int kRowsMaxCtas = 240;    // most CTAs of a grid team
constexpr int kRowsChunk = 2048;     // columns per streamed chunk (1024 for D > 10)
constexpr int kRowsPass = 384;       // most rows of a CTA reduced in one pass over the columns
constexpr int kRowsOwnFloats = 8192; // most floats of a CTA's own rows kept in shared memory
constexpr int kRowsKeptRows = 8192;  // most own rows whose last log-sum-exp is kept
constexpr int kRowsKeyBytes = 3840;  // grid: the shift-change keys, behind the CTAs' sums
// Dynamic shared memory a CTA may ask for: 227 KB less the kernels' static
// part (rows.cu checks that it is below 3 KB).
constexpr int kRowsSmemMax = 224 * 1024;

struct RowsArgs {
  ProbDev* probs;
  ProbState* state;
  Sched* sched;
  Globals* gl;
  const int* ids;       // the launch's problems, table positions
  int count;
  int resident;         // grid team: a sweep's columns are in shared memory at once
  int turns;            // ... both point sets in one buffer, in turns
  int seqwords;         // grid team: values exchanged as {value, sweep number} words
  unsigned expected;    // barrier arrivals (CTAs + phantom arrivals; clusters: 0 without phantoms)
  uint64_t timeout_ns;
  ottb_solver_cfg cfg;
};

__host__ __device__ constexpr int rows_chunk(int D) { return D > 10 ? kRowsChunk / 2 : kRowsChunk; }

// Column groups (of 4) that a lane takes per iteration: two while their
// products fit beside the rows' coordinates in registers; one leaves more
// parts of a CTA's columns, so fewer iterations are padding (n = 3000, m =
// 4100, d = 10, two against one: 1.34 and 1.19 ms; n = m = 3000, d = 8: 0.95
// and 0.85; n = 6000, m = 5000, d = 5: 1.51 and 1.54).
__host__ __device__ constexpr int rows_groups(int D) { return D <= 6 ? 2 : 1; }

// First row of team member `rank` of `size`: whole quads of rows.
__host__ __device__ __forceinline__ int64_t rows_begin(int64_t n, int rank, int size) {
  const int64_t q = (n + 3) / 4;
  const int64_t r = 4 * (q * rank / size);
  return r < n ? r : n;
}

// Most rows a member of a team of `size` owns of n, rounded up to a quad.
__host__ __device__ __forceinline__ int64_t rows_most(int64_t n, int size) {
  const int64_t q = (n + 3) / 4;
  return 4 * ((q + size - 1) / size);
}

// Shared-memory layout of a CTA for one problem, offsets in floats (0 where
// the mode has no such array). Every array starts on 16 bytes.
//   cluster: points, norms, the exchanged column values of both sides (y
//     twice, by g parity), the own rows' potentials
//   grid, resident: points; in turns: one buffer for either side's points,
//     the own rows' points
//   grid, streamed: two chunks of the column side's points; the own rows'
//     points where they fit
// then the own rows' norms, potentials and log-sum-exps, the column shifts,
// the warps' partial (shift, sum) of the CTA's rows
// and the own rows' log weights.
//
// A streamed layout fits kRowsSmemMax at every size: where it would not (D >=
// 7: two chunks take 128 or 160 KB), the own rows' data stay in global
// memory, and passes have at most kRowsPass / 2, then kRowsPass / 4 rows
// (`cut` 1 to 3).
struct RowsLayout {
  int n4, m4;          // points rounded up to a quad
  int rf, rg;          // most own rows of the f- and g-sweep (whole quads)
  int rp;              // rows per pass
  int own;             // own rows' data in shared memory
  int cx, cy, nx, ny;  // points [D][n4], [D][m4], norms
  int ax, ay, anx, any;  // in turns, streamed: own rows' points [D][rf], [D][rg], norms
  int vx, vy;          // cluster: exchanged values [n4 + 4], [2][m4 + 4]
  int px, py;          // own rows' potentials [rf], [2][rg]
  int lx, ly;          // own rows' log-sum-exps of their last sweep [rf], [rg] (0: not kept)
  int wx, wy;          // resident: column shifts of both sides
  int w, wstride;      // streamed: two chunks' column shifts
  int pm, pl, logm;
  int total;
};

__host__ __device__ inline RowsLayout rows_layout_cut(int64_t n, int64_t m, int D, int size,
                                                      int warps, bool cluster, bool resident,
                                                      bool turns, int cut) {
  RowsLayout L{};
  L.n4 = (int)((n + 3) / 4 * 4);
  L.m4 = (int)((m + 3) / 4 * 4);
  L.rf = (int)rows_most(n, size);
  L.rg = (int)rows_most(m, size);
  const int most = L.rf > L.rg ? L.rf : L.rg;
  const int pass = cut < 2 ? kRowsPass : kRowsPass >> (cut - 1);
  L.rp = most < pass ? most : pass;
  L.own = cluster || (cut == 0 && (int64_t)(L.rf + L.rg) * (D + 1) <= kRowsOwnFloats) ? 1 : 0;
  int64_t p = 0;
  auto take = [&](int64_t k) {
    const int64_t o = p;
    p += (k + 3) / 4 * 4;
    return (int)o;
  };
  if (cluster || resident) {
    if (turns) {
      L.cx = L.cy = take((int64_t)D * (L.n4 > L.m4 ? L.n4 : L.m4));
      L.ax = take((int64_t)D * L.rf);
      L.ay = take((int64_t)D * L.rg);
    } else {
      L.cx = take((int64_t)D * L.n4);
      L.cy = take((int64_t)D * L.m4);
    }
    if (cluster) {
      L.nx = take(L.n4);
      L.ny = take(L.m4);
    }
    L.wx = take(L.n4 + 4);
    L.wy = take(L.m4 + 4);
    if (cluster) {
      L.vx = take(L.n4 + 4);
      L.vy = take(2 * ((int64_t)L.m4 + 4));
    }
  } else {
    L.cx = take(2 * (int64_t)rows_chunk(D) * D);
    L.wstride = rows_chunk(D) + 4;
    L.w = take(2 * (int64_t)L.wstride);
    if (L.own) {
      L.ax = take((int64_t)D * L.rf);
      L.ay = take((int64_t)D * L.rg);
    }
  }
  if (!cluster && L.own) {
    L.anx = take(L.rf);
    L.any = take(L.rg);
  }
  if (L.rf + L.rg <= kRowsKeptRows) {
    L.lx = take(L.rf);
    L.ly = take(L.rg);
  }
  L.pm = take((int64_t)warps * L.rp);
  L.pl = take((int64_t)warps * L.rp);
  if (L.own) {
    L.px = take(L.rf);
    L.py = take(2 * (int64_t)L.rg);
    L.logm = take(2 * ((int64_t)L.rf + L.rg));
  }
  L.total = p > (1 << 28) ? 1 << 28 : (int)p;
  return L;
}

__host__ __device__ inline RowsLayout rows_layout(int64_t n, int64_t m, int D, int size, int warps,
                                                  bool cluster, bool resident, bool turns) {
  int cut = 0;
  RowsLayout L = rows_layout_cut(n, m, D, size, warps, cluster, resident, turns, cut);
  while (!cluster && !resident && cut < 3 && L.total > kRowsSmemMax / 4)
    L = rows_layout_cut(n, m, D, size, warps, cluster, resident, turns, ++cut);
  return L;
}

// What the grid team's CTAs exchange, 8 bytes a point of workspace: column
// shifts (potentials where the epsilon multiplier varies), x's and two
// buffers of y's, either plain floats behind the barrier or words {value,
// sweep number}: a reader polls the data itself, so a new value reaches it
// in one trip through L2 (write, poll) instead of three (write and release,
// barrier, load). They live in the region of the tiled engines' split
// partials, behind the CTAs' error sums, where they fit. What a word held is
// overwritten only by a CTA that has read every word of the sweep between,
// and every CTA that reads the old ones writes those after it has read them
// (the g words have two buffers). A CTA without rows of a sweep therefore
// reads none of its values: with n = 4000, m = 200 on 148 CTAs, 98 own no
// row of y and publish nothing in g-sweeps, so nothing would hold back the
// f-sweep that overwrites what they read. Every CTA with rows reads every
// word, so the words lose where there are many: an iteration of n = m, d = 2
// takes, with words and with the barrier, 16.9 and 19.2 us at 1000, 18.3 and
// 20.8 at 2000, 27.5 and 24.3 at 2500, 24.2 and 26.6 at 3000, 27.5 and 29.6
// at 4000, 55 and 39 at 5000, 61 and 47 at 6000 (B200; d = 4 and 8 alike):
// they turn between n + m = 8000 and 10000. The limit lies below that.
constexpr int64_t kRowsWordsMax = 6000;
constexpr size_t kRowsSumBytes = 4096;  // 2 doubles a CTA (up to kRowsMaxCtas), the keys
__host__ __device__ __forceinline__ size_t rows_words_bytes(int64_t n, int64_t m) {
  return kRowsSumBytes + 8 * (size_t)(n + 2 * m);
}
// Dynamic shared memory of a CTA, in bytes.
__host__ __device__ inline size_t rows_smem(int64_t n, int64_t m, int D, int size, int warps,
                                            bool cluster, bool resident, bool turns = false) {
  // beyond any CTA's shared memory (and the offsets' range)
  if ((cluster || resident) && (n + m) * (int64_t)(D + 1) > (1 << 20)) return (size_t)1 << 30;
  const RowsLayout L = rows_layout(n, m, D, size, warps, cluster, resident, turns);
  if (turns && !L.own) return (size_t)1 << 30;
  return (size_t)L.total * 4;
}

struct RowsKernel {
  int D = 0;                      // coordinates the kernel reads (>= d)
  const void* grid = nullptr;     // one team: the whole grid (cooperative launch)
  const void* cluster = nullptr;  // teams: thread-block clusters of any size
};

// The kernels for dimension d; D = 0 above kRowsMaxDim.
RowsKernel rows_kernel(int d);

// Static shared memory of the kernels, in bytes.
size_t rows_static_smem();

}  // namespace ottb
