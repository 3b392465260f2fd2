// Which engine an FP32 call takes, from the sizes alone: the row-owner engine
// (engine_rows.cuh), and with which teams, or the tiled one (engine_simt.cuh).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "rows.h"

namespace ottb {

// Column splits of one sweep: enough units to keep every CTA busy with
// little tail (efficiency = units / (waves * grid)).
inline int choose_split(int rb, int ntiles, int grid, int num_problems) {
  if (num_problems > 1 || grid <= 0) return 1;
  int best = 1;
  double best_score = -1.0;
  const int smax = std::max(1, std::min(ntiles, 32));
  for (int s = 1; s <= smax; ++s) {
    const double units = (double)rb * s;
    const double waves = std::ceil(units / grid);
    const double eff = units / (waves * grid);
    const double score = eff - 0.004 * s;
    if (score > best_score + 1e-9) {
      best_score = score;
      best = s;
    }
  }
  return best;
}

// CTAs of the tiled engine's grid and of the row-owner engine's on a B200.
constexpr int kTiledCtas = 296, kRowsCtas = 148;

inline bool rows_fits(size_t bytes) { return bytes <= (size_t)kRowsSmemMax; }
// Either both sides' points stay in a CTA's shared memory, or either side's.
inline bool rows_resident(int64_t n, int64_t m, int D) {
  return rows_fits(rows_smem(n, m, D, kRowsCtas, kRowsWarps, false, true)) ||
         rows_fits(rows_smem(n, m, D, kRowsCtas, kRowsWarps, false, true, true));
}

// Microseconds of an iteration (both sweeps) of one problem by the whole grid
// of the row-owner engine, D <= 10: the CTA with the most quads of rows over
// all columns, and what a sweep costs beyond (streamed: and a chunk of
// columns, whose loads are one chunk ahead). Fitted to B200 solves of 150 to
// 131072 points a side.
inline double rows_grid_us(int64_t n, int64_t m, int D) {
  const double entry =  // an entry of a CTA
      1e-3 * (D <= 2   ? 0.044
              : D == 3 ? 0.047
              : D == 4 ? 0.050
              : D <= 6 ? 0.065
              : D <= 8 ? 0.075
                       : 0.090);
  const bool res = rows_resident(n, m, D);
  double t = 0.0;
  for (int side = 0; side < 2; ++side) {
    const int64_t C = side ? n : m, rows = rows_most(side ? m : n, kRowsCtas);
    const double passes = (double)((rows + kRowsPass - 1) / kRowsPass);
    const double chunks = (double)((C + rows_chunk(D) - 1) / rows_chunk(D));
    const double work = (double)rows * (double)C * entry;
    t += res ? 8.5 + 1.08 * work : 6.5 + (2.2 + 0.17 * D) * passes * chunks + work;
  }
  return t;
}

// The same of a call by the tiled engine: units of whole tiles of 128 x 128
// over the grid. A single problem keeps its first split; several start
// without one and grow it to 8 (an average of about 4) while they offer less
// than two units a CTA.
inline double tiled_us(const ottb_problem* probs, int num, int dp) {
  // a tile, by one CTA of two an SM
  const double tile = dp <= 2 ? 1.95 : dp <= 4 ? 2.4 : dp <= 8 ? 3.1 : 4.6;
  const double unit = 7.5, sweep = 8.8;
  double t = 0.0;
  for (int side = 0; side < 2; ++side) {
    double work = 0.0, units = 0.0, longest = 0.0;
    for (int i = 0; i < num; ++i) {
      const int64_t R = side ? probs[i].m : probs[i].n, C = side ? probs[i].n : probs[i].m;
      const int64_t rb = (R + kBM - 1) / kBM, nt = (C + kBM - 1) / kBM;
      if (num == 1) {
        const int s = choose_split((int)rb, (int)nt, kTiledCtas, 1);
        const int64_t u = rb * s, left = u % kTiledCtas;
        const double one = std::ceil((double)nt / s) * tile;
        t += sweep + (double)(u / kTiledCtas) * (one + unit);
        // a CTA that has its SM to itself is faster
        if (left) t += (left > kTiledCtas / 2 ? one : 0.74 * one) + unit;
      }
      work += (double)rb * ((double)nt * tile + unit);
      units += (double)rb;
      longest = std::max(longest, (double)nt * tile);
    }
    const double grown = std::min(4.0, std::max(1.0, 2.0 * kTiledCtas / units));
    if (num > 1) t += sweep + std::max(1.05 * work / kTiledCtas, longest / grown + unit);
  }
  return t;
}

// Whether an FP32 call goes to the row-owner engine (D: its padded dimension,
// 0 for none; dp: the tiled engine's).
//
// d <= 10, one problem, and d <= 4, several: where every problem fits a
// cluster or (one problem) the grid's shared memory, always (20 iterations of
// n = 4000, m = 200, d = 2: 0.65 -> 0.39 ms by the row-owner engine; 64
// problems of 4000 x 100, d = 2, 60 iterations: 8.1 -> 4.7). Beyond, the one
// that the models above find faster. The row-owner engine's weak spot is a
// short side's sweep: few rows a CTA do not pay for streaming the other
// side's columns, and quads of rows do not divide evenly. Measured, tiled
// against row-owner, an iteration: 200 x 100000, d = 2: 0.10 and 0.18 ms;
// 1200 x 100000, d = 8: 0.26 and 0.36; 16 problems of 20000 x 300, d = 2: 0.23
// and 0.66; 32 of 6000 x 6000: 1.1 and 1.3. The other way: 64 x 100000, d = 2,
// (one row block: no split): 1.07 and 0.18; n = m = 30000, d = 10: 1.84 and
// 1.18; 2000 x 40000, d = 3: 0.24 and 0.12; 4 problems of 8000 x 8000: 0.30
// and 0.24. Where the two are within 10 % the models may be wrong.
//
// Other dimensions: one problem while the points stay in shared memory, both
// sides or in turns (n = m = 3500, d = 12: 1.22 against 2.26 ms; n = 2900, m
// = 2800, d = 16: 1.37 against 1.48; n = m = 16000, d = 16, streamed: 20.5
// against 16.8). A batch when each of its problems fits a cluster of 8 (96
// problems up to 4096 points, d = 8, of which a part had to go through the
// grid one by one: 12.8 against 7.6).
inline bool rows_wanted(const ottb_problem* probs, int num, int D, int dp) {
  if (D == 0) return false;
  // row and column numbers are ints there
  for (int i = 0; i < num; ++i)
    if (std::max(probs[i].n, probs[i].m) > (int64_t)1 << 30) return false;
  if (D > 10 || (num > 1 && D > 4)) {
    if (num == 1) return rows_resident(probs[0].n, probs[0].m, D);
    for (int i = 0; i < num; ++i)
      if (!rows_fits(rows_smem(probs[i].n, probs[i].m, D, 8, kRowsWarps, true, false))) return false;
    return true;
  }
  if (num == 1 && rows_resident(probs[0].n, probs[0].m, D)) return true;
  double grid = 0.0;
  for (int i = 0; i < num; ++i) {
    const int64_t n = probs[i].n, m = probs[i].m;
    if (!rows_fits(rows_smem(n, m, D, kRowsMaxCluster, kRowsWarps, true, false)))
      grid += rows_grid_us(n, m, D);
  }
  return grid == 0.0 || grid <= tiled_us(probs, num, dp);
}

// Problem of a call, and the CTAs that the whole grid would solve it with.
struct RowsSize {
  int64_t n, m;
  int grid_ctas;
};

// Teams of a call: the first `grid` problems one after another by the whole
// grid, the others drawn by clusters of `csize` CTAs.
struct RowsTeams {
  int grid = 0, csize = 1, cthreads = 0, nclusters = 0;
  size_t csmem = 0;
};

// Team sizes of the row-owner engine for problems in decreasing work, from a
// model of one sweep in SM cycles: entries x cycles per entry / CTAs, plus
// what a sweep costs beyond its entries (column shifts, lane and warp merges,
// the update in FP64, the team's barrier). clusters(size, threads, smem): how
// many clusters the device holds at once; where it holds none of the best
// size (SMs of a GPC left to others), smaller ones and the grid are tried.
template <class Clusters>
inline RowsTeams rows_teams(const std::vector<RowsSize>& probs, int D, int sms, size_t static_smem,
                            Clusters clusters) {
  const double per_entry = D <= 4 ? 0.105 : (D + 8) / 75.0;
  const int num = (int)probs.size();
  const double over_one = 4500, over_cluster = 5500, over_warp = 100;
  // Several problems in turn take the grid 11000 to 22000 cycles a sweep
  // beyond their entries (an iteration of 8 problems of 3400 x 3400, d = 2:
  // 177 us, 95 in clusters of 16; 4 of 2600 x 2600: 113 and 47).
  const double over_grid = num > 1 ? 15000 : 11000;
  // The share of the longest problem that a batch ends with: above d = 4 large
  // clusters gain less (64 problems of 2500 x 1000, d = 8: 360 us an iteration
  // with 1, 230 with 0.5; 900 of 300 x 200, d = 2: 426 and 445).
  const double tail = D > 4 ? 0.5 : 1.0;
  auto entries = [&](const RowsSize& p) { return (double)p.n * (double)p.m * per_entry; };
  // grid_t[k]: the k largest problems by the whole grid
  std::vector<double> grid_t(num + 1, 0.0);
  for (int t = 0; t < num; ++t)
    grid_t[t + 1] = grid_t[t] + entries(probs[t]) / probs[t].grid_ctas + over_grid;
  for (int most = kRowsMaxCluster;;) {
    RowsTeams T;
    T.grid = num;
    double best = grid_t[num];
    for (int C = 1; C <= most; C *= 2) {
      for (int threads = kRowsThreads; threads >= 128; threads /= 2) {
        const int warps = threads / 32;
        double sum = 0.0, longest = 0.0;
        size_t smem = 0;
        for (int k = num - 1; k >= 0; --k) {
          const RowsSize& p = probs[k];
          smem = std::max(smem, rows_smem(p.n, p.m, D, C, warps, true, false));
          if (!rows_fits(smem)) break;
          // CTAs that share an SM share its pipes; one alone needs about ten
          // warps to fill them
          const int per_sm = std::min<int>(kRowsThreads / threads,
                                           (int)(kRowsSmemMax / (smem + static_smem + 1024)));
          // large clusters leave SMs of a GPC over (7 of 9 clusters of 16 fit)
          const double slots = (double)sms * std::max(per_sm, 1) / C *
                               (C >= 8 ? 0.78 : C >= 4 ? 0.88 : 1.0);
          const double alone = std::min(1.0, warps / 10.0);
          const double share = std::max(1.0, std::min((double)per_sm, (num - k) * C / (double)sms));
          const double t = entries(p) / C / std::min(alone, 1.0 / share) +
                           (C > 1 ? over_cluster : over_one) + over_warp * warps;
          sum += t;
          longest = std::max(longest, t);
          // problems stop at different iterations: a batch ends with its
          // longest-running ones, unless every problem has a cluster at once
          const bool at_once = C == kRowsMaxCluster && num <= (int)slots;
          const double est = at_once ? longest : std::max(longest, sum / slots + tail * longest);
          if (grid_t[k] + est < best) {
            best = grid_t[k] + est;
            T.grid = k;
            T.csize = C;
            T.cthreads = threads;
            T.csmem = smem;
          }
        }
      }
    }
    if (T.grid == num) return T;
    T.nclusters = std::min(clusters(T.csize, T.cthreads, T.csmem), num - T.grid);
    if (T.nclusters > 0) return T;
    most = T.csize / 2;
  }
}

}  // namespace ottb
