// How the persistent kernels' work is dealt to CTAs: host and device code without CUDA calls
// (tests/test_work_lists.py runs it on the CPU).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

namespace sp2b {

// ---- FP64 dense solve (k_f64_solve) ----
// The work of one step in units of one 16-row k-block of one tile, tile after tile: first
// the ntiles products X^2 (kb units each), then, with a response, the ntiles
// anticommutator tiles X Delta + Delta X (2 kb units each, K concatenated).  CTA c takes
// the units [bound(c), bound(c + 1)): equal shares, so no partial last wave of tiles leaves
// SMs idle.  A tile cut by a bound is summed by the CTA that holds its last units; the
// others leave their accumulators in a workspace slot.  A bound closer than `snap` units to
// a tile edge moves to that edge.
struct F64Split {
  int kb, ntiles, snap, G;
  long long total;

  __host__ __device__ inline int len(int job) const { return job < ntiles ? kb : 2 * kb; }
  __host__ __device__ inline void locate(long long u, int& job, int& off) const {
    const long long first = (long long)ntiles * kb;
    if (u < first) {
      job = (int)(u / kb);
      off = (int)(u - (long long)job * kb);
    } else {
      const long long v = u - first;
      const int q = (int)(v / (2 * kb));
      job = ntiles + q;
      off = (int)(v - (long long)q * 2 * kb);
    }
  }
  __host__ __device__ inline long long bound(int c) const {
    const long long u = total * c / G;
    int job, off;
    locate(u, job, off);
    if (off == 0) return u;
    if (off < snap) return u - off;
    const int rest = len(job) - off;
    return rest < snap ? u + rest : u;
  }
};

constexpr int kMaxPieces = 64;   // pieces of one tile that other CTAs may hold

struct F64Plan {
  int bt, tiles, grid, snap;
};

// Grid of an order-n solve: one CTA per SM, but at least min_units k-blocks each (a cut tile
// costs its owner and the others ~2 us of workspace traffic, four to eight k-blocks of a
// 64-edge tile; cutting 32-edge tiles, 0.13 us a k-block, pays only for longer pieces).
inline F64Plan f64_plan(int n, int bt, bool resp, int sms) {
  F64Plan pl;
  pl.bt = bt;
  pl.tiles = (n + bt - 1) / bt;
  const int kb = (n + 15) / 16, min_units = bt == 32 ? 24 : 8;
  const long long tiles = (long long)pl.tiles * (pl.tiles + 1) / 2;
  const long long units = tiles * kb * (resp ? 3 : 1), jobs = tiles * (resp ? 2 : 1);
  pl.snap = 4;
  pl.grid = (int)std::min<long long>(sms, std::max(jobs, units / min_units));
  return pl;
}

// Tile edge of an order-n solve, a rule on n alone: the pieces of cut tiles depend on it, and
// so the last bits of a result, which are to be the same in every process.  32 up to 416, where
// 64-edge tiles are too few for the SMs (n = 300: 235 us a solve with 32, 270 us with 64;
// n = 500: 296 and 284).  128 from 4096 on, without a response (its tile of sums does not fit
// beside the stages): eight steps at n = 3000 take 7.49 ms with 128 and 7.12 with 64, at 4096
// 17.40 and 17.55, at 8192 134.3 and 137.7, at 12288 447 and 477.
inline int f64_edge(int n, bool resp) { return n <= 416 ? 32 : n < 4096 || resp ? 64 : 128; }

// Steps per launch, so that a long solve leaves the GPU to others in between: a launch of more
// than one step takes about a tenth of a second at most.  Large steps cost their products (30
// TFLOP/s of symmetric ones), the smallest their fixed 6 us, up to 25 at n = 740.
inline int f64_steps_per_launch(int n, bool resp) {
  const double flops = (double)n * n * n * (resp ? 3.0 : 1.0);
  return (int)std::max(1.0, std::min(5e3, 2e12 / flops));
}

constexpr int kF64Sums = 5;   // ||X'||^2, Tr X', ||X - X^2||^2 (core rows), Tr X^2, Tr Delta'

// Workspace of a launch, in doubles: one piece per CTA, the partial sums of two steps, then
// a flag per CTA and the barrier counter.
inline size_t f64_plan_doubles(const F64Plan& pl) {
  return (size_t)pl.grid * pl.bt * pl.bt + 2 * (size_t)pl.grid * kF64Sums + pl.grid / 2 + 2;
}

// Workspace that covers every launch of order n.  With a response also the launches without
// one: a set-up for X and Delta serves passes over X alone too (SP2-Fermi generates its
// sequence that way).
inline size_t f64_solve_doubles(int n, bool resp, int sms) {
  const size_t w = f64_plan_doubles(f64_plan(n, f64_edge(n, false), false, sms));
  return resp ? std::max(w, f64_plan_doubles(f64_plan(n, f64_edge(n, true), true, sms))) : w;
}

// ---- INT8 residue products (k_oz_gemm) ----
// INT8 residue products of nb x nb 128-blocks: {plane, 128-row block, first 128-column
// block, 128-column blocks} for a persistent grid (returned: its CTAs), CTA c taking the entries c,
// c + grid, ... until one with no blocks.  Upper 128-blocks of every plane: pairs of column
// blocks as 128 x 256 tiles, the odd one left (the first at or right of the diagonal in odd
// row blocks, the last of an odd count) as a 128 x 128 tile.  Wide tiles go first in panels
// of kOzPanel column pairs, row blocks top to bottom inside a panel, so one wave shares few
// operand row blocks (their K-slices stay in L2).  The wide tiles past the last whole wave
// and the narrow ones are then dealt to the CTA with the least work, the wide ones cut in
// two when every CTA can have one half.  In 128 x 128 tiles per SM: n = 2744 takes 16 (15.4
// on average) where 1188 wide tiles took nine waves, 18; n = 1000 takes 3 instead of 4.
constexpr int kOzPanel = 6;
inline int oz_work_items(int nb, int planes, int sms, std::vector<int4>& out) {
  std::vector<int4> wide, narrow;
  for (int t = 0; t < planes; ++t)
    for (int p0 = 0; p0 < nb; p0 += 2 * kOzPanel) {
      const int p1 = std::min(nb, p0 + 2 * kOzPanel);
      for (int bi = 0; bi < p1; ++bi) {
        int c = std::max(p0, bi);
        if (c & 1) {   // an odd first block: alone
          narrow.push_back(make_int4(t, bi, c, 1));
          ++c;
        }
        for (; c + 1 < p1; c += 2) wide.push_back(make_int4(t, bi, c, 2));
        if (c < p1) narrow.push_back(make_int4(t, bi, c, 1));
      }
    }
  const int grid = (int)std::min<size_t>(2 * wide.size() + narrow.size(), (size_t)sms);
  const size_t whole = wide.size() / grid * grid;
  out.assign(wide.begin(), wide.begin() + whole);
  const size_t rest = wide.size() - whole;
  const bool cut = 2 * rest + narrow.size() <= (size_t)grid;
  std::vector<std::vector<int4>> tail(grid);
  std::vector<int> load(grid, 0);
  auto deal = [&](const int4& w) {
    const int c = (int)(std::min_element(load.begin(), load.end()) - load.begin());
    tail[c].push_back(w);
    load[c] += w.w;
  };
  for (size_t i = whole; i < wide.size(); ++i) {
    int4 w = wide[i];
    if (cut) {
      w.w = 1;
      deal(w);
      ++w.z;
    }
    deal(w);
  }
  for (const int4& w : narrow) deal(w);
  size_t rounds = 0;
  for (const auto& v : tail) rounds = std::max(rounds, v.size());
  for (size_t r = 0; r < rounds; ++r)
    for (int c = 0; c < grid; ++c)
      out.push_back(r < tail[c].size() ? tail[c][r] : make_int4(0, 0, 0, 0));
  return grid;
}

// ---- paired split-precision products (k_tc_pair) ----
constexpr int kPairNarrow = 1 << 24;   // marks a 64-column tile in a list of wider ones

// Tiles of the paired kernel, {bi2, bj} with bj >= 2 bi2 (128-column blocks), in panels of
// kPanel column blocks (row pairs top to bottom inside a panel).
inline void pair_tile_order(int nb, int panel, std::vector<int2>& out) {
  out.clear();
  for (int p0 = 0; p0 < nb; p0 += panel) {
    const int p1 = std::min(nb, p0 + panel);
    for (int bi2 = 0; 2 * bi2 < p1; ++bi2)
      for (int bj = std::max(2 * bi2, p0); bj < p1; ++bj) out.push_back(make_int2(bi2, bj));
  }
}
inline int pair_tile_count(int nb) {
  const int np2 = (nb + 1) / 2;
  return nb * np2 - np2 * (np2 - 1);   // row pair bi2 has the column blocks from 2 bi2 on
}

// The first `whole` tiles, then the others as two 64-column tiles each (y in 64-column
// blocks), marked kPairNarrow in .x when `mark`.
inline void pair_work_items(int nb, int panel, int whole, bool mark, std::vector<int2>& out) {
  std::vector<int2> blocks;
  pair_tile_order(nb, panel, blocks);
  out.clear();
  for (size_t i = 0; i < blocks.size(); ++i) {
    int2 q = blocks[i];
    if ((int)i < whole) {
      out.push_back(q);
      continue;
    }
    if (mark) q.x |= kPairNarrow;
    out.push_back(make_int2(q.x, 2 * q.y));
    out.push_back(make_int2(q.x, 2 * q.y + 1));
  }
}

}  // namespace sp2b
