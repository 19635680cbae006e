// Host-side checks of how the persistent kernels' work is dealt (work_lists.h), built by
// tests/test_work_lists.py with the host C++ compiler.  Each returns 0 or the number of the
// check that failed.
#include <set>
#include <tuple>

#include "work_lists.h"

using namespace sp2b;

// Every k-block of every tile of an order-n FP64 step belongs to one CTA; the pieces that a
// tile's last holder looks for (k_f64_solve's list) are exactly the ones the CTAs before it
// leave, one per CTA, and fit its list.
extern "C" int check_f64(int n, int bt, int resp, int sms) {
  const F64Plan pl = f64_plan(n, bt, resp != 0, sms);
  F64Split s;
  s.kb = (n + 15) / 16;
  s.ntiles = pl.tiles * (pl.tiles + 1) / 2;
  s.snap = pl.snap;
  s.G = pl.grid;
  s.total = (long long)s.ntiles * s.kb * (resp ? 3 : 1);
  if (pl.grid < 1 || pl.grid > sms) return 1;
  if (s.bound(0) != 0 || s.bound(s.G) != s.total) return 2;
  for (int c = 0; c < s.G; ++c) {
    const long long u0 = s.bound(c), u1 = s.bound(c + 1);
    if (u1 < u0) return 3;
    int ja, oa, jb, ob;
    s.locate(u0, ja, oa);
    s.locate(u1, jb, ob);
    if (ob >= (u1 < s.total ? s.len(jb) : 1) || oa < 0) return 4;
    if (u1 == u0 || ja == jb || oa == 0) continue;
    // the owner of tile ja's end: pieces back to the tile's start, without a gap
    long long at = u0;
    int pieces = 0;
    for (int q = c - 1; q >= 0 && at > u0 - oa; --q) {
      const long long lo = s.bound(q), hi = s.bound(q + 1);
      if (hi != at) return 5;
      if (lo == hi) continue;
      int jl, ol, jh, oh;
      s.locate(lo, jl, ol);
      s.locate(hi, jh, oh);
      if (jh != ja || oh == 0) return 6;   // its open piece lies in this tile
      at = std::max(lo, u0 - oa);
      if (++pieces > kMaxPieces) return 7;
    }
    if (at != u0 - oa) return 8;
  }
  return 0;
}

// The workspace of an order-n set-up holds every launch that may use it: with a response both
// the launches with it and those without, at the edge each of them takes.
extern "C" int check_f64_workspace(int n, int resp, int sms) {
  const size_t have = f64_solve_doubles(n, resp != 0, sms);
  for (int r = 0; r <= resp; ++r) {
    const int bt = f64_edge(n, r != 0);
    const F64Plan pl = f64_plan(n, bt, r != 0, sms);
    // pieces, sums of two steps, flags and the barrier counter
    const size_t words = (size_t)pl.grid + 1;
    if ((size_t)pl.grid * bt * bt + 10 * (size_t)pl.grid + (words + 1) / 2 > have) return 1 + r;
  }
  return 0;
}

// Milliseconds of the longest launch of order n: 6 us a step and its products at 30 TFLOP/s
// (0 when a launch is one step).
extern "C" double f64_launch_ms(int n, int resp) {
  const int steps = f64_steps_per_launch(n, resp != 0);
  const double flops = (double)n * n * n * (resp ? 3.0 : 1.0);
  return steps <= 1 ? 0.0 : 1e3 * steps * (6e-6 + flops / 30e12);
}

// Every upper 128-block of every plane once, lists without holes, tiles inside the matrix.
extern "C" int check_oz(int nb, int planes, int sms) {
  std::vector<int4> w;
  const int grid = oz_work_items(nb, planes, sms, w);
  if (grid < 1 || grid > sms || w.size() % grid) return 1;
  std::set<std::tuple<int, int, int>> seen;
  std::vector<char> ended(grid, 0);
  for (size_t i = 0; i < w.size(); ++i) {
    if (w[i].w == 0) {
      ended[i % grid] = 1;
      continue;
    }
    if (ended[i % grid] || w[i].w > 2) return 2;
    for (int b = 0; b < w[i].w; ++b) {
      if (w[i].z + b >= nb || w[i].z + b < w[i].y) return 3;
      if (!seen.insert({w[i].x, w[i].y, w[i].z + b}).second) return 4;
    }
  }
  return seen.size() == (size_t)planes * nb * (nb + 1) / 2 ? 0 : 5;
}

// Every 64-column block of every row pair from its diagonal on once, for any number of
// whole tiles.
extern "C" int check_pair(int nb, int whole, int mark) {
  std::vector<int2> t;
  pair_work_items(nb, 12, whole, mark != 0, t);
  const int count = pair_tile_count(nb);
  if ((int)t.size() != whole + 2 * (count - whole)) return 1;
  std::set<std::pair<int, int>> seen;
  for (size_t i = 0; i < t.size(); ++i) {
    const bool narrow = (int)i >= whole;
    if (mark && narrow != ((t[i].x & kPairNarrow) != 0)) return 2;
    const int bi2 = t[i].x & (kPairNarrow - 1), y = narrow ? t[i].y : 2 * t[i].y;
    for (int h = 0; h < (narrow ? 1 : 2); ++h) {
      if (y + h >= 2 * nb || y + h < 4 * bi2) return 3;
      if (!seen.insert({bi2, y + h}).second) return 4;
    }
  }
  return (int)seen.size() == 2 * count ? 0 : 5;
}
