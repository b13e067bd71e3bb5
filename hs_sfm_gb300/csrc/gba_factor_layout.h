// gba_factor_layout.h -- who owns which tile in the dataflow factorization
// (k_chol_dataflow).  Host code without CUDA, so that it can be checked for any
// number of SMs.
#pragma once

#include <algorithm>
#include <vector>

namespace gba {

// Tiles of row i kept by its own CTA: (i, i), (i, i-1) and, in FP32, (i, i-2).
// An FP64 update takes 8 us of one SM's FP64 pipe, so a third tile would make
// the row's updates slower than the chain they have to keep ahead of.
constexpr int df_row_tiles(bool mixed) { return mixed ? 3 : 2; }
// Tiles kept by row i's second CTA, left of those.
constexpr int df_helper_tiles(bool mixed) { return mixed ? 3 : 0; }
// Most tiles of a worker CTA beside row CTAs: a lane for each in two warps.
constexpr int kDfWorkerTiles = 64;

struct DfTile {
  int i, j;
};

struct DfLayout {
  int grid = 0;
  int rows = 0;      // CTAs 0 .. rows - 1 keep the last tiles of their row (nt, or 0)
  int helpers = 0;   // the next `helpers` keep the tiles left of those (nt, or 0)
  int max_own = 0;
  std::vector<std::vector<DfTile>> own;   // each CTA's tiles, sorted by (j, i)
};

// The layout of an nt-tile system (nt >= 2) on `sms` SMs.  Row i's last tiles
// go to CTA i mod grid; the rest, heaviest first, to the CTA with the least
// work so far.  When there are at least twice as many CTAs as tile rows, the
// rows' CTAs take none of the rest (and run the rows' fixed program): a CTA
// busy with an update when its row's chain task becomes ready would delay the
// chain by that update.  With at least four times as many (FP32) a second CTA
// of each row keeps the tiles left of the first one's, and as many CTAs as
// both remain for the rest.
inline DfLayout df_layout(int nt, bool mixed, int sms) {
  DfLayout l;
  const long long ntiles = (long long)nt * (nt + 1) / 2;
  const int G = int(std::min<long long>(sms, ntiles));
  l.grid = G;
  l.own.resize(G);
  const bool dedicated = G >= 2 * nt;
  const int row_tiles = dedicated ? df_row_tiles(mixed) : 2;
  const int helper_tiles = G >= 4 * nt ? df_helper_tiles(mixed) : 0;
  const int band = row_tiles + helper_tiles;   // tiles of a row kept by its own CTAs
  l.rows = dedicated ? nt : 0;
  l.helpers = helper_tiles > 0 ? nt : 0;
  const int first_worker = l.rows + l.helpers;
  std::vector<long long> load(G, 0);
  for (int i = 0; i < nt; ++i) {
    const int g = i % G;
    for (int u = 0; u < row_tiles && u <= i; ++u) {
      l.own[g].push_back({i, i - u});
      load[g] += i - u + 1;
    }
    for (int u = row_tiles; u < band && u <= i; ++u) l.own[nt + i].push_back({i, i - u});
  }
  for (int j = nt - 1; j >= 0; --j)
    for (int i = j + band; i < nt; ++i) {
      int g = first_worker;
      for (int h = first_worker + 1; h < G; ++h)
        if (load[h] < load[g]) g = h;
      l.own[g].push_back({i, j});
      load[g] += j + 1;
    }
  for (auto& o : l.own) {
    std::sort(o.begin(), o.end(), [](const DfTile& a, const DfTile& b) { return a.j != b.j ? a.j < b.j : a.i < b.i; });
    l.max_own = std::max(l.max_own, int(o.size()));
  }
  return l;
}

}  // namespace gba
