// x1_split.cuh — the split of the x1 sweep over warps (host code; needs no CUDA).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace snapb {

// An item is either K whole columns (consecutive, so their cells are one
// contiguous span per variable) or one of nseg segments of seglen cells of a
// single column.
struct X1Split {
  int K, nseg, seglen;
  int pitch;  // elements per variable row in the warp's shared memory
};

// Fewest cells of a column's last segment.  A segment's faces take cells up to
// two above its upper face's, and only the item that holds a wall's own cells
// revises the wall's ghosts: with one or two cells in the last segment, the one
// below it would read ghosts as the boundary fill left them.
constexpr int kX1LastCells = 3;

// The split for columns of nx1 cells and ng ghosts at each end, ncol of them
// (ghost columns included): rows of nvt variables of at most row_bytes a warp
// where some split has them, `resident` warps on the GPU at once (whole: no
// segments).
//
// A warp's time is about one unit per round of 32 cells, a third of one per 32
// cells converted, and a start-up; the FP64 form's 16 warps per SM are resident
// when a warp's rows stay within 14 KB.  Packing K short columns end to end
// fills the last round of each column (64 layers alone: 66 cells in 3 rounds,
// 69 %; five columns: 330 in 11, 94 %); segments of a column spread a few long
// columns over the SMs (1024 cells of a 1-D block: one CTA took 43 us).
inline X1Split x1_split(int nx1, int ng, int64_t ncol, int nvt, size_t item, size_t row_bytes,
                        double resident, bool whole) {
  const int nc1 = nx1 + 2 * ng;
  X1Split best{1, 1, nx1, nc1};
  double best_cost = 0.;
  size_t best_bytes = 0;
  auto consider = [&](X1Split s, int n, int nn) {
    const int64_t items = (ncol + s.K - 1) / s.K * s.nseg;
    const size_t bytes = (size_t)s.pitch * nvt * item;
    const double waves = std::max(1., items / resident + 0.5);
    const double cost = waves * (1. + (s.K * nn + 31) / 32 + ((s.K * n + 31) / 32) / 3.);
    const bool fits = bytes <= row_bytes, best_fits = best_bytes <= row_bytes;
    if (best_bytes == 0 || (fits && !best_fits) ||
        (fits == best_fits && (fits ? cost < best_cost : bytes < best_bytes))) {
      best = s;
      best_cost = cost;
      best_bytes = bytes;
    }
  };
  for (int K = 1; K <= 8; ++K) consider({K, 1, nx1, K * nc1}, nc1, nx1 + 2);
  for (int want = 2; !whole && want <= (nx1 + 29) / 30; ++want) {
    const int S = (nx1 + want - 1) / want, nseg = (nx1 + S - 1) / S;
    if (nseg > 1 && nx1 - (nseg - 1) * S >= kX1LastCells)
      consider({1, nseg, S, S + ng + 3}, S + 6, S + 2);
  }
  return best;
}

// Most whole columns of an item: a warp marks the interior ones of them in one
// word, a bit each.
constexpr int kX1MaxColumns = 32;

// `columns` whole columns per item instead of the rule's split, as many of them
// as an item takes and 48 KB of rows hold; the rule's where not one fits (whole:
// one all the same).
inline X1Split x1_split_columns(const X1Split& rule, int nx1, int ng, int nvt, size_t item,
                                int columns, bool whole) {
  const int nc1 = nx1 + 2 * ng, fit = (int)((48 * 1024) / ((size_t)nvt * nc1 * item));
  if (fit < 1 && !whole) return rule;
  const int K = std::max(1, std::min({columns, fit, kX1MaxColumns}));
  return X1Split{K, 1, nx1, K * nc1};
}

}  // namespace snapb
