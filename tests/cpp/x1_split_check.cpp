// Host check of csrc/x1_split.cuh over every column length up to the longest
// that a block may have, the column counts of lines, planes and boxes, both
// forms' limits, the shares of the chip that an ensemble's members get and the
// columns per item that a caller may ask for.
// Prints "splits <n> faults <n>" and the first faults.
#include <cstdio>

#include "../../snapy_linfel_b200/csrc/x1_split.cuh"

using namespace snapb;

static long splits = 0, faults = 0;

static void fault(const char* what, int nx1, int ng, long ncol, const X1Split& s) {
  if (faults++ < 8)
    printf("%s: nx1 %d ng %d columns %ld -> K %d nseg %d seglen %d pitch %d\n", what, nx1, ng, ncol,
           s.K, s.nseg, s.seglen, s.pitch);
}

static void check(const X1Split& s, int nx1, int ng, long ncol) {
  ++splits;
  const int nc1 = nx1 + 2 * ng, il = ng, iu = ng + nx1 - 1;
  if (s.K < 1 || s.K > 32) fault("columns of an item", nx1, ng, ncol, s);
  if (s.K > 1 && s.nseg > 1) fault("segments of several columns", nx1, ng, ncol, s);
  int cells = 0;
  for (int seg = 0; seg < s.nseg; ++seg) {
    // the item's cells and rows, as the kernels form them
    const int c0 = il + seg * s.seglen, c1 = c0 + s.seglen < iu + 1 ? c0 + s.seglen : iu + 1;
    const bool bottom = c0 == il, top = c1 == iu + 1;
    const int lo = bottom ? 0 : c0 - 3, n = (top ? nc1 : c1 + 3) - lo;
    if (c1 <= c0) fault("empty segment", nx1, ng, ncol, s);
    cells += c1 - c0;
    if (s.K * n > s.pitch) fault("row shorter than its cells", nx1, ng, ncol, s);
    // the windows of cells c0 - 1 .. c1 stay in the rows, and only the item that
    // revises a wall's ghosts reads them
    if (c0 - 3 < lo || c1 + 2 >= lo + n) fault("window outside the rows", nx1, ng, ncol, s);
    if (!bottom && c0 - 3 < il) fault("lower ghosts read by another item", nx1, ng, ncol, s);
    if (!top && c1 + 2 > iu) fault("upper ghosts read by another item", nx1, ng, ncol, s);
  }
  if (cells != nx1) fault("cells missing", nx1, ng, ncol, s);
}

int main() {
  const long columns[] = {1, 9, 10, 13, 20, 26, 38, 49, 64, 70, 81, 107, 128, 262, 518, 1030, 4900, 20000};
  for (int ng : {3, 4, 8})
    for (int nvt : {5, 6, 8})
      for (int nx1 = ng; (2 * nvt + 2) * (nx1 + 2 * ng) * 4 <= 200 * 1024; ++nx1)
        for (long ncol : columns) {
          if ((2 * nvt + 2) * (nx1 + 2 * ng) * 8 <= 200 * 1024)
            check(x1_split(nx1, ng, ncol, nvt, 8, 14 * 1024, 148. * 16., false), nx1, ng, ncol);
          for (double share : {1., 0.3, 0.02})
            check(x1_split(nx1, ng, ncol, nvt, 4, 7 * 1024, 148. * 24. * share, false), nx1, ng,
                  ncol);
          for (bool whole : {false, true}) {
            const X1Split rule = x1_split(nx1, ng, ncol, nvt, 4, 7 * 1024, 148. * 24., whole);
            check(rule, nx1, ng, ncol);
            if (ncol != 1030) continue;
            for (int columns : {1, 2, 7, 16, 31, 32, 33, 64, 1000})
              check(x1_split_columns(rule, nx1, ng, nvt, 4, columns, whole), nx1, ng, ncol);
          }
        }
  printf("splits %ld faults %ld\n", splits, faults);
  return 0;
}
