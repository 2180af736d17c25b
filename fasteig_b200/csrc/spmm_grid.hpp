// The order in which spmm_rows.cu deals an operator's rows to its groups of lanes: host code,
// and the index function that the kernel shares with it.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define FE_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FE_HOST_DEVICE inline
#endif

namespace fe {

// What an operator's rows are like: a grid's, the same offsets from row to row without a grid,
// other offsets in each row (most entries near the diagonal, or far from it). Unknown for
// operators put together from others.
enum class RowKind : uint8_t { kUnknown, kGrid, kBanded, kIrregular, kScattered };

// How a CTA's groups go through the rows. Neighbours that lie a plane apart are read again
// while a sweep down the planes still has them; with a grid of lines only the same holds from
// line to line. Small planes, short lines and operators without a grid are taken in runs of
// consecutive rows, which L1 or L2 holds anyway (us, FP32 step of 64 columns, bricks and runs:
// 10 x 10 x 4000 104, 82; 5 x 5 x 12000 with 13 points 133, 79; but 16 x 16 x 1500 76, 82).
// Lines of up to 2,047 rows are swept several at a time (600 x 600, 200 columns: 191 so, 211
// in runs), longer ones singly (40000 x 8, 320 columns: 233 so, 311 in runs).
enum class Sweep { kPlanes, kLines, kRuns };
constexpr int kMinPlane = 256, kMinLine = 128;
constexpr int kSmallPlane = 800;  // below, wide rows gain little from a sweep
constexpr int kLongLine = 2048;   // from here a sweep takes one line at a time

inline Sweep row_sweep(int grid_s1, int grid_s2) {
  if (grid_s2 >= kMinPlane) return Sweep::kPlanes;
  if (grid_s2 == 0 && grid_s1 >= kMinLine) return Sweep::kLines;
  return Sweep::kRuns;
}

// Rows are numbered by planes of s2 rows, planes by lines of s1 (s2 a multiple of s1). A CTA's
// groups take a brick of 2^lbx rows of neighbouring lines, and sweep down the planes below it.
struct RowOrder {
  int s1, s2, lines;  // lines of a plane
  int lbx, by;        // log2 of a brick's rows along a line, lines of a brick
  int nx, ny;         // bricks along a line and across a plane
};

// Where group `group` of brick `brick` starts.
struct RowPlace {
  int x, y, z;  // row of the line, line of the plane, step of the sweep's start
};
FE_HOST_DEVICE RowPlace row_place(int brick, int group, int lbx, int by, int nx, int ny) {
  const int bx = brick % nx, byz = brick / nx;
  return {(bx << lbx) + (group & ((1 << lbx) - 1)), byz % ny * by + (group >> lbx), byz / ny};
}

// Bricks of four rows of a line by groups / 4 lines, or, where more than a quarter of the
// groups would have no row (lines or planes of a few rows), the shape that leaves fewest idle.
inline RowOrder row_order(int grid_s1, int grid_s2, int groups) {
  RowOrder o{groups, groups, 1, 0, 1, 1, 1};
  const Sweep sweep = row_sweep(grid_s1, grid_s2);
  if (sweep != Sweep::kRuns) {
    o.s1 = grid_s1;
    o.lines = sweep == Sweep::kPlanes ? grid_s2 / grid_s1
                                      : grid_s1 < kLongLine ? std::max(1, groups / 4) : 1;
    o.s2 = o.s1 * o.lines;
  }
  auto shape = [&](int lbx) {
    o.lbx = lbx;
    o.by = groups >> lbx;
    o.nx = (o.s1 - 1) / (1 << lbx) + 1;
    o.ny = (o.lines - 1) / o.by + 1;
    return static_cast<double>(o.s2) / groups / o.nx / o.ny;  // share of groups with a row
  };
  if (o.lines > 1 && shape(2) >= 0.75) return o;
  int best = 0;
  double most = 0.0;
  for (int lbx = 0; (1 << lbx) <= groups; ++lbx)
    if (const double used = shape(lbx); used >= most) {
      most = used;
      best = lbx;
    }
  shape(best);
  return o;
}

// Line and plane strides of the grid behind one row's column offsets, taken without their
// signs (a row on the grid's edge has its neighbours on one side only): runs of offsets that
// differ by 1 are one neighbour along the line (s1: the centre of the first run past the
// line's own neighbours), runs of those that differ by up to two lines one plane.
inline void grid_strides(const int32_t* cols, int count, int64_t row, int64_t rows, int* s1,
                         int* s2) {
  *s1 = *s2 = 0;
  std::vector<int> d;
  for (int i = 0; i < count; ++i)
    if (cols[i] != row) d.push_back(static_cast<int>(cols[i] > row ? cols[i] - row : row - cols[i]));
  std::sort(d.begin(), d.end());
  size_t i = 0;
  while (i < d.size() && d[i] < 4) ++i;
  if (i == d.size()) return;
  size_t j = i;
  while (j + 1 < d.size() && d[j + 1] - d[j] <= 1) ++j;
  const int line = d[i] + (d[j] - d[i]) / 2;
  if (line < 4 || line > rows / 2) return;
  *s1 = line;
  i = j + 1;
  while (i < d.size() && d[i] <= 3 * static_cast<int64_t>(line)) ++i;
  if (i == d.size()) return;
  j = i;
  while (j + 1 < d.size() && d[j + 1] - d[j] <= 2 * static_cast<int64_t>(line) + 2) ++j;
  const int plane = d[i] + (d[j] - d[i]) / 2;
  if (plane % line == 0 && plane <= rows / 2) *s2 = plane;
}

// A few consecutive rows of an operator: their row pointers (count + 1) and column indices.
struct RowWindow {
  const int32_t* rowptr;
  const int32_t* colind;  // of entry rowptr[0]
  int64_t row0;
  int count;
};

struct RowPattern {
  int s1 = 0, s2 = 0;  // rows from line to line, from plane to plane; 0: none seen
  RowKind kind = RowKind::kUnknown;
};
constexpr int64_t kNearDiagonal = 4096;

// The pattern behind an operator, from windows of its rows: the strides that the longest
// row suggests, if three quarters of all the rows have an entry that far before or behind
// their diagonal. (One row of a scattered or permuted operator suggests strides as well: 994
// of 1000 random rows of seven entries do.)
inline RowPattern find_pattern(const std::vector<RowWindow>& windows, int64_t rows) {
  RowPattern p;
  const RowWindow* at = nullptr;
  int best = 0;
  for (const RowWindow& w : windows)
    for (int i = 0; i < w.count; ++i)
      if (!at || w.rowptr[i + 1] - w.rowptr[i] > at->rowptr[best + 1] - at->rowptr[best]) {
        at = &w;
        best = i;
      }
  if (!at) return p;
  grid_strides(at->colind + (at->rowptr[best] - at->rowptr[0]),
               at->rowptr[best + 1] - at->rowptr[best], at->row0 + best, rows, &p.s1, &p.s2);
  int64_t all = 0, with_s1 = 0, with_s2 = 0, entries = 0, near = 0, again = 0;
  std::vector<int64_t> last, offsets;
  for (const RowWindow& w : windows)
    for (int i = 0; i < w.count; ++i, ++all) {
      bool has1 = false, has2 = false;
      last.swap(offsets);
      if (i == 0) last.clear();
      offsets.clear();
      for (int32_t e = w.rowptr[i]; e < w.rowptr[i + 1]; ++e, ++entries) {
        const int64_t c = w.colind[e - w.rowptr[0]], r = w.row0 + i, d = c > r ? c - r : r - c;
        has1 = has1 || d == p.s1;
        has2 = has2 || d == p.s2;
        near += d <= kNearDiagonal;
        offsets.push_back(c - r);
        again += std::find(last.begin(), last.end(), c - r) != last.end();
      }
      with_s1 += has1;
      with_s2 += has2;
    }
  if (4 * with_s1 < 3 * all) p.s1 = 0;
  if (p.s1 == 0 || 4 * with_s2 < 3 * all) p.s2 = 0;
  p.kind = p.s1 > 0                ? RowKind::kGrid
           : 2 * again >= entries ? RowKind::kBanded
           : 2 * near >= entries  ? RowKind::kIrregular
                                  : RowKind::kScattered;
  return p;
}

}  // namespace fe
