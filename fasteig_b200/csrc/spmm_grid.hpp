// What an operator's rows are like, for the dispatch and the row order of spmm_rows.cu.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

namespace fe {

// What an operator's rows are like: a grid's, the same offsets from row to row without a grid,
// other offsets in each row (most entries near the diagonal, or far from it). Unknown for
// operators put together from others.
enum class RowKind : uint8_t { kUnknown, kGrid, kBanded, kIrregular, kScattered };

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
