// Driver for the row order of the multi-row SpMM (fasteig_b200/csrc/spmm_grid.hpp).
// "deal": reads rows, grid strides s1 and s2, groups of a CTA; deals the operator's rows as
// the kernel does and prints how many were dealt other than once, out of range, and the share
// of the groups' slots that have a row. "place": the order and the last row of a plane's last
// brick for the same four numbers (any size). "find": reads rows, the number of windows and, for
// each, its first row, row count, row lengths and columns; prints the strides found and
// the kind of the rows.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../fasteig_b200/csrc/spmm_grid.hpp"

static long long next() {
  long long v = 0;
  if (std::scanf("%lld", &v) != 1) std::exit(2);
  return v;
}

int main(int argc, char** argv) {
  if (argc != 2) return 2;
  if (!std::strcmp(argv[1], "find")) {
    const int64_t rows = next();
    const int count = static_cast<int>(next());
    std::vector<std::vector<int32_t>> rp(count), ci(count);
    std::vector<fe::RowWindow> w;
    for (int i = 0; i < count; ++i) {
      const int64_t row0 = next();
      const int n = static_cast<int>(next());
      rp[i].push_back(7);  // windows start anywhere in the operator's entries
      for (int r = 0; r < n; ++r) rp[i].push_back(rp[i].back() + static_cast<int32_t>(next()));
      for (int e = 7; e < rp[i].back(); ++e) ci[i].push_back(static_cast<int32_t>(next()));
      w.push_back({rp[i].data(), ci[i].data(), row0, n});
    }
    const fe::RowPattern p = fe::find_pattern(w, rows);
    std::printf("%d %d %d\n", p.s1, p.s2, static_cast<int>(p.kind));
    return 0;
  }
  const int64_t rows = next();
  const int g1 = static_cast<int>(next()), g2 = static_cast<int>(next());
  const int groups = static_cast<int>(next());
  const fe::RowOrder o = fe::row_order(g1, g2, groups);
  const long long bricks = static_cast<long long>(o.nx) * o.ny;
  auto row = [&](long long brick, int group, int64_t plane) -> int64_t {
    const fe::RowPlace p = fe::row_place(static_cast<int>(brick), group, o.lbx, o.by, o.nx, o.ny);
    if (p.z != 0 || p.x >= o.s1 || p.y >= o.lines) return -1;
    return p.x + static_cast<int64_t>(o.s1) * p.y + plane * o.s2;
  };
  if (!std::strcmp(argv[1], "place")) {
    int64_t last = -1;
    for (int g = 0; g < groups; ++g) last = std::max(last, row(bricks - 1, g, 0));
    std::printf("%d %d %d %d %lld %lld\n", o.s1, o.s2, o.lines, 1 << o.lbx, bricks,
                static_cast<long long>(last));
    return 0;
  }
  std::vector<int> seen(rows, 0);
  long long slots = 0, dealt = 0, outside = 0;
  for (int64_t plane = 0; plane * o.s2 < rows; ++plane)
    for (long long brick = 0; brick < bricks; ++brick)
      for (int g = 0; g < groups; ++g) {
        ++slots;
        const int64_t r = row(brick, g, plane);
        if (r < 0) continue;
        if (r >= (plane + 1) * o.s2) ++outside;
        if (r >= rows) continue;
        ++seen[r];
        ++dealt;
      }
  long long wrong = 0;
  for (int v : seen) wrong += v != 1;
  std::printf("%lld %lld %.6f\n", wrong, outside, static_cast<double>(dealt) / slots);
  return 0;
}
