// Driver for the row patterns of the multi-row SpMM (fasteig_b200/csrc/spmm_grid.hpp).
// "find": reads rows, the number of windows and, for each, its first row, row count, row
// lengths and columns; prints the strides found and the kind of the rows.
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
  return 2;
}
