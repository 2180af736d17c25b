// Block SpMM and Chebyshev step with several rows to a warp, over bricks of the grid that
// the operator's diagonals show (sm_100a).
//
// A group of G lanes owns a row and reads up to three 16-byte vectors a lane, so a warp works
// on 32 / G rows of one column panel. What bounds it, after DRAM, is the instructions and the
// load-store wavefronts of an SM rather than the bytes: one warp per row with 8-byte lanes
// spends them on a row of few columns as on a wide one (96^3 grid, 7 points, FP32 step of 64
// columns: 380 us so, 146 us here, 113 us of DRAM traffic at the copy rate). Hence 16-byte
// lanes, byte pitches in 32 bits (one wide multiply-add per address), few lanes to a row, and
// no predicates where the rows of the warp have as many entries.
//
// Rows are dealt out in bricks: a CTA's groups take bx x by rows of neighbouring lines and
// sweep down bz planes, so that the neighbours along a line, across lines and from plane to
// plane are read while L1 still holds them: 57 % of the loads hit L1 against 24 % for
// consecutive rows (128^3, FP32 step of 320 columns: 1.91 ms with one warp per row, 2.35 ms
// with consecutive rows here, 1.67 ms in bricks, 1.27 ms of DRAM traffic). The brick is
// only an order (spmm_grid.hpp): any strides s1 (line) and s2 (plane, a multiple of s1)
// number every row once.
//
// A row's arithmetic is that of the kernel of spmm.cu which such a block would have there,
// bit for bit: with FOLD, alpha and gamma are folded into the coefficients (the row
// kernel); without, they are applied to the finished sum (the loop kernel), which is the
// more exact of the two over a filter's steps (13 points, degree 16, FP32: 8.8e-8 off the
// 64-bit result against 3.3e-7).

#include "fe_common.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace fe {
namespace {

template <typename T, int VEC>
struct __align__(VEC * sizeof(T)) Lane {
  T v[VEC];
};
template <typename T, int VEC>
struct LaneRaw;
template <> struct LaneRaw<float, 4> { using type = float4; };
template <> struct LaneRaw<float, 2> { using type = float2; };
template <> struct LaneRaw<float, 1> { using type = float; };
template <> struct LaneRaw<double, 2> { using type = double2; };
template <> struct LaneRaw<double, 1> { using type = double; };

template <typename T>
struct RowsParams {
  const int32_t* rowptr;
  const int32_t* colind;
  const T* vals;
  const T* X;
  T* Y;
  const T* Z;
  const T* R;
  const T* delta;
  int ldx, ldy, ldz, ldr;  // bytes from row to row
  int nrows, last_x;       // rows; the last row of X
  int ncols, pc, panels;   // columns of the block and of a panel, panels
  int s1, s2, lines;       // order of the rows (RowOrder)
  int lbx, nx, ny;
  int bz;                  // planes that a brick sweeps down
  T alpha, gamma, beta;
  int use_gamma, use_beta;
};

template <typename T, int VEC>
__device__ __forceinline__ Lane<T, VEC> load_ro(const T* p) {
  using R = typename LaneRaw<T, VEC>::type;
  return __builtin_bit_cast(Lane<T, VEC>, __ldg(reinterpret_cast<const R*>(p)));
}

constexpr int kRowsThreads = 256;

// G lanes a row, CPL vectors of VEC values a lane, up to M G entries a row, KC neighbours in
// flight. FOLD: alpha and gamma in the coefficients. TAIL: the columns end inside a vector.
// CORR: + delta[j] R[row, j].
template <typename T, int VEC, int G, int CPL, int M, int KC, bool FOLD, bool TAIL, bool CORR>
__global__ void __launch_bounds__(kRowsThreads, 4)
spmm_rows_kernel(const __grid_constant__ RowsParams<T> P) {
  using V = Lane<T, VEC>;
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int NG = kRowsThreads / G;
  const int lane = threadIdx.x & 31;
  const int gl = threadIdx.x % G;
  const int grp = threadIdx.x / G;
  const int panel = blockIdx.x % P.panels;  // panels side by side: whole rows from DRAM
  const int brick = blockIdx.x / P.panels;
  const RowPlace at0 = row_place(brick, grp, P.lbx, NG >> P.lbx, P.nx, P.ny);
  const int c0 = panel * P.pc;
  const int nvec = (min(P.pc, P.ncols - c0) + VEC - 1) / VEC;
  bool act[CPL];
#pragma unroll
  for (int q = 0; q < CPL; ++q) act[q] = gl + q * G < nvec;
  // idle lanes read their group's first vector and store nothing
  int col[CPL];
#pragma unroll
  for (int q = 0; q < CPL; ++q) col[q] = c0 + (act[q] ? (gl + q * G) * VEC : 0);
  // A last vector that reaches past the block's columns stays inside the row pitch, except
  // in the last row, whose padding may not be there: read by elements.
  bool over = false;
  if constexpr (TAIL) {
#pragma unroll
    for (int q = 0; q < CPL; ++q) over |= col[q] + VEC > P.ncols;
  }
  const int last_x = over ? P.last_x : -1, last_z = over ? P.nrows - 1 : -2;
  const char* xp[CPL];
  const char* zp[CPL];
  char* yp[CPL];
#pragma unroll
  for (int q = 0; q < CPL; ++q) {
    xp[q] = reinterpret_cast<const char*>(P.X + col[q]);
    zp[q] = reinterpret_cast<const char*>(P.Z + col[q]);
    yp[q] = reinterpret_cast<char*>(P.Y + col[q]);
  }
  auto at = [](const char* p, int row, int pitch) {
    return p + static_cast<int64_t>(row) * pitch;
  };
  const unsigned mine = G == 32 ? kFull : ((1u << (G & 31)) - 1u) << (lane - gl);
  const bool in = at0.x < P.s1 && at0.y < P.lines;
  const int64_t r64 = at0.x + static_cast<int64_t>(P.s1) * at0.y +
                      static_cast<int64_t>(P.s2) * at0.z * P.bz;
  int row = in && r64 < P.nrows ? static_cast<int>(r64) : -1;
  int zi = 0;
  auto next_of = [&](int r) {
    const unsigned n = static_cast<unsigned>(r) + static_cast<unsigned>(P.s2);
    return r >= 0 && n < static_cast<unsigned>(P.nrows) ? static_cast<int>(n) : -1;
  };
  int s = 0, e = 0;
  if (row >= 0) {
    s = __ldg(P.rowptr + row);
    e = __ldg(P.rowptr + row + 1);
  }
  int c[M];
  T w[M];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    c[m] = -2;
    w[m] = T(0);
    if (s + m * G + gl < e) {
      c[m] = __ldg(P.colind + s + m * G + gl);
      w[m] = __ldg(P.vals + s + m * G + gl);
    }
  }
  int nrow = P.bz > 1 ? next_of(row) : -1;
  int ns = 0, ne = 0;
  if (nrow >= 0) {
    ns = __ldg(P.rowptr + nrow);
    ne = __ldg(P.rowptr + nrow + 1);
  }
  while (true) {
    const int cnt = e - s;
    V z[CPL];
    if (P.use_beta && row >= 0) {
#pragma unroll
      for (int q = 0; q < CPL; ++q) {
        const T* p = reinterpret_cast<const T*>(at(zp[q], row, P.ldz));
        if (TAIL && row == last_z) {
#pragma unroll
          for (int f = 0; f < VEC; ++f) z[q].v[f] = col[q] + f < P.ncols ? p[f] : T(0);
        } else {
          z[q] = *reinterpret_cast<const V*>(p);
        }
      }
    }
    bool self = false;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      if (!FOLD) break;
      w[m] = P.alpha * w[m];
      if (P.use_gamma) {
        const bool own = c[m] == row;  // lanes past the row's entries hold column -2
        self |= own;
        if (own) w[m] += P.gamma;
      }
    }
    V acc[CPL];
#pragma unroll
    for (int q = 0; q < CPL; ++q)
#pragma unroll
      for (int f = 0; f < VEC; ++f) acc[q].v[f] = T(0);
    int cn[M];
    T wn[M];
    int nrow2 = -1, ns2 = 0, ne2 = 0;
    auto prefetch = [&] {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        cn[m] = -2;
        wn[m] = T(0);
        if (ns + m * G + gl < ne) {
          cn[m] = __ldg(P.colind + ns + m * G + gl);
          wn[m] = __ldg(P.vals + ns + m * G + gl);
        }
      }
      nrow2 = zi + 2 < P.bz ? next_of(nrow) : -1;
      if (nrow2 >= 0) {
        ns2 = __ldg(P.rowptr + nrow2);
        ne2 = __ldg(P.rowptr + nrow2 + 1);
      }
    };
    auto fetch = [&](int cj, int q, bool careful) -> V {
      const T* p = reinterpret_cast<const T*>(at(xp[q], cj, P.ldx));
      if (TAIL && careful) {
        if (cj == last_x) {
          V r;
#pragma unroll
          for (int f = 0; f < VEC; ++f) r.v[f] = col[q] + f < P.ncols ? __ldg(p + f) : T(0);
          return r;
        }
      }
      return load_ro<T, VEC>(p);
    };
    const int cnt0 = __shfl_sync(kFull, cnt, 0);
    bool plain = cnt == cnt0;
    if constexpr (TAIL) {  // rows that touch X's last row take the careful path
#pragma unroll
      for (int m = 0; m < M; ++m) plain = plain && c[m] != P.last_x;
    }
    if (__all_sync(kFull, plain)) {
      // every row of the warp has as many entries: no lane is held back
#pragma unroll
      for (int m = 0; m < M; ++m) {
#pragma unroll
        for (int j0 = 0; j0 < G; j0 += KC) {
          const int base = m * G + j0;
          if (base + KC <= cnt0 && j0 + KC <= G) {
            V xv[KC][CPL];
#pragma unroll
            for (int j = 0; j < KC; ++j) {
              const int cj = __shfl_sync(kFull, c[m], j0 + j, G);
#pragma unroll
              for (int q = 0; q < CPL; ++q) xv[j][q] = fetch(cj, q, false);
            }
            if (base == 0) prefetch();
#pragma unroll
            for (int j = 0; j < KC; ++j) {
              const T wj = __shfl_sync(kFull, w[m], j0 + j, G);
#pragma unroll
              for (int q = 0; q < CPL; ++q)
#pragma unroll
                for (int f = 0; f < VEC; ++f) acc[q].v[f] = fma(wj, xv[j][q].v[f], acc[q].v[f]);
            }
          } else if (base < cnt0) {
            if (base == 0) prefetch();
#pragma unroll
            for (int j = 0; j < KC; ++j) {
              if (j0 + j < G && base + j < cnt0) {
                const int cj = __shfl_sync(kFull, c[m], j0 + j, G);
                const T wj = __shfl_sync(kFull, w[m], j0 + j, G);
#pragma unroll
                for (int q = 0; q < CPL; ++q) {
                  const V xv = fetch(cj, q, false);
#pragma unroll
                  for (int f = 0; f < VEC; ++f) acc[q].v[f] = fma(wj, xv.v[f], acc[q].v[f]);
                }
              }
            }
          }
        }
      }
      if (cnt0 == 0) prefetch();
    } else {
      prefetch();
      int most = cnt;
#pragma unroll
      for (int o = 16; o >= G; o >>= 1) most = max(most, __shfl_xor_sync(kFull, most, o));
#pragma unroll
      for (int m = 0; m < M; ++m) {
        for (int j = 0; j < G; ++j) {
          if (m * G + j >= most) break;
          const int cj = __shfl_sync(kFull, c[m], j, G);
          const T wj = __shfl_sync(kFull, w[m], j, G);
          if (m * G + j < cnt) {
#pragma unroll
            for (int q = 0; q < CPL; ++q) {
              const V xv = fetch(cj, q, true);
#pragma unroll
              for (int f = 0; f < VEC; ++f) acc[q].v[f] = fma(wj, xv.v[f], acc[q].v[f]);
            }
          }
        }
      }
    }
    if (FOLD && P.use_gamma) {
      const unsigned found = __ballot_sync(kFull, self);
      if (row >= 0 && !(found & mine)) {
#pragma unroll
        for (int q = 0; q < CPL; ++q) {
          const V xv = fetch(row, q, true);
#pragma unroll
          for (int f = 0; f < VEC; ++f) acc[q].v[f] = fma(P.gamma, xv.v[f], acc[q].v[f]);
        }
      }
    }
    if (row >= 0) {
#pragma unroll
      for (int q = 0; q < CPL; ++q) {
        V out = acc[q];
        if constexpr (!FOLD) {
#pragma unroll
          for (int f = 0; f < VEC; ++f) out.v[f] = P.alpha * out.v[f];
          if (P.use_gamma) {  // the row of X is in L1
            const V xv = fetch(row, q, true);
#pragma unroll
            for (int f = 0; f < VEC; ++f) out.v[f] = fma(P.gamma, xv.v[f], out.v[f]);
          }
        }
        if (P.use_beta) {
#pragma unroll
          for (int f = 0; f < VEC; ++f) out.v[f] = fma(P.beta, z[q].v[f], out.v[f]);
        }
        if (act[q]) {
          if constexpr (CORR) {
            const V rv = *reinterpret_cast<const V*>(
                at(reinterpret_cast<const char*>(P.R + col[q]), row, P.ldr));
#pragma unroll
            for (int f = 0; f < VEC; ++f)
              out.v[f] = fma(__ldg(P.delta + col[q] + f), rv.v[f], out.v[f]);
          }
          T* yr = reinterpret_cast<T*>(yp[q] + static_cast<int64_t>(row) * P.ldy);
          if (TAIL && col[q] + VEC > P.ncols) {
#pragma unroll
            for (int f = 0; f < VEC; ++f)
              if (col[q] + f < P.ncols) yr[f] = out.v[f];
          } else {
            *reinterpret_cast<V*>(yr) = out;
          }
        }
      }
    }
    if (++zi >= P.bz || !__any_sync(kFull, nrow >= 0)) break;
    row = nrow;
    nrow = nrow2;
    s = ns;
    e = ne;
    ns = ns2;
    ne = ne2;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      c[m] = cn[m];
      w[m] = wn[m];
    }
  }
}

template <typename T, int VEC, int G, int CPL, int M, int KC, bool FOLD, bool CORR>
void launch(RowsParams<T> P, int64_t rows, bool tail, cudaStream_t s) {
  constexpr int NG = kRowsThreads / G;
  const RowOrder order = row_order(P.s1, P.s2, NG);
  P.s1 = order.s1;
  P.s2 = order.s2;
  P.lines = order.lines;
  P.lbx = order.lbx;
  P.nx = order.nx;
  P.ny = order.ny;
  const int64_t planes = (rows + P.s2 - 1) / P.s2;
  const int64_t columns = static_cast<int64_t>(P.nx) * P.ny * P.panels;
  // A CTA's first rows wait for a chain of loads that the later ones hide, and deep bricks
  // re-read fewer planes; but the deeper they are, the longer the last CTAs run alone. With W
  // rows to each of the four CTAs of every SM, W / d starts and a tail of d are least at
  // d = sqrt(W) (13 points, 34 FP64 columns, 63^3: 112 us so, 148 us in bricks of 16).
  const double share = static_cast<double>(columns * planes) / (4.0 * num_sms());
  P.bz = std::max(1, std::min(16, static_cast<int>(std::sqrt(share) + 0.5)));
  const int64_t grid = columns * ((planes + P.bz - 1) / P.bz);
  FE_REQUIRE(grid <= 0x7fffffffLL, "csr_spmm: too many rows for one launch");
  // a correction comes with whole vectors only
  if (VEC > 1 && !CORR && tail)
    spmm_rows_kernel<T, VEC, G, CPL, M, KC, FOLD, (VEC > 1 && !CORR), CORR>
        <<<static_cast<unsigned>(grid), kRowsThreads, 0, s>>>(P);
  else
    spmm_rows_kernel<T, VEC, G, CPL, M, KC, FOLD, false, CORR>
        <<<static_cast<unsigned>(grid), kRowsThreads, 0, s>>>(P);
  check_launch("spmm_rows_kernel");
}

}  // namespace

// Looks at 32 rows each in the middle and at the quarters of the operator (a heuristic: the
// result only orders the work).
constexpr int64_t kGridRows = 32;
static int64_t grid_window(int64_t rows, int i) {
  const int64_t quarter[] = {2, 1, 3};
  return rows / 4 * quarter[i] - kGridRows / 2;
}

static void set_pattern(Csr& A, const std::vector<RowWindow>& w) {
  const RowPattern p = find_pattern(w, A.rows);
  A.grid_s1 = p.s1;
  A.grid_s2 = p.s2;
  A.row_kind = p.kind;
}

void csr_find_grid(Csr& A, const int32_t* rowptr, const int32_t* colind) {
  std::vector<RowWindow> w;
  for (int i = 0; i < 3 && A.rows >= 8 * kGridRows; ++i) {
    const int64_t r = grid_window(A.rows, i);
    w.push_back({rowptr + r, colind + rowptr[r], r, static_cast<int>(kGridRows)});
  }
  set_pattern(A, w);
}

// The same for an operator whose arrays are on the device.
void csr_find_grid_device(Csr& A) {
  std::vector<RowWindow> w;
  std::vector<int32_t> rp[3], ci[3];
  for (int i = 0; i < 3 && A.rows >= 8 * kGridRows; ++i) {
    const int64_t r = grid_window(A.rows, i);
    rp[i].resize(kGridRows + 1);
    FE_CHECK_CUDA(cudaMemcpy(rp[i].data(), A.rowptr + r, rp[i].size() * sizeof(int32_t),
                             cudaMemcpyDeviceToHost));
    const int64_t entries = rp[i][kGridRows] - rp[i][0];
    ci[i].resize(entries);
    if (entries > 0)
      FE_CHECK_CUDA(cudaMemcpy(ci[i].data(), A.colind + rp[i][0], entries * sizeof(int32_t),
                               cudaMemcpyDeviceToHost));
    w.push_back({rp[i].data(), ci[i].data(), r, static_cast<int>(kGridRows)});
  }
  set_pattern(A, w);
}

template <typename T>
bool csr_spmm_rows(const Csr& A, const T* X, int64_t ldx, T* Y, int64_t ldy, const T* Z,
                   int64_t ldz, const T* R, int64_t ldr, const T* delta, int64_t ncols,
                   double alpha, double gamma, double beta, cudaStream_t s) {
  constexpr int V16 = 16 / sizeof(T);
  const bool ub = beta != 0.0;
  const int k = static_cast<int>(std::min<int64_t>(A.max_row_nnz, 64));
  const int64_t bytes = ncols * static_cast<int64_t>(sizeof(T));
  const int64_t far = std::max(std::max(ldx, ldy), std::max(ub ? ldz : 0, R ? ldr : 0));
  // Blocks of up to four vectors keep the loop kernel's smaller groups.
  if (k < 1 || k > 32 || bytes <= 64 || far * static_cast<int64_t>(sizeof(T)) > 0x7fffffffLL)
    return false;
  auto multiple = [&](size_t b) {
    auto ok = [b](const void* p, int64_t ld) {
      return reinterpret_cast<uintptr_t>(p) % b == 0 && (ld * sizeof(T)) % b == 0;
    };
    return ok(X, ldx) && ok(Y, ldy) && (!ub || ok(Z, ldz)) && (!R || ok(R, ldr));
  };
  const int vec = multiple(16) ? V16 : sizeof(T) == 4 && multiple(8) ? 2 : 1;
  if (R && (vec != V16 || ncols % V16 != 0)) return false;
  RowsParams<T> P{};
  P.rowptr = A.rowptr;
  P.colind = A.colind;
  if constexpr (sizeof(T) == 8) P.vals = A.val64; else P.vals = A.val32;
  P.X = X;
  P.Y = Y;
  P.Z = Z;
  P.R = R;
  P.delta = delta;
  P.ldx = static_cast<int>(ldx * sizeof(T));
  P.ldy = static_cast<int>(ldy * sizeof(T));
  P.ldz = static_cast<int>(ldz * sizeof(T));
  P.ldr = static_cast<int>(ldr * sizeof(T));
  P.nrows = static_cast<int>(A.rows);
  P.last_x = static_cast<int>(A.cols) - 1;
  P.ncols = static_cast<int>(ncols);
  P.s1 = A.grid_s1;
  P.s2 = A.grid_s2;
  P.alpha = static_cast<T>(alpha);
  P.gamma = static_cast<T>(gamma);
  P.beta = static_cast<T>(beta);
  P.use_gamma = gamma != 0.0 ? 1 : 0;
  P.use_beta = ub ? 1 : 0;
  // as the row kernel of spmm.cu would take it: short rows, 32 or more 8-byte vectors
  const bool fold = k <= 7 && vec * sizeof(T) >= 8 && bytes % 8 == 0 && bytes >= 256;
  const bool tail = ncols % vec != 0;
  // Where the kernels of spmm.cu are the better ones (us, there and here):
  // - few rows (94 FP32 columns, 25^3: 13.2, 16.1), small blocks of whole vectors, which
  //   stay in L2 (16 FP64 columns, 43^3: 12.4, 15.8), larger ones of wide rows (158 FP64
  //   columns, 29^3: 25, 29; but 100 FP32 columns, 43^3, 32 MB: 40, 31) and of rows of up to
  //   8 vectors (28 FP32 columns, 57^3: 21, 25; 32, 96^3: 104, 100);
  // - 17 or more entries a row: rows of more than 48 vectors, whose lanes are full there (124
  //   FP64 columns, 51^3: 192, 207), blocks of up to 16 whole vectors, whose lanes there are
  //   fewer (16 FP64 columns, 76^3: 126, 193), and element-wide lanes (49 FP64 columns, 31^3:
  //   31, 45);
  // - element-wide lanes: FP32 (113 columns, 57^3: 95, 136); FP64 where the row kernel's lanes
  //   are full (149 columns, 71^3: 334, 356, but 70 columns, 55^3: 140, 88) and, with longer
  //   rows, up to 224 columns (193, 42^3: 129, 142, but 275, 38^3: 244, 153), and the 49 to 64
  //   columns that go in two panels here (51, 64^3: 154, 158; 45, 154, 91; 65, 211, 163);
  // - FP32 rows of 8-byte lanes, up to 7 entries, where the row kernel's panels (of up to 160
  //   vectors) take four or five vectors a lane (258 columns, 64^3: 228, 309; 162, 212, 192);
  // - rows of more than 64 16-byte vectors that do not fill panels of 32, in blocks of up to 64 MB
  //   (320 FP32 columns, 35^3: 43, 48) and on grids of small planes (5 x 80 x 800: 284, 305),
  //   and any row of more than 64 vectors on thinner grids, short lines with far couplings and
  //   operators of unknown rows (10 x 10 x 4000: 355, 355; lines of 77 rows and a coupling
  //   100,003 rows off: 262, 283; but 600 x 600, 297, 242, and tridiagonal, 234, 189);
  // - scattered entries (a row's loads come from L2 one by one, and the row kernel has a whole
  //   short row in flight): rows of more than 48 vectors (200 FP32 columns, 64^3 permuted:
  //   243, 288), FP32 rows of up to 8 (32 columns, 100^3 permuted: 166, 181), and more than 8
  //   entries a row (64 FP32 columns, 13 points, 64^3 permuted: 90, 111) but for FP32 columns
  //   that end inside a vector, which go by elements there (51 columns: 142, 128); 8-byte
  //   vectors from 33 on with up to 8 entries (98 FP32 columns, 64^3 permuted: 145, 176) and
  //   FP64 rows by elements from 49 columns on (65: 223, 237).
  const int64_t block = A.rows * bytes, MB = int64_t(1) << 20;
  const int nvec = static_cast<int>((ncols + vec - 1) / vec);
  const int lanes16 = (nvec + 15) / 16 * 16, lanes32 = (nvec + 31) / 32 * 32;
  const bool panels32 = lanes32 * 19 <= lanes16 * 20;
  if (A.rows < 32768) return false;
  if (!tail && (block < 16 * MB || (bytes >= 1024 && block < 32 * MB) ||
                (bytes <= 192 && block < 24 * MB) || (bytes <= 128 && block < 64 * MB)))
    return false;
  if (k > 16 && (bytes > 768 || vec != V16 || bytes <= (tail ? 128 : 256))) return false;
  if (vec == 1 &&
      (sizeof(T) == 4 ||
       (k <= 7 ? ncols < 32 || (ncols > 48 && ncols <= 64) || ncols > 96 : ncols <= 224)))
    return false;
  if (sizeof(T) == 4 && vec == 2 && k <= 7) {  // the row kernel's panels of up to 160 vectors
    const int parts = (nvec + 159) / 160;
    if ((nvec + parts - 1) / parts > 96) return false;
  }
  const Sweep sweep = row_sweep(A.grid_s1, A.grid_s2);
  const bool scattered = A.row_kind == RowKind::kScattered;
  if (bytes > 1024 && vec == V16) {
    if (sweep == Sweep::kRuns && A.row_kind != RowKind::kBanded &&
        A.row_kind != RowKind::kIrregular && (k <= 8 || A.row_kind != RowKind::kGrid))
      return false;
    if (k <= 8 && !panels32 &&
        (block < 64 * MB || (sweep == Sweep::kPlanes && A.grid_s2 < kSmallPlane)))
      return false;
  }
  if (scattered) {
    const bool whole = vec == V16 && bytes <= 768 && (k <= 8 || (sizeof(T) == 4 && tail));
    const bool narrow = vec != V16 && (k > 8 || nvec <= (sizeof(T) == 4 ? 32 : 48));
    if ((!whole && !narrow) || (sizeof(T) == 4 && bytes <= 128)) return false;
  }
  auto panels = [&](int cap) {
    P.panels = (nvec + cap - 1) / cap;
    P.pc = (nvec + P.panels - 1) / P.panels * vec;
  };
#define FE_ROWS_F(V_, G_, C_, M_, K_, FOLD_, CORR_)                 \
  do {                                                              \
    panels(G_ * C_);                                                \
    launch<T, V_, G_, C_, M_, K_, FOLD_, CORR_>(P, A.rows, tail, s); \
    return true;                                                    \
  } while (0)
#define FE_ROWS(V_, G_, C_, M_, K_, CORR_)                      \
  do {                                                          \
    if (fold) FE_ROWS_F(V_, G_, C_, M_, K_, true, CORR_);       \
    FE_ROWS_F(V_, G_, C_, M_, K_, false, CORR_);                \
  } while (0)
  if (vec == V16) {
    // One panel of the fewest lanes and vectors that hold the row, two neighbours in flight:
    // a row's share of the instructions falls with the vectors of a lane (96^3, 7 points,
    // FP32, us: 64 columns 146 with (8 lanes, 2 vectors) against 161 with (16, 1), 80 columns
    // 201 (8, 3) against 262, 160 columns 373 (16, 3) against 431; 64^3, 13 points, FP64, 96
    // columns 194 (16, 3) against 220). Wider rows: panels of (16, 2) where they fill their
    // lanes (256 columns 544 against 574), else of (16, 1) with a whole short row in flight
    // (320 columns, 128^3: 1.67 against 1.80 ms). FP64 rows of 9 to 16 and 25 to 32 vectors
    // do as well or better in (16, 1) panels where a sweep is deep or, with irregular rows, L1
    // has little to give; elsewhere (8, 2) and (16, 2) (us: 24 columns of a 600 x 600 grid 98
    // -> 66, 64 columns of a 40000 x 8 grid 133 -> 111), and (8, 2) for the widest (320 FP32
    // columns, 600 x 600: 430 -> 242).
    const int lanes24 = (nvec + 23) / 24 * 24;
    const bool f64 = sizeof(T) == 8;
    const bool deep = sweep == Sweep::kPlanes ? A.rows / 16 >= A.grid_s2
                                              : A.row_kind != RowKind::kGrid &&
                                                    A.row_kind != RowKind::kBanded;
    // 0: (8, 1), 1: (8, 2), 2: (8, 3), 3: (16, 1), 4: (16, 2), 5: (16, 3), 6: (32, 3)
    int shape = 3;
    if (nvec <= 8) shape = 0;
    else if (scattered && f64) shape = 3;
    else if (nvec <= 16) shape = f64 && k <= 8 && deep ? 3 : 1;
    else if (nvec <= 24) shape = 2;
    else if (nvec <= 32) shape = f64 && k <= 8 && deep ? 3 : 4;
    else if (nvec <= 48) shape = 5;
    else if (k > 8 && k <= 16 && nvec > 64 && nvec <= 96) shape = 6;
    else if (panels32) shape = f64 && k <= 8 && deep ? 3 : 4;
    else if (k <= 8 && !deep) shape = 1;
    else if (lanes24 < lanes16) shape = 2;
    if (k > 16 && shape < 3) shape = nvec <= 16 ? 3 : 4;  // 8 lanes hold 16 entries
#define FE_SHAPES(CORR_)                                          \
  do {                                                            \
    if (k <= 8) {                                                 \
      if (shape == 0) FE_ROWS_F(V16, 8, 1, 1, 7, false, CORR_);   \
      if (shape == 1) FE_ROWS(V16, 8, 2, 1, 2, CORR_);            \
      if (shape == 2) FE_ROWS(V16, 8, 3, 1, 2, CORR_);            \
      if (shape == 3) FE_ROWS(V16, 16, 1, 1, 7, CORR_);           \
      if (shape == 4) FE_ROWS(V16, 16, 2, 1, 2, CORR_);           \
      FE_ROWS(V16, 16, 3, 1, 2, CORR_);                           \
    }                                                             \
    if (k <= 16) {                                                \
      if (shape == 0) FE_ROWS_F(V16, 8, 1, 2, 4, false, CORR_);   \
      if (shape == 1) FE_ROWS_F(V16, 8, 2, 2, 2, false, CORR_);   \
      if (shape == 2) FE_ROWS_F(V16, 8, 3, 2, 2, false, CORR_);   \
      if (shape == 3) FE_ROWS_F(V16, 16, 1, 1, 13, false, CORR_); \
      if (shape == 4) FE_ROWS_F(V16, 16, 2, 1, 2, false, CORR_);  \
      if (shape == 6) FE_ROWS_F(V16, 32, 3, 1, 2, false, CORR_);  \
      FE_ROWS_F(V16, 16, 3, 1, 2, false, CORR_);                  \
    }                                                             \
    if (shape == 3) FE_ROWS_F(V16, 16, 1, 2, 8, false, CORR_);    \
    if (shape == 4) FE_ROWS_F(V16, 16, 2, 2, 2, false, CORR_);    \
    FE_ROWS_F(V16, 16, 3, 2, 2, false, CORR_);                    \
  } while (0)
    if constexpr (sizeof(T) == 4) {
      if (R) FE_SHAPES(true);
    }
    FE_SHAPES(false);
#undef FE_SHAPES
  }
  if constexpr (sizeof(T) == 4) {
    if (vec == 2) FE_ROWS(2, 16, 2, 1, 4, false);
  } else {
    FE_ROWS(1, 16, 3, 1, 4, false);  // FP64 rows that start at any element
  }
  return false;
#undef FE_ROWS_F
#undef FE_ROWS
}
template bool csr_spmm_rows<float>(const Csr&, const float*, int64_t, float*, int64_t,
                                   const float*, int64_t, const float*, int64_t, const float*,
                                   int64_t, double, double, double, cudaStream_t);
template bool csr_spmm_rows<double>(const Csr&, const double*, int64_t, double*, int64_t,
                                    const double*, int64_t, const double*, int64_t,
                                    const double*, int64_t, double, double, double,
                                    cudaStream_t);

}  // namespace fe
