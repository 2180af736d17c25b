"""The order in which the multi-row SpMM deals rows to its groups of lanes
(fasteig_b200/csrc/spmm_grid.hpp, compiled with g++ through tests/cpp/grid_check.cpp): every
row once and none outside its plane, also at sizes where an int product of two strides would
overflow; groups kept busy on thin grids and far couplings; the strides found on grids, and
none on scattered, permuted or banded operators."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from fasteig_b200 import matrices as M

ROOT = Path(__file__).resolve().parents[1]
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = tmp_path_factory.mktemp("grid") / "grid_check"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror",
                        str(ROOT / "tests" / "cpp" / "grid_check.cpp"), "-o", str(out)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return out


def run(exe, what, text):
    r = subprocess.run([str(exe), what], input=text, capture_output=True, text=True, check=True)
    return [float(v) for v in r.stdout.split()]


# rows, line, plane: cubes, thin and flat grids, far couplings, lines only, no grid
ORDERS = [(117649, 49, 2401), (262144, 64, 4096), (40000, 10, 100), (32771, 4, 16),
          (60000, 5, 1025), (60000, 7, 1400), (90000, 300, 30000), (66000, 1023, 2046),
          (60000, 20000, 0), (60000, 30000, 0), (90000, 300, 0), (70000, 130, 0),
          (70000, 2047, 0), (70000, 77, 0), (33333, 0, 0)]


@pytest.mark.parametrize("groups", [8, 16, 32])
@pytest.mark.parametrize("rows,s1,s2", ORDERS)
def test_every_row_once_and_groups_busy(exe, rows, s1, s2, groups):
    wrong, outside, used = run(exe, "deal", f"{rows} {s1} {s2} {groups}")
    assert wrong == 0 and outside == 0
    assert used >= 0.75


@pytest.mark.parametrize("s1,s2", [(268435455, 0), (1073741823, 0), (16384, 268435456),
                                   (5, 268435455), (536870911, 1073741822), (0, 0)])
@pytest.mark.parametrize("groups", [8, 16, 32])
def test_order_at_the_index_limit(exe, s1, s2, groups):
    o1, o2, lines, bx, bricks, last = run(exe, "place", f"2147483646 {s1} {s2} {groups}")
    assert o1 * lines == o2 <= 2 ** 30
    assert bricks * groups >= o2 and bricks < 2 ** 31
    assert last == o2 - 1  # the last brick ends with the plane's last row


UNKNOWN, GRID, BANDED, IRREGULAR, SCATTERED = range(5)


def _find(exe, H):
    rows = H.n
    text = [f"{rows} 3"]
    for q in (2, 1, 3):
        r0 = rows // 4 * q - 16
        a, b = H.rowptr[r0], H.rowptr[r0 + 32]
        text.append(f"{r0} 32 " + " ".join(map(str, np.diff(H.rowptr[r0:r0 + 33]))))
        text.append(" ".join(map(str, H.colind[a:b])))
    return tuple(int(v) for v in run(exe, "find", "\n".join(text) + "\n"))


@pytest.mark.parametrize("dims,kind", [((20, 20, 20), "star1"), ((32, 32, 32), "star1"),
                                       ((33, 33, 33), "star1"), ((17, 17, 17), "star2"),
                                       ((32, 32, 32), "star2"), ((16, 16, 16), "box"),
                                       ((10, 10, 400), "star1"), ((12, 30, 9), "star1")])
def test_grid_found(exe, dims, kind):
    H = M._stencil_csr(dims, M._offsets(3, kind), lambda r, c: np.ones(r.size),
                       np.ones(int(np.prod(dims))))
    assert _find(exe, H) == (dims[0], dims[0] * dims[1], GRID)


def test_lines_found(exe):
    assert _find(exe, M.laplacian_uniform_potential(70, 2)) == (70, 0, GRID)


def _csr(n, rows, cols):
    key = np.unique(rows.astype(np.int64) * n + cols)
    rowptr = np.zeros(n + 1, np.int64)
    np.add.at(rowptr, key // n + 1, 1)
    return M.HostCsr(n, np.cumsum(rowptr).astype(np.int32), (key % n).astype(np.int32),
                     np.ones(key.size))


def test_no_grid_found(exe):
    rng = np.random.default_rng(0)
    n = 65536
    diag = np.arange(n)
    for trial in range(4):  # seven scattered entries a row
        rows = np.concatenate([diag, np.repeat(diag, 6)])
        cols = np.concatenate([diag, rng.integers(0, n, 6 * n)])
        assert _find(exe, _csr(n, rows, cols)) == (0, 0, SCATTERED)
    H = M.laplacian_wells(40, wells=2, seed=1)  # a grid whose rows were permuted
    p = rng.permutation(H.n)
    rows = np.repeat(np.arange(H.n), np.diff(H.rowptr))
    assert _find(exe, _csr(H.n, p[rows], p[H.colind])) == (0, 0, SCATTERED)
    cols = np.clip(np.repeat(diag, 6) + rng.integers(-500, 501, 6 * n), 0, n - 1)
    assert _find(exe, _csr(n, np.repeat(diag, 6), cols)) == (0, 0, IRREGULAR)
    band = np.concatenate([np.stack([diag[:n - 2], diag[:n - 2] + d]) for d in (0, 1, 2)], axis=1)
    assert _find(exe, _csr(n, np.concatenate([band[0], band[1]]),
                           np.concatenate([band[1], band[0]]))) == (0, 0, BANDED)
