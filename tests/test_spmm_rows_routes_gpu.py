"""The multi-row SpMM on every kind of operator that its dispatch tells apart: planes (also
thin ones), lines (short, long, couplings as far as half the rows), bands with and without
repeating offsets, permuted rows; FP64 rows at odd pitches with folded coefficients; and the
correction term of the refined filter through whole solves.
References: the product in 64 bits from SciPy, with the bound of test_spmm_rows_gpu.py (an
output is a chain of at most 15 rounded multiply-adds: 32 units of the type's rounding of the
sum of the terms' sizes), and, bit for bit, the kernels of one warp per row (mode 7), whose
arithmetic this one states to be its own."""
import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _csr(n, rows, cols, seed):
    from fasteig_b200 import matrices as M
    key = np.unique(np.asarray(rows, np.int64) * n + cols)
    rowptr = np.zeros(n + 1, np.int64)
    np.add.at(rowptr, key // n + 1, 1)
    rng = np.random.default_rng(seed)
    return M.HostCsr(n, np.cumsum(rowptr).astype(np.int32), (key % n).astype(np.int32),
                     rng.standard_normal(key.size))


def _diagonals(n, offsets, seed):
    i = np.arange(n)
    pairs = [(i[(i + d >= 0) & (i + d < n)], d) for d in offsets]
    return _csr(n, np.concatenate([r for r, _ in pairs]),
                np.concatenate([r + d for r, d in pairs]), seed)


def _grid(dims, kind, seed, permute=False):
    from fasteig_b200 import matrices as M
    n = int(np.prod(dims))
    H = M._stencil_csr(dims, M._offsets(len(dims), kind), lambda r, c: np.ones(r.size),
                       np.ones(n))
    rows = np.repeat(np.arange(n), np.diff(H.rowptr))
    p = np.random.default_rng(seed).permutation(n) if permute else np.arange(n)
    return _csr(n, p[rows], p[H.colind], seed)


@functools.lru_cache(maxsize=None)
def _operator(kind):
    n = 40003
    rng = np.random.default_rng(7)
    if kind == "band":  # other offsets in each row
        rows = np.concatenate([np.arange(n), np.repeat(np.arange(n), 5)])
        cols = np.concatenate([np.arange(n), np.clip(np.repeat(np.arange(n), 5)
                                                     + rng.integers(-900, 901, 5 * n), 0, n - 1)])
        return _csr(n, rows, cols, 1)
    return {
        "tridiagonal": lambda: _diagonals(n, (-1, 0, 1), 2),
        "half": lambda: _diagonals(n, (-(n // 2), -1, 0, 1, n // 2), 3),
        "third": lambda: _diagonals(39999, (-13333, -1, 0, 1, 13333), 4),
        "far": lambda: _diagonals(n, (-15013, -77, 0, 77, 15013), 5),
        "thin": lambda: _grid((10, 10, 401), "star1", 6),
        "thin16": lambda: _grid((16, 16, 150), "star1", 7),
        "sliver": lambda: _grid((5, 90, 80), "star1", 8),
        "flat": lambda: _grid((120, 115, 3), "star1", 9),
        "lines": lambda: _grid((197, 201), "star1", 10),
        "long_lines": lambda: _grid((2100, 19), "star1", 11),
        "thin13": lambda: _grid((9, 9, 500), "star2", 12),
        "permuted": lambda: _grid((34, 34, 35), "star1", 13, permute=True),
        "permuted13": lambda: _grid((34, 34, 35), "star2", 14, permute=True),
    }[kind]()


def _block(n, cols, ld, dtype, seed):
    """An n x cols view of pitch ld over storage that ends with the last row's last column."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    flat = torch.full(((n - 1) * ld + cols,), float("nan"), dtype=dtype, device="cuda")
    t = torch.as_strided(flat, (n, cols), (ld, 1))
    return t.copy_(torch.randn(n, cols, generator=g, device="cuda", dtype=dtype))


def _check(H, cols, ld, dtype):
    import scipy.sparse as sp
    import fasteig_b200 as fe
    from fasteig_b200 import CsrMatrix, ops
    A = CsrMatrix(H.n, H.rowptr, H.colind, H.values)
    vals = H.values.astype(np.float32 if dtype == torch.float32 else np.float64).astype(np.float64)
    S = sp.csr_matrix((vals, H.colind, H.rowptr), shape=(H.n, H.n))
    X, Z = _block(H.n, cols, ld, dtype, 1), _block(H.n, cols, ld, dtype, 2)
    part = np.r_[0:8, cols - 16:cols]  # columns compared in 64 bits; the others bit for bit
    Xd, Zd = X[:, part].double().cpu().numpy(), Z[:, part].double().cpu().numpy()
    a, g, b = 0.75, -0.25, -1.0
    Y, W = _block(H.n, cols, ld, dtype, 3), _block(H.n, cols, ld, dtype, 3)
    ops.cheb_step(A, X, Z, Y, a, g, b)
    ref = a * (S @ Xd) + g * Xd + b * Zd
    scale = a * (abs(S) @ np.abs(Xd)) + abs(g * Xd) + abs(b * Zd)
    err = np.abs(Y[:, part].double().cpu().numpy() - ref)
    assert np.all(err <= 32 * torch.finfo(dtype).eps * scale), err.max()
    assert fe.lib.fe_set_spmm_kernel(7) == 0
    try:
        ops.cheb_step(A, X, Z, W, a, g, b)
    finally:
        assert fe.lib.fe_set_spmm_kernel(0) == 0
    assert torch.equal(Y, W)
    assert ops.device_status(clear=True) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["tridiagonal", "band", "half", "third", "far", "thin", "thin16",
                                  "sliver", "flat", "lines", "long_lines", "thin13", "permuted",
                                  "permuted13"])
@pytest.mark.parametrize("cols,ld", [(51, 56), (64, 64), (109, 112), (128, 128), (322, 328),
                                     (512, 512)])
def test_kinds_of_operators(kind, cols, ld, dtype):
    _check(_operator(kind), cols, ld, dtype)


@pytest.mark.parametrize("cols,ld", [(51, 51), (61, 63), (95, 95)])
def test_f64_odd_pitch_folded(cols, ld):
    from fasteig_b200 import matrices as M
    _check(M.laplacian_wells(37, wells=4, seed=3), cols, ld, torch.float64)


@pytest.mark.parametrize("kind", ["lines", "thin16", "permuted", "permuted13", "thin13"])
@pytest.mark.parametrize("cols,dtype", [(45, torch.float64), (71, torch.float64),
                                        (227, torch.float64), (50, torch.float32),
                                        (98, torch.float32), (258, torch.float32),
                                        (322, torch.float32)])
def test_narrow_vectors(kind, cols, dtype):
    """Rows that start at multiples of 8 bytes only: FP32 in 8-byte vectors, FP64 by elements."""
    _check(_operator(kind), cols, cols, dtype)


@pytest.mark.parametrize("stencil,nev,block", [("star1", 48, 72), ("star1", 100, 136),
                                               ("star2", 72, 100)])
def test_refined_filter_correction(stencil, nev, block):
    """The mixed solve's FP64 cycles add the correction term in this kernel (64,000 rows);
    tail_filter=fp64 does without it. Residuals are formed in FP64 from the operator, relative
    to 1 + |lambda|; both solves stop at 1e-8, which bounds their eigenvalues' distance."""
    import fasteig_b200 as fe
    from fasteig_b200 import matrices as M
    H = M.laplacian_wells(40, wells=16, seed=2, stencil=stencil)
    A = fe.CsrMatrix(H.n, H.rowptr, H.colind, H.values)
    got = {}
    for tail in ("refined", "fp64"):
        o = fe.fasteig_options(A.rows)
        for k, v in dict(solver="Chebyshev", nev=nev, block=block, degree=16, which="SR", tol=1e-8,
                         maxiter=200, precision="mixed", bounds="ritz", amplification=1e6,
                         init="device", seed=5, tail_filter=tail).items():
            o.set(k, v)
        p = fe.fasteig_problem(A, solver="Chebyshev")
        p.solve(o)
        assert np.max(p.residual_norms()) <= 1e-8
        got[tail] = np.array(p.eigenvalues())
    assert np.all(np.abs(got["refined"] - got["fp64"]) <= 2e-8 * (1 + np.abs(got["fp64"])))
