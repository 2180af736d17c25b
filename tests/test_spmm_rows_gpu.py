"""The multi-row SpMM kernel where it can go wrong: block widths around its panels and
vectors, rows that end inside a vector with no padding behind the last row, pitches that are
not whole vectors, rows of 0 to 30 entries, with and without a grid behind the operator (the
smallest that the kernel takes: 32,768 rows).
Reference: the product in 64 bits from SciPy. Bound: every output is a chain of at most 29
rounded multiply-adds of terms bounded by |alpha| |A| |X| + |gamma| |X| + |beta| |Z|, so
32 units of the type's rounding of that sum cover it."""
import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@functools.lru_cache(maxsize=None)
def _operator(kind):
    from fasteig_b200 import matrices as M
    if kind == "7pt":
        return M.laplacian_wells(33, wells=4, seed=1)
    if kind == "13pt":
        return M.laplacian_wells(33, wells=4, seed=1, stencil="star2")
    if kind == "27pt":
        return M.stiffness_mass_27pt(33, seed=1)[0]
    if kind == "2d":
        return M.laplacian_uniform_potential(197, 2, seed=2)
    rng = np.random.default_rng(5)  # no grid: rows of 0..30 scattered entries
    n = 32771
    counts = rng.integers(0, 31, n)
    rowptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    # distinct columns: sorted residues of distinct multiples
    start = np.repeat(rng.integers(0, n, n), counts)
    step = np.concatenate([np.arange(c) for c in counts])
    rows = np.repeat(np.arange(n), counts)
    colind = (start + 1009 * step) % n
    order = np.lexsort((colind, rows))
    colind = colind[order]
    return M.HostCsr(n, rowptr, colind.astype(np.int32), rng.standard_normal(int(rowptr[-1])))


def _block(n, cols, ld, dtype, seed):
    """An n x cols view of pitch ld over storage that ends with the last row's last column."""
    g = torch.Generator().manual_seed(seed)
    flat = torch.full(((n - 1) * ld + cols,), float("nan"), dtype=dtype)
    t = torch.as_strided(flat, (n, cols), (ld, 1))
    t.copy_(torch.randn(n, cols, generator=g, dtype=torch.float64).to(dtype))
    return torch.as_strided(flat.cuda(), (n, cols), (ld, 1))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["7pt", "13pt", "27pt", "2d", "scattered"])
@pytest.mark.parametrize("cols,ld", [(17, 20), (31, 32), (33, 40), (51, 56), (51, 51), (66, 66),
                                     (97, 98), (128, 128), (161, 168), (259, 264), (275, 275),
                                     (300, 304), (384, 384)])
def test_rows_kernel(kind, cols, ld, dtype):
    import scipy.sparse as sp
    from fasteig_b200 import CsrMatrix, ops
    H = _operator(kind)
    A = CsrMatrix(H.n, H.rowptr, H.colind, H.values)
    vals = H.values.astype(np.float32 if dtype == torch.float32 else np.float64).astype(np.float64)
    S = sp.csr_matrix((vals, H.colind, H.rowptr), shape=(H.n, H.n))
    X, Z = _block(H.n, cols, ld, dtype, 1), _block(H.n, cols, ld, dtype, 2)
    Xd, Zd = X.double().cpu().numpy(), Z.double().cpu().numpy()
    eps = torch.finfo(dtype).eps
    for alpha, gamma, beta in ((1.0, 0.0, 0.0), (0.75, -0.25, -1.0)):
        Y = _block(H.n, cols, ld, dtype, 3) if beta == 0 else Z  # beta: in place over Z
        ref = alpha * (S @ Xd) + gamma * Xd + beta * Zd
        scale = alpha * (abs(S) @ np.abs(Xd)) + abs(gamma * Xd) + abs(beta * Zd)
        ops.cheb_step(A, X, Z, Y, alpha, gamma, beta)
        got = Y.double().cpu().numpy()
        assert np.all(np.abs(got - ref) <= 32 * eps * scale), np.abs(got - ref).max()
    assert ops.device_status(clear=True) == 0
