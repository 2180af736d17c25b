"""The calls whose speed counts, as a program of the eigensolver's user makes them.

Each case is one call (or the short chain of calls that belongs together) through the
package's public entry points, on operators of the stencils and sizes that the solvers,
the serving mix and the tests run on: 3D Laplacians (7-, 13- and 27-point) with Gaussian
wells or a uniform potential, blocks from 8 to 320 columns, FP32 and FP64.

``listed`` are the cases measured by name, ``draw`` gives more of the same ranges,
``prepare`` makes what the program holds before the call, ``run`` is one pass, ``work``
the bytes and operations a pass cannot do without (inputs read once, outputs written
once), and ``exact`` the outputs in 64 bits from plain torch.
"""
import math

import torch

import fasteig_b200 as fe
from fasteig_b200 import ops

# One filter's interval parameters: the operators below have their spectra in
# [-30, 16]; the filter damps [2, 16] and lets the lower end through.
DAMPED = (2.0, 16.0)
# Nominal cycles of a Chebyshev solve and iterations of an LOBPCG solve, for work().
CYCLES, LOBPCG_ITERATIONS = 13, 60


def listed():
    return [
        # One operator apply of a small problem (24^3 grid, block 12): latency only. What
        # an LOBPCG or Davidson user's loop calls between its own steps.
        dict(name="spmm_f64_24cube_12", kind="spmm", dtype="f64", stencil="7pt", side=24, cols=12,
             pad=False),
        # K X of the generalized problem (80^3 grid, 27-point stiffness, block 96).
        dict(name="spmm_f64_27pt_80cube_96", kind="spmm", dtype="f64", stencil="27pt", side=80,
             cols=96, pad=True),
        # FP64 filter of an ordinary solve, odd grid and block, the default degree, rows that
        # are not padded: a caller's own tensor.
        dict(name="filter_f64_49cube_45", kind="filter", dtype="f64", stencil="7pt", side=49,
             cols=45, degree=10, pad=False),
        # FP32 filter on a 13-point operator of the serving mix.
        dict(name="filter_f32_13pt_77cube_51", kind="filter", dtype="f32", stencil="13pt", side=77,
             cols=51, degree=16, pad=True),
        # FP32 filter of the headline problem (128^3 wells, block 320, degree 16).
        dict(name="filter_f32_128cube_320", kind="filter", dtype="f32", stencil="7pt", side=128,
             cols=320, degree=16, pad=True),
        # Cholesky QR of a small block: Gram, factor, inverse, rotation.
        dict(name="cholqr_f64_33cube_48", kind="cholqr", rows=35937, cols=48),
        # Cholesky QR of an LOBPCG basis (three blocks of 96 on the 80^3 grid).
        dict(name="cholqr_f64_80cube_288", kind="cholqr", rows=512000, cols=288),
        # Basis rotation of the mixed path on the tensor cores, headline size.
        dict(name="rotate_f32_128cube_320", kind="rotate", rows=2097152, cols=320, out=320),
        # Residual block and its norms, generalized (80^3, block 96).
        dict(name="residual_f64_80cube_96", kind="residual", dtype="f64", rows=512000, cols=96),
        # Projected eigenproblems of a group of solves that advance together.
        dict(name="eig_f64_8x96", kind="eig", count=8, cols=96),
        # A whole small solve: LOBPCG, 24^3 uniform potential, 8 lowest pairs, block 12.
        dict(name="solve_lobpcg_24cube_8", kind="solve", solver="LOBPCG", stencil="7pt", side=24,
             wells=0, nev=8, block=12, degree=10, precision="fp64"),
        # The headline solve: mixed-precision Chebyshev, 128^3 wells, 256 pairs.
        dict(name="solve_mixed_128cube_256", kind="solve", solver="Chebyshev", stencil="7pt",
             side=128, wells=32, nev=256, block=320, degree=16, precision="mixed"),
    ]


def _between(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmm", "spmm", "filter", "filter", "filter", "cholqr", "cholqr", "rotate",
                       "residual", "eig", "solve"])
    dtype = rng.choice(["f32", "f64"])
    if kind in ("spmm", "filter"):
        stencil = rng.choice(["7pt", "13pt", "27pt"] if kind == "spmm" else ["7pt", "13pt"])
        side = _between(rng, 22, 128)
        cols = min(_between(rng, 8, 320), int(320 * 128 ** 3 * (0.5 if dtype == "f64" else 1.0)
                                              / side ** 3))
        case = dict(kind=kind, dtype=dtype, stencil=stencil, side=side, cols=cols,
                    pad=rng.random() < 0.7)
        if kind == "filter":
            case["degree"] = rng.choice([8, 10, 16, 20])
        return case
    if kind == "cholqr":
        return dict(kind=kind, rows=_between(rng, 10000, 500000), cols=_between(rng, 8, 320))
    if kind == "rotate":
        cols = 8 * _between(rng, 4, 40)
        return dict(kind=kind, rows=_between(rng, 10000, 2000000), cols=cols,
                    out=max(8, 8 * int(cols * rng.uniform(0.3, 1.0) / 8)))
    if kind == "residual":
        return dict(kind=kind, dtype=dtype, rows=_between(rng, 10000, 1000000),
                    cols=_between(rng, 8, 256))
    if kind == "eig":
        count = rng.choice([1, 1, 2, 4, 8, 16])
        return dict(kind=kind, count=count, cols=_between(rng, 16, 320))
    nev = _between(rng, 6, 48)
    return dict(kind="solve", solver="Chebyshev", stencil=rng.choice(["7pt", "13pt"]),
                side=_between(rng, 22, 64), wells=16, nev=nev, block=nev + max(8, nev // 4),
                degree=16, precision=rng.choice(["fp64", "mixed"]))


# ---------------------------------------------------------------- inputs

def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000003 * (int(seed) % 2000000) + salt)


def _ld(cols, pad):
    return -(-cols // 8) * 8 if pad else cols  # the solvers pad a block's rows to 8 values


def _normal(rows, cols, dtype, g, pad=True):
    """A Gaussian block; with ``pad`` a view of one whose rows are 16-byte aligned."""
    t = torch.randn(rows, _ld(cols, pad), generator=g, device="cuda",
                    dtype=torch.float64 if dtype == "f64" else torch.float32)
    return t[:, :cols]


def _potential(side, wells, g):
    """Sum of Gaussian wells (depth 1 to 5, width 2 to 6 grid units), one to a cell of the
    box, as atoms keep apart: one structure, of which every seed is another configuration
    (wells displaced by up to a grid unit, depths by 2 %). Uniform in [0, 1) when ``wells``
    is 0. x fastest."""
    n = side ** 3
    if wells == 0:
        return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    u = torch.rand(wells, 5, generator=torch.Generator().manual_seed(5), dtype=torch.float64)
    moved = torch.rand(wells, 4, generator=g, device="cuda", dtype=torch.float64).cpu() * 2 - 1
    x = torch.arange(side, device="cuda", dtype=torch.float64)
    v = torch.zeros(side, side, side, device="cuda", dtype=torch.float64)
    cells = math.ceil(round(wells ** (1.0 / 3.0), 9))
    for k in range(wells):
        a = (1.0 + 4.0 * float(u[k, 0])) * (1.0 + 0.02 * float(moved[k, 0]))
        w = 2.0 + 4.0 * float(u[k, 1])
        e = []
        for i in range(3):
            cell = k // cells ** i % cells
            at = (cell + float(u[k, 2 + i])) / cells * (side - 1) + float(moved[k, 1 + i])
            e.append(torch.exp(-(x - at) ** 2 / (2.0 * w * w)))
        v -= a * e[2][:, None, None] * e[1][None, :, None] * e[0][None, None, :]
    return v.reshape(-1)


def _operator(stencil, side, wells, seed):
    """(rowptr, colind, values) on the GPU, columns ascending within each row: a Dirichlet
    operator on a side^3 grid in natural order."""
    g = _generator(seed, 17)
    if stencil == "27pt":
        offs = [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]
    else:
        reach = 1 if stencil == "7pt" else 2
        offs = [(0, 0, 0)] + [tuple(s * (i == a) for i in range(3)) for a in range(3)
                              for s in range(-reach, reach + 1) if s]
    shift = {o: o[0] + side * (o[1] + side * o[2]) for o in offs}
    offs.sort(key=lambda o: shift[o])
    n = side ** 3
    i = torch.arange(n, device="cuda")
    xyz = [i % side, (i // side) % side, i // (side * side)]
    ok = torch.stack([((xyz[0] + o[0] >= 0) & (xyz[0] + o[0] < side)
                       & (xyz[1] + o[1] >= 0) & (xyz[1] + o[1] < side)
                       & (xyz[2] + o[2] >= 0) & (xyz[2] + o[2] < side)) for o in offs], dim=1)
    col = i[:, None] + torch.tensor([shift[o] for o in offs], device="cuda")[None, :]
    val = torch.empty(n, len(offs), device="cuda", dtype=torch.float64)
    if stencil == "27pt":  # K_ij = -(c_i + c_j) / 2, K_ii = sum_j |K_ij| + 1e-3
        c = torch.exp(0.5 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
        val = -(c[:, None] + c[col.clamp(0, n - 1)]) / 2.0
        val = torch.where(ok, val, torch.zeros_like(val))
        val[:, 13] = 0.0
        val[:, 13] = val.abs().sum(dim=1) + 1e-3
    else:
        v = _potential(side, wells, g)
        for k, o in enumerate(offs):
            far = max(abs(t) for t in o)
            if far == 0:
                val[:, k] = (6.0 if stencil == "7pt" else 7.5) + v
            elif stencil == "7pt":
                val[:, k] = -1.0
            else:
                val[:, k] = -4.0 / 3.0 if far == 1 else 1.0 / 12.0
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(ok.sum(dim=1), 0)
    return rowptr, col[ok], val[ok]


def _device_csr(rowptr, colind, values):
    """The package's operator from a host CSR, as a program that assembled one has it."""
    return fe.CsrMatrix(rowptr.numel() - 1, rowptr.to(torch.int32).cpu().numpy(),
                        colind.to(torch.int32).cpu().numpy(), values.cpu().numpy())


def _wells(case):
    return case.get("wells", 32)


def _interval():
    lo, hi = DAMPED
    c = 2.0 / (hi - lo)
    return c, -c * (hi + lo) / 2.0  # maps [lo, hi] to [-1, 1]


def _blocks(case, seed):
    """The dense inputs of a case."""
    kind, g = case["kind"], _generator(seed, 5)
    if kind in ("spmm", "filter"):
        return dict(X=_normal(case["side"] ** 3, case["cols"], case["dtype"], g, case["pad"]))
    if kind == "cholqr":  # filtered columns: mixed, of unequal length
        k = case["cols"]
        X = _normal(case["rows"], k, "f64", g)
        mix = torch.eye(k, device="cuda", dtype=torch.float64) + 0.5 / math.sqrt(k) * torch.randn(
            k, k, generator=g, device="cuda", dtype=torch.float64)
        scale = torch.logspace(-1, 1, k, device="cuda", dtype=torch.float64)
        X.copy_(X @ (mix * scale))
        return dict(X=X)
    if kind == "rotate":  # an orthonormal block (length 1 a column) and near-orthogonal coefficients
        X = _normal(case["rows"], case["cols"], "f32", g).div_(math.sqrt(case["rows"]))
        C = torch.randn(case["cols"], case["out"], generator=g, device="cuda", dtype=torch.float64)
        return dict(X=X, C=C / math.sqrt(case["cols"]))
    if kind == "residual":  # Ritz vectors part of the way: residuals 1e-3 of the products
        n, k = case["rows"], case["cols"]
        X = _normal(n, k, case["dtype"], g)
        BX = _normal(n, k, case["dtype"], g)
        BX.mul_(0.1).add_(X)
        lam = torch.rand(k, generator=g, device="cuda", dtype=torch.float64).mul_(8).add_(0.5)
        AX = _normal(n, k, case["dtype"], g)
        AX.mul_(1e-3).add_(BX * lam.to(BX.dtype))
        return dict(X=X, BX=BX, AX=AX, lam=lam)
    k = case["cols"]  # eig: projected matrices
    M = torch.randn(case["count"], k, k, generator=g, device="cuda", dtype=torch.float64)
    M = (M + M.transpose(1, 2)) / math.sqrt(2.0 * k)
    M += torch.diag(torch.linspace(-4.0, 8.0, k, device="cuda", dtype=torch.float64))
    return dict(A=M.contiguous())


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A = _device_csr(*_operator(case["stencil"], case["side"], _wells(case), seed))
        o = fe.fasteig_options(A.rows)
        for k, v in dict(solver=case["solver"], nev=case["nev"], block=case["block"],
                         degree=case["degree"], which="SR", tol=1e-8, maxiter=300,
                         precision=case["precision"], seed=1 + int(seed) % 1000000).items():
            o.set(k, v)
        if case["solver"] == "Chebyshev":
            for k, v in dict(bounds="ritz", amplification=1e6, init="device").items():
                o.set(k, v)
        return dict(problem=fe.fasteig_problem(A, solver=case["solver"]), options=o)
    s = _blocks(case, seed)
    if kind in ("spmm", "filter"):
        s["A"] = _device_csr(*_operator(case["stencil"], case["side"], _wells(case), seed))
        s["Y"] = torch.empty_like(s["X"]) if not case["pad"] else _normal(
            s["X"].shape[0], case["cols"], case["dtype"], _generator(seed, 6))
        if kind == "filter":
            s["scratch"] = torch.empty_strided(s["X"].shape, s["X"].stride(), device="cuda",
                                               dtype=s["X"].dtype)
    elif kind in ("cholqr", "rotate"):
        s["Y"] = torch.zeros(case["rows"], _ld(case.get("out", case["cols"]), True), device="cuda",
                             dtype=s["X"].dtype)[:, :case.get("out", case["cols"])]
    elif kind == "residual":
        s["R"] = torch.zeros_like(s["X"])
    s["case"] = case
    return s


def run(state):
    if "problem" in state:
        # The spectrum. (Vectors are defined up to their sign and to the tolerance only.)
        state["problem"].solve(state["options"], want_vectors=False)
        return state["problem"].eigenvalues()
    kind = state["case"]["kind"]
    if kind == "spmm":
        return ops.spmm(state["A"], state["X"], state["Y"])
    if kind == "filter":  # in place on a copy: the caller keeps its block
        state["Y"].copy_(state["X"])
        return ops.cheb_filter(state["A"], state["Y"], state["scratch"], state["case"]["degree"],
                               *_interval())
    if kind == "cholqr":
        X = state["X"]
        R, info = ops.potrf_upper(ops.gram(X, X))
        Q = ops.rotate(X, ops.trinv_upper(R), state["Y"])
        return dict(Q=Q, R=R, info=info)
    if kind == "rotate":
        return ops.rotate_tf32x3(state["X"], state["C"], state["Y"])
    if kind == "residual":
        norms = ops.residual_norms(state["AX"], state["X"], state["lam"], state["BX"], state["R"])
        return dict(R=state["R"], rnorm=norms[0], xnorm=norms[1], rel=norms[2])
    W, Z = ops.syevd_batched(state["A"], [state["case"]["cols"]] * state["case"]["count"])
    return dict(W=W, Z=Z)


# ---------------------------------------------------------------- work and 64-bit results

_POINTS = {"7pt": (7, 6), "13pt": (13, 18), "27pt": (27, None)}


def _nnz(stencil, side):
    if stencil == "27pt":
        return (3 * side - 2) ** 3
    points, lost = _POINTS[stencil]
    return points * side ** 3 - lost * side ** 2


def work(case):
    kind = case["kind"]
    s = 4 if case.get("dtype") == "f32" or case.get("precision") == "mixed" else 8
    if kind in ("spmm", "filter"):
        n, b, nnz = case["side"] ** 3, case["cols"], _nnz(case["stencil"], case["side"])
        steps = case.get("degree", 1)
        flops = steps * 2.0 * nnz * b + (steps * 4.0 * n * b if kind == "filter" else 0.0)
        return dict(bytes=nnz * (s + 4) + 4 * (n + 1) + 2.0 * n * b * s, flops=flops)
    if kind == "cholqr":
        n, k = case["rows"], case["cols"]
        return dict(bytes=8.0 * (2 * n * k + k * k), flops=3.0 * n * k * k + 2.0 * k ** 3 / 3)
    if kind == "rotate":
        n, k, m = case["rows"], case["cols"], case["out"]
        return dict(bytes=4.0 * n * (k + m) + 8.0 * k * m, flops=2.0 * n * k * m)
    if kind == "residual":
        n, k = case["rows"], case["cols"]
        return dict(bytes=s * 3.0 * n * k + 32.0 * k, flops=6.0 * n * k)
    if kind == "eig":
        p, k = case["count"], case["cols"]
        return dict(bytes=8.0 * p * (2 * k * k + k), flops=p * (4.0 / 3 + 2.0 + 1.0) * k ** 3)
    n, b, nnz = case["side"] ** 3, case["block"], _nnz(case["stencil"], case["side"])
    if case["solver"] == "LOBPCG":  # per iteration: one apply, Gram and rotations of a 3b basis
        flops = LOBPCG_ITERATIONS * (2.0 * nnz * b + 18.0 * n * b * b + 12.0 * n * b * b)
    else:  # per cycle: the filter, two Grams and two rotations
        flops = CYCLES * (case["degree"] * (2.0 * nnz + 4.0 * n) * b + 6.0 * n * b * b)
    return dict(bytes=12.0 * nnz + 4.0 * n + 8.0 * case["nev"], flops=flops)


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        n = case["side"] ** 3
        if n > 16000:
            return None
        rowptr, colind, values = _operator(case["stencil"], case["side"], _wells(case), seed)
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), rowptr.diff())
        dense = torch.zeros(n, n, device="cuda", dtype=torch.float64)
        dense[rows, colind] = values
        return torch.linalg.eigvalsh(dense)[:case["nev"]].cpu().numpy()
    s = _blocks(case, seed)
    if kind in ("spmm", "filter"):
        rowptr, colind, values = _operator(case["stencil"], case["side"], _wells(case), seed)
        n = case["side"] ** 3
        if case["dtype"] == "f32":  # the operator's values as an FP32 caller's data holds them
            values = values.float().double()
        A = torch.sparse_csr_tensor(rowptr, colind, values, size=(n, n))
        X = s["X"].double()
        if kind == "spmm":
            return A @ X
        c, d = _interval()
        prev, cur = X, (A @ X).mul_(c).add_(X, alpha=d)
        for _ in range(case["degree"] - 1):
            nxt = (A @ cur).mul_(2 * c).add_(cur, alpha=2 * d).sub_(prev)
            prev, cur = cur, nxt
        return cur
    if kind == "cholqr":
        X = s["X"]
        R = torch.linalg.cholesky(X.T @ X, upper=True)
        Q = torch.linalg.solve_triangular(R, X, upper=True, left=False)
        return dict(Q=Q, R=R, info=None)
    if kind == "rotate":
        return s["X"].double() @ s["C"]
    if kind == "residual":
        X, BX, AX, lam = s["X"].double(), s["BX"].double(), s["AX"].double(), s["lam"]
        R = AX - BX * lam
        # relative to (1 + |lambda|) times the length of M x
        rn, bn = R.norm(dim=0), BX.norm(dim=0)
        return dict(R=R, rnorm=rn, xnorm=bn, rel=rn / ((1.0 + lam.abs()) * bn))
    return dict(W=torch.linalg.eigvalsh(s["A"]), Z=None)
