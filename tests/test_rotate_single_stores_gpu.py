"""FP64 rotation into outputs that are stored one value at a time (odd columns or pitches), at
the widths whose column tile that decides, with and without the output added: against torch in
FP64, 1e-13 of |alpha| |X| |C| + |beta| |Y| as test_dmma_gpu.py has it."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("n,k,m", [(130, 3, 51), (300, 45, 64), (1000, 97, 97), (257, 161, 161),
                                   (129, 64, 127), (5000, 20, 63)])
def test_single_stores(n, k, m, beta):
    from fasteig_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(n + m)
    X = torch.randn(n, k, generator=g, device="cuda", dtype=torch.float64)
    C = torch.randn(k, m, generator=g, device="cuda", dtype=torch.float64)
    Y = torch.randn(n, m + 1 + m % 2, generator=g, device="cuda", dtype=torch.float64)[:, 1:m + 1]
    ref = -0.5 * (X @ C) + beta * Y
    scale = 0.5 * (X.abs() @ C.abs()) + beta * Y.abs()
    ops.rotate(X, C, Y, -0.5, beta)
    assert bool(((Y - ref).abs() <= 1e-13 * scale).all())
