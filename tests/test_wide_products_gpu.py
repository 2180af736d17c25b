"""FP64 Gram and rotation with more columns than narrow tiles can cover in one launch (65,535
tiles across), against torch in FP64: k = 2 products of entries of size one."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m", [65535 * 32, 3_000_008, 65535 * 48 + 1])
def test_millions_of_columns(m):
    from fasteig_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m)
    X = torch.rand(4, 2, generator=g, device="cuda", dtype=torch.float64)
    Y = torch.rand(4, m, generator=g, device="cuda", dtype=torch.float64)
    C = torch.rand(2, m, generator=g, device="cuda", dtype=torch.float64)
    assert (ops.gram(X, Y) - X.T @ Y).abs().max() <= 1e-14
    assert (ops.rotate(X, C, torch.empty_like(Y)) - X @ C).abs().max() <= 1e-14
