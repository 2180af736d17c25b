"""FP64 Grams of few columns over many row chunks (the chunk sum in 32 shares) and at the
edges of that rule: 64 and 65 chunks, outputs of one and of just over one wave of CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [4096, 4097, 13824, 35937])
@pytest.mark.parametrize("k,m", [(1, 1), (12, 12), (5, 33), (97, 97), (98, 97)])
def test_gram_chunk_sums(n, k, m):
    from fasteig_b200 import ops
    g = torch.Generator().manual_seed(n + 7 * k + m)
    X = torch.randn(n, k, dtype=torch.float64, generator=g).cuda()
    Y = X if k == m else torch.randn(n, m, dtype=torch.float64, generator=g).cuda()
    G = ops.gram(X, Y).cpu().numpy()
    Xh, Yh = X.cpu().numpy(), Y.cpu().numpy()
    assert np.all(np.abs(G - Xh.T @ Yh) <= 1e-13 * (np.abs(Xh).T @ np.abs(Yh)))
    assert np.array_equal(G, ops.gram(X, Y).cpu().numpy())
