"""The triangular inverse of a matrix with a zero pivot or an entry that is not finite: column c
of R^{-1} depends on R's leading c + 1 rows and columns alone, so the columns before the first
bad one are the inverse of that leading block, as back substitution column by column gives
it. Bound: |X - inv| <= 32 k eps |inv| |R| |inv| (k multiply-adds a chain, residual form)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("k", [10, 40, 100, 320, 640])
@pytest.mark.parametrize("bad", ["pivot", "nan", "inf"])
@pytest.mark.parametrize("where", [0.3, 0.5, 0.96])
def test_columns_before_a_bad_one(k, bad, where):
    from fasteig_b200 import ops
    rng = np.random.default_rng(k)
    R = np.triu(rng.standard_normal((k, k)) / np.sqrt(k)) + 2 * np.eye(k)
    q = max(1, int(where * k))
    if bad == "pivot":
        R[q, q] = 0.0
    else:
        R[q // 2, q] = np.nan if bad == "nan" else np.inf
    X = ops.trinv_upper(torch.from_numpy(R).cuda()).cpu().numpy()
    ref = np.linalg.inv(R[:q, :q])
    bound = 32 * k * np.finfo(float).eps * (abs(ref) @ abs(R[:q, :q]) @ abs(ref))
    assert np.all(np.abs(X[:q, :q] - ref) <= bound)
    assert np.all(X[q:, :q] == 0.0)
    assert not np.all(np.isfinite(X[:, q]))
