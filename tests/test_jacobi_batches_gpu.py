"""The batched Jacobi eigensolver at the edges of its rule for threads (32, 64 and 96 rows;
batches of one, of a matrix to every SM and a few more): eigenvalues and vectors against
NumPy, bounds as in test_syevd_gpu.py, and every matrix bit for bit as in a batch of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ragged", [False, True])
@pytest.mark.parametrize("m,count", [(2, 700), (17, 149), (31, 593), (32, 592), (33, 148),
                                     (40, 149), (63, 150), (64, 148), (65, 3), (96, 149)])
def test_threads_by_size_and_count(m, count, ragged):
    from fasteig_b200 import ops
    rng = np.random.default_rng(m * count)
    A = rng.standard_normal((count, m, m))
    A = A + A.transpose(0, 2, 1)
    A[count // 2] = np.eye(m) + 1e-9 * A[count // 2]
    sizes = [m - (p % 3 if ragged and p else 0) for p in range(count)]
    sizes = [max(1, v) for v in sizes]
    dA = torch.from_numpy(A).cuda()
    W, Z = ops.syevd_batched(dA, sizes)
    for p in sorted({0, 1 % count, count // 2, count - 1}):
        k = sizes[p]
        B = A[p, :k, :k]
        w, z = W[p, :k].cpu().numpy(), Z[p, :k, :k].cpu().numpy()
        nrm = np.abs(B).sum(axis=1).max()
        assert np.abs(w - np.linalg.eigvalsh(B)).max() <= 1e-12 * nrm
        assert np.abs(B @ z - z * w[None, :]).max() <= 1e-12 * nrm
        assert np.abs(z.T @ z - np.eye(k)).max() <= 1e-12 * max(k, 10) / 10
        w1, z1 = ops.syevd_batched(dA[p:p + 1].contiguous(), [k])
        assert torch.equal(w1[0, :k], W[p, :k]) and torch.equal(z1[0, :k, :k], Z[p, :k, :k])
