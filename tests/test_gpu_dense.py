"""Dense coarse operators on the GPU against plain float64 linear algebra."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _one_level(n, seed):
    """A one-level hierarchy of a dense matrix whose largest entries lie off the diagonal (rows permuted), so the
    elimination has to interchange rows."""
    import scipy.sparse as sp
    from impes_b200.amg import ClassicalAMG
    rng = np.random.default_rng(seed)
    A = 2.0 * np.eye(n) + 0.3 * rng.standard_normal((n, n)) / np.sqrt(n)
    A = A[rng.permutation(n)]
    A[np.arange(n), np.arange(n)] += np.where(np.abs(np.diag(A)) < 0.05, 0.05, 0.0)
    return ClassicalAMG(sp.csr_matrix(A), coarsest_size=n, max_levels=4, mixed_precision=True), rng


# edges of the kernel's column blocks and clusters, one row, the largest size
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 96, 97, 128, 129, 200, 256, 257, 499, 500])
def test_coarsest_inverse(n):
    amg, rng = _one_level(n, n)
    assert len(amg.levels) == 1
    A = amg.levels[0]["A"].to_dense().cpu().numpy()
    P = A.copy()
    P[0, :] = 0.0
    P[:, 0] = 0.0
    P[0, 0] = 1.0
    b = rng.standard_normal(n)
    bp = b.copy()
    bp[0] = 0.0
    ref = np.linalg.solve(P, bp)
    x = amg.vcycle_scaled(torch.from_numpy(b).cuda()).cpu().numpy()
    # inverse and product of Gauss-Jordan with partial pivoting: a few n eps cond
    tol = 8.0 * n * np.finfo(np.float64).eps * np.linalg.cond(P)
    assert np.linalg.norm(x - ref) <= tol * max(np.linalg.norm(ref), 1e-300)
    if n > 1:
        # the unpinned inverse is an exact preconditioner of the whole system
        xs, st = amg.fgmres(torch.from_numpy(b).cuda(), tol=1e-10, norm="equilibrated")
        assert st["converged"] and st["iterations"] <= 2
