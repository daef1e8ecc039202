"""The coarsest inverse in clusters of eight CTAs, for GPUs (or parts of one) where sixteen cannot run together."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# the smallest and largest of its range, and column blocks that end inside a CTA's 64 columns and at their edge
@pytest.mark.parametrize("n", [257, 320, 321, 449, 499, 500])
def test_inverse_of_eight_ctas(monkeypatch, n):
    import scipy.sparse as sp
    from impes_b200.amg import ClassicalAMG
    monkeypatch.setenv("IMPES_COARSE_CLUSTER", "8")
    rng = np.random.default_rng(n)
    A = 2.0 * np.eye(n) + 0.3 * rng.standard_normal((n, n)) / np.sqrt(n)
    A = A[rng.permutation(n)]            # the elimination has to interchange rows
    A[np.arange(n), np.arange(n)] += np.where(np.abs(np.diag(A)) < 0.05, 0.05, 0.0)
    amg = ClassicalAMG(sp.csr_matrix(A), coarsest_size=n, max_levels=4, mixed_precision=True)
    P = amg.levels[0]["A"].to_dense().cpu().numpy()
    P[0, :] = 0.0
    P[:, 0] = 0.0
    P[0, 0] = 1.0
    b = rng.standard_normal(n)
    bp = b.copy()
    bp[0] = 0.0
    ref = np.linalg.solve(P, bp)
    x = amg.vcycle_scaled(torch.from_numpy(b).cuda()).cpu().numpy()
    # inverse and product of Gauss-Jordan with partial pivoting: a few n eps cond
    assert np.linalg.norm(x - ref) <= 8.0 * n * np.finfo(np.float64).eps * np.linalg.cond(P) * np.linalg.norm(ref)
    _, st = amg.fgmres(torch.from_numpy(b).cuda(), tol=1e-10, norm="equilibrated")
    assert st["converged"] and st["iterations"] <= 2
