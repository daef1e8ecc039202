"""Rows of more than 512 entries: two and four warps a row of the V-cycle's kernels, against scipy."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


def _banded(n, row, seed):
    """Symmetric M-matrix of about `row` entries a row, strong next neighbours and a weak band (its coarse levels stay
    banded)."""
    rng = np.random.default_rng(seed)
    half = (row - 1) // 2
    d = [rng.uniform(0.5, 1.5, n - 1)] + [rng.uniform(0.5, 1.5, n - k) * 0.02 for k in range(2, half + 1)]
    G = sp.diags(d, range(1, half + 1), shape=(n, n)).tocsr()
    G = (G + G.T).tocsr()
    return (sp.diags(np.asarray(G.sum(axis=1)).ravel() + 0.5) - G).tocsr()


def _host(t):
    t = t.cpu()
    return sp.csr_matrix((t.values().numpy(), t.col_indices().numpy(), t.crow_indices().numpy()), shape=tuple(t.shape))


def _vcycle(levels, l, b):
    L = levels[l]
    A, w = L["A"], 0.7 * L["inv"]
    n = A.shape[0]
    if L["last"]:
        bp = b.copy()
        bp[0] = 0.0
        if n <= 500:
            M = A.toarray()
            M[0, :] = 0.0
            M[:, 0] = 0.0
            M[0, 0] = 1.0
            return np.linalg.solve(M, bp)
        x = np.zeros(n)
        for _ in range(50):
            x = x + w * (bp - A @ x)
        return x
    x = np.zeros(n)
    for _ in range(3):
        x = x + w * (b - A @ x)
    x = x + L["P"] @ _vcycle(levels, l + 1, L["P"].T @ (b - A @ x))
    for _ in range(2):
        x = x + w * (b - A @ x)
    return x


# two warps a row (513 to 1,536 entries, eight a thread at a time and a remainder), four warps (more); a last block that
# is not full, one whose rows end with it; more rows than the launch's blocks take at once (18,944 blocks of eight rows
# a warp each, of four of two warps), so that a block goes on to its next rows
@pytest.mark.parametrize("n,row,warps", [(1603, 700, 2), (2404, 1100, 2), (3001, 1301, 2), (3203, 2101, 4), (4002, 2601, 4),
                                         (152003, 121, 1), (75991, 525, 2)])
def test_vcycle_wide_rows(monkeypatch, n, row, warps):
    from impes_b200.amg import ClassicalAMG
    monkeypatch.setenv("IMPES_NO_SELL", "1")
    A = _banded(n, row, n)
    off = A - sp.diags(A.diagonal())
    amg = ClassicalAMG(A, coarsest_size=30, max_levels=1, mixed_precision=True)
    mean = A.nnz / n
    assert {1: 96 < mean <= 512, 2: 512 < mean <= 1536, 4: mean > 1536}[warps]
    b = np.random.default_rng(1).standard_normal(n)
    bt = torch.from_numpy(b).cuda()
    for f in (1.0, 0.3):
        B = (sp.diags(A.diagonal()) + f * off).tocsr()
        amg.update_values(torch.from_numpy(B.data).cuda())
        x32 = amg.vcycle_scaled(bt, precision="mixed").cpu().numpy()
        x64 = amg.vcycle_scaled(bt, precision="fp64").cpu().numpy()
        levels = [{"A": _host(L["A"]), "last": L["is_coarsest"], "inv": L["inv_relax"].cpu().numpy(),
                   "P": None if L["P"] is None else _host(L["P"])} for L in amg.levels]
        ref = _vcycle(levels, 0, b)
        # the system's condition, at most the largest row sum of absolute values over the smallest excess of a diagonal;
        # roundings of sums of `row` terms, and in single precision of each value once and each sum a few times
        excess = np.asarray(B.sum(axis=1)).ravel().min()
        kappa = np.abs(B).sum(axis=1).max() / excess
        for x, tol in ((x64, 4.0 * row * np.finfo(np.float64).eps * kappa), (x32, 8.0 * np.finfo(np.float32).eps * kappa)):
            assert tol < 1e-3
            assert np.linalg.norm(x - ref) <= tol * np.linalg.norm(ref)
