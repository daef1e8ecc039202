"""Row kernels of the V-cycle over the row lengths and level sizes that choose between them, against scipy."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


def _banded_system(n, row, seed):
    """Symmetric M-matrix of about `row` entries a row: strong next neighbours, weak ones within a band (so that the
    coarse rows stay banded), and two rows several times as long."""
    rng = np.random.default_rng(seed)
    half = max((row - 1) // 2, 1)
    d = [rng.uniform(0.5, 1.5, n - 1)] + [rng.uniform(0.5, 1.5, n - k) * 0.02 for k in range(2, half + 1)]
    G = sp.diags(d, range(1, half + 1), shape=(n, n)).tolil()
    for h in (n // 3, n // 2):
        far = np.unique(rng.integers(0, n, min(4 * row, n // 4)))
        far = far[np.abs(far - h) > half]
        G[h, far] = 0.01
    G = G.tocsr()
    G = (G + G.T).tocsr()
    return (sp.diags(np.asarray(G.sum(axis=1)).ravel() + 0.5) - G).tocsr()


def _vcycle(levels, l, b):
    L = levels[l]
    A, w = L["A"], 0.7 * L["inv"]
    if L["is_coarsest"]:
        bp = b.copy()
        bp[0] = 0.0
        if L["n"] <= 500:
            P = A.toarray()
            P[0, :] = 0.0
            P[:, 0] = 0.0
            P[0, 0] = 1.0
            return np.linalg.solve(P, bp)
        x = np.zeros(L["n"])
        for _ in range(50):
            x = x + w * (bp - A @ x)
        return x
    x = np.zeros(L["n"])
    for _ in range(3):
        x = x + w * (b - A @ x)
    x = x + L["P"] @ _vcycle(levels, l + 1, L["P"].T @ (b - A @ x))
    for _ in range(2):
        x = x + w * (b - A @ x)
    return x


def _host(t):
    t = t.cpu()
    return sp.csr_matrix((t.values().numpy(), t.col_indices().numpy(), t.crow_indices().numpy()), shape=tuple(t.shape))


# short rows (one to four lanes, batches with a remainder), eight lanes and more, one warp a row with four entries in
# flight (more rows than one wave of warps) and with eight
@pytest.mark.parametrize("n,row", [(3001, 4), (5003, 9), (4001, 24), (2003, 50), (12007, 100), (9001, 100),
                                   (10007, 300)])
def test_vcycle_row_kernels(monkeypatch, n, row):
    from impes_b200.amg import ClassicalAMG
    monkeypatch.setenv("IMPES_NO_SELL", "1")
    A = _banded_system(n, row, n)
    off = A - sp.diags(A.diagonal())
    amg = ClassicalAMG(A, coarsest_size=30, max_levels=2, mixed_precision=True)
    b = np.random.default_rng(1).standard_normal(n)
    bt = torch.from_numpy(b).cuda()
    for f in (1.0, 0.3, 0.9):
        # new values and the V-cycle behind them with nothing in between
        B = (sp.diags(A.diagonal()) + f * off).tocsr()
        vals = torch.from_numpy(B.data).cuda()
        amg.update_values(vals)
        x32 = amg.vcycle_scaled(bt, precision="mixed")
        amg.update_values(vals)
        x64 = amg.vcycle_scaled(bt, precision="fp64")
        levels = [{"A": _host(L["A"]), "n": L["n"], "is_coarsest": L["is_coarsest"],
                   "inv": L["inv_relax"].cpu().numpy(), "P": None if L["P"] is None else _host(L["P"])}
                  for L in amg.levels]
        ref = _vcycle(levels, 0, b)
        # a few hundred roundings of sums of at most some thousand terms, and the coarsest solve's condition (< 1e4)
        assert np.linalg.norm(x64.cpu().numpy() - ref) <= 1e-10 * np.linalg.norm(ref)
        assert np.linalg.norm(x32.cpu().numpy() - ref) <= 2e-3 * np.linalg.norm(ref)
