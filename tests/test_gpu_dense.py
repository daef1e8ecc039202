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


def _plain_vcycle(levels, l, b, light_rows):
    """The V-cycle from zero on level l in numpy, from the exported levels."""
    L = levels[l]
    A, n = L["A"], L["n"]
    w = 0.7 * L["inv"]
    if L["is_coarsest"]:
        bp = b.copy()
        bp[0] = 0.0
        if n <= 500:
            P = A.copy()
            P[0, :] = 0.0
            P[:, 0] = 0.0
            P[0, 0] = 1.0
            return np.linalg.solve(P, bp)
        x = np.zeros(n)
        for _ in range(50):
            x = x + w * (bp - A @ x)
        return x
    light = n <= light_rows
    x = np.zeros(n)
    for _ in range(1 if light else 3):
        x = x + w * (b - A @ x)
    x = x + L["P"] @ _plain_vcycle(levels, l + 1, L["P"].T @ (b - A @ x), light_rows)
    for _ in range(1 if light else 2):
        x = x + w * (b - A @ x)
    return x


def _export(amg):
    out = []
    for L in amg.levels:
        out.append({"A": L["A"].to_dense().cpu().numpy(), "n": L["n"], "is_coarsest": L["is_coarsest"],
                    "inv": L["inv_relax"].cpu().numpy(),
                    "P": None if L["P"] is None else L["P"].to_dense().cpu().numpy()})
    return out


# short rows (sparse products), long rows (dense products), one sweep a side on the coarse levels, a capped
# interpolation, and a coarsest level of more than 500 rows (fifty sweeps)
@pytest.mark.parametrize("dims,kw", [((45, 45, 1), {}), ((15, 13, 11), {}), ((15, 13, 11), {"light_sweep_rows": 2000}),
                                     ((16, 16, 9), {"p_max_elements": 2}), ((17, 15, 11), {"max_levels": 2}),
                                     ((40, 44, 1), {"max_levels": 1})])
def test_coarse_operator_vcycle(dims, kw):
    from impes_b200 import scenarios
    from impes_b200.amg import ClassicalAMG
    from impes_b200.simulator import build_from_config
    cfg, f = scenarios.two_phase_2d(seed=5, nx=dims[0], ny=dims[1], nz=dims[2])
    cfg["wells"] = cfg["wells"][:1]
    _, _, _, sim = build_from_config(cfg, f)
    rowptr, col, val, _ = sim.assemble(86400.0)
    n = dims[0] * dims[1] * dims[2]
    amg = ClassicalAMG((rowptr, col, val, (n, n)), coarsest_size=60, mixed_precision=True, **kw)
    rng = np.random.default_rng(3)
    b = rng.standard_normal(n)
    bt = torch.from_numpy(b).cuda()
    for scale in (1.0, 1.7):       # the operator follows the values
        if scale != 1.0:
            d = torch.linspace(1.0, scale, val.numel(), dtype=torch.float64, device=val.device)
            sym = 0.5 * (d + d.mean())          # keeps the matrix an M-matrix
            amg.update_values(val * sym)
        x64 = amg.vcycle_scaled(bt, precision="fp64").cpu().numpy()
        x32 = amg.vcycle_scaled(bt, precision="mixed").cpu().numpy()
        levels = _export(amg)
        ref = _plain_vcycle(levels, 0, b, kw.get("light_sweep_rows", 0))
        # the coarsest solve's rounding (n eps cond of a scaled matrix of at most ~1e5) bounds the first
        assert np.linalg.norm(x64 - ref) <= 1e-9 * np.linalg.norm(ref)
        # fp32 level values: eps32 times the same condition on the coarsest level
        assert np.linalg.norm(x32 - ref) <= 2e-2 * np.linalg.norm(ref)
        x, st = amg.fgmres(bt, tol=1e-10, precision="mixed", max_iters=400)
        assert st["converged"]


# rows of a few products, long rows (a block each), and a hierarchy whose P rows repeat a column (a row whose weights all
# vanished takes its first coarse neighbour a second time)
@pytest.mark.parametrize("dims", [(20, 20, 1), (15, 13, 11), (26, 24, 14)])
def test_galerkin_plan(dims):
    import scipy.sparse as sp
    from impes_b200.amg import ClassicalAMG

    def d1(m, a):
        return sp.diags([-a * np.ones(m - 1), 2 * a * np.ones(m), -a * np.ones(m - 1)], [-1, 0, 1])

    ix, iy, iz = (sp.identity(d) for d in dims)
    A = (sp.kron(sp.kron(d1(dims[0], 1.0), iy), iz) + sp.kron(sp.kron(ix, d1(dims[1], 1.0)), iz)
         + sp.kron(sp.kron(ix, iy), d1(dims[2], 0.1)) + 1e-3 * sp.identity(int(np.prod(dims)))).tocsr()
    amg = ClassicalAMG(A, coarsest_size=30, mixed_precision=True)
    A2 = A.copy()
    A2.data = A2.data * np.where(A2.data > 0, 1.0, np.linspace(0.8, 1.0, A2.nnz))
    amg.update_matrix(A2)
    levels = amg.levels
    for a, b in zip(levels[:-1], levels[1:]):
        L, P, C = (t.to_dense().cpu().numpy() for t in (a["A"], a["P"], b["A"]))
        ref = P.T @ L @ P
        # sums of at most a few thousand products in another order
        assert np.abs(C - ref).max() <= 1e-12 * np.abs(ref).max()
    if dims[2] == 14:
        rows = [a["P"].crow_indices().cpu().numpy() for a in levels[:-1]]
        cols = [a["P"].col_indices().cpu().numpy() for a in levels[:-1]]
        assert any(len(set(c[p[i]:p[i + 1]])) < p[i + 1] - p[i] for p, c in zip(rows, cols) for i in range(len(p) - 1))
