"""The coarse levels' dense operator: formed where it is expected, and the V-cycle it stands for."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


def _build(dims, **kw):
    from impes_b200 import scenarios
    from impes_b200.amg import ClassicalAMG
    from impes_b200.simulator import build_from_config
    cfg, f = scenarios.two_phase_2d(seed=5, nx=dims[0], ny=dims[1], nz=dims[2])
    cfg["wells"] = cfg["wells"][:1]
    _, _, _, sim = build_from_config(cfg, f)
    rowptr, col, val, _ = sim.assemble(86400.0)
    n = int(np.prod(dims))
    return ClassicalAMG((rowptr, col, val, (n, n)), coarsest_size=60, mixed_precision=True, **kw), val


def _host(t):
    t = t.cpu()
    return sp.csr_matrix((t.values().numpy(), t.col_indices().numpy(), t.crow_indices().numpy()), shape=tuple(t.shape))


def _levels(amg):
    return [{"A": _host(L["A"]), "inv": L["inv_relax"].cpu().numpy(), "last": L["is_coarsest"],
             "P": None if L["P"] is None else _host(L["P"])} for L in amg.levels]


def _pinned(A):
    M = A.toarray()
    M[0, :] = 0.0
    M[:, 0] = 0.0
    M[0, 0] = 1.0
    return M


def _vcycle(levels, l, b, light, without=-1):
    """The V-cycle from zero; ``without``: a level whose correction is left out."""
    L = levels[l]
    A, n, w = L["A"], L["A"].shape[0], 0.7 * L["inv"]
    if l == without:
        return np.zeros(n)
    if L["last"]:
        bp = b.copy()
        bp[0] = 0.0
        if n <= 500:
            return np.linalg.solve(_pinned(A), bp)
        x = np.zeros(n)
        for _ in range(50):
            x = x + w * (bp - A @ x)
        return x
    few = n <= light
    x = np.zeros(n)
    for _ in range(1 if few else 3):
        x = x + w * (b - A @ x)
    x = x + L["P"] @ _vcycle(levels, l + 1, L["P"].T @ (b - A @ x), light, without)
    for _ in range(1 if few else 2):
        x = x + w * (b - A @ x)
    return x


# the operator's level and how it is made: sparse products alone; dense ones on the levels below; light sweeps; a capped
# interpolation; a coarsest level of more than 500 rows with short and with long rows; the coarsest inverse by a cluster;
# dense products on the operator's own level
@pytest.mark.parametrize("dims,kw,made", [
    ((45, 45, 1), {}, {"sparse"}), ((15, 13, 11), {}, {"sparse", "dense"}),
    ((15, 13, 11), {"light_sweep_rows": 2000}, {"sparse", "dense"}), ((16, 16, 9), {"p_max_elements": 2}, {"sparse", "dense"}),
    ((40, 44, 1), {"max_levels": 1}, {"sweeps"}), ((19, 17, 11), {"max_levels": 2}, {"sweeps", "long"}),
    ((33, 29, 9), {"max_levels": 3}, {"sweeps", "long"}), ((29, 23, 11), {"max_levels": 3}, {"sparse", "cluster"}),
    ((40, 40, 12), {}, {"dense"})])
def test_operator_is_formed_and_right(dims, kw, made):
    amg, val = _build(dims, **kw)
    light = kw.get("light_sweep_rows", 0)
    levels = _levels(amg)
    assert amg.coarse_operator is not None
    first, rows, _ = amg.coarse_operator
    n = [L["A"].shape[0] for L in levels]
    long_rows = [L["A"].nnz // L["A"].shape[0] >= L["A"].shape[0] // 6 for L in levels]
    assert first >= 1 and rows == n[first] <= 1152
    found = {"dense" if r else "sparse" for r in long_rows[first:-1]}
    if n[-1] > 500:
        found |= {"sweeps"} | ({"long"} if long_rows[-1] else set())
    elif n[-1] > 256:
        found |= {"cluster"}
    assert made <= found, (n, found)
    b = np.random.default_rng(3).standard_normal(n[0])
    bt = torch.from_numpy(b).cuda()
    half32 = 0.5 * float(np.finfo(np.float32).eps)

    def check(x, levels, precision):
        ref = _vcycle(levels, 0, b, light)
        part = ref - _vcycle(levels, 0, b, light, without=first)
        kappa = np.linalg.cond(_pinned(levels[first]["A"]))
        # roundings of sums of at most n terms, times the condition of the level that the operator stands for (single
        # precision values: of each value once and of each sum a few times)
        tol = 4.0 * n[first] * np.finfo(np.float64).eps * kappa if precision == "fp64" else 16.0 * half32 * kappa
        assert tol < 5e-3
        err = np.linalg.norm(x.cpu().numpy() - ref)
        assert err <= tol * np.linalg.norm(ref), (precision, err / np.linalg.norm(ref), tol)
        assert err <= 0.1 * np.linalg.norm(part)            # the coarse levels' part cannot be missing

    check(amg.vcycle_scaled(bt, precision="fp64"), levels, "fp64")
    check(amg.vcycle_scaled(bt, precision="mixed"), levels, "mixed")
    # both precisions behind each update, in either order and again
    for top, order in ((1.7, ("mixed", "fp64", "fp64", "mixed")), (0.4, ("fp64", "mixed", "fp64")), (0.9, ("mixed", "mixed"))):
        amg.update_values(val * torch.linspace(1.0, top, val.numel(), dtype=torch.float64, device=val.device))
        got = [(amg.vcycle_scaled(bt, precision=p), p) for p in order]
        its = [amg.fgmres(bt, tol=1e-10, precision=p, max_iters=400)[1] for p in order]
        levels = _levels(amg)
        for x, p in got:
            check(x, levels, p)
        assert all(s["converged"] for s in its)
        assert max(s["iterations"] for s in its) - min(s["iterations"] for s in its) <= 2


@pytest.mark.parametrize("kw", [{"smoother": "chebyshev"}, {"max_levels": 1, "coarsest_size": 400}])
def test_no_operator(kw):
    """Other smoothers keep their levels; a coarsest level of at most 500 rows right below the first is one product
    already."""
    from impes_b200 import scenarios
    from impes_b200.amg import ClassicalAMG
    from impes_b200.simulator import build_from_config
    cfg, f = scenarios.two_phase_2d(seed=5, nx=31, ny=27, nz=1)
    _, _, _, sim = build_from_config(cfg, f)
    rowptr, col, val, _ = sim.assemble(86400.0)
    amg = ClassicalAMG((rowptr, col, val, (837, 837)), **{"coarsest_size": 60, **kw})
    assert amg.coarse_operator is None
