"""Memory of the coarse operator: what it holds, and hierarchies built when little of the device's is free."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _system(nx, ny):
    from impes_b200 import scenarios
    from impes_b200.simulator import build_from_config
    cfg, f = scenarios.two_phase_2d(seed=5, nx=nx, ny=ny, nz=1)
    cfg["wells"] = cfg["wells"][:1]
    _, _, _, sim = build_from_config(cfg, f)
    rowptr, col, val, _ = sim.assemble(86400.0)
    n = nx * ny
    b = torch.from_numpy(np.random.default_rng(7).standard_normal(n)).cuda()
    return (rowptr, col, val, (n, n)), b


# two modes (an inverse of the coarsest matrix to choose) and one (sweeps there), one precision and two
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("dims,levels,modes", [((45, 45), 10, 2), ((40, 44), 1, 1)])
def test_operator_gives_way_to_a_full_device(dims, levels, modes, mixed):
    from impes_b200.amg import ClassicalAMG
    csr, b = _system(*dims)

    def build():
        return ClassicalAMG(csr, coarsest_size=60, max_levels=levels, mixed_precision=mixed)
    amg = build()
    level, rows, size = amg.coarse_operator
    assert level >= 1 and rows == amg.levels[level]["n"]
    matrix = 8 * rows * ((rows + 7) // 8 * 8)
    assert size == (6 + modes * (2 if mixed else 1)) * matrix
    x = amg.vcycle_scaled(b)
    y, st = amg.fgmres(b, tol=1e-10, precision="mixed" if mixed else "fp64")
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    keep = max(48 * size, 1 << 30)             # less than 64 times the operator, enough for everything else
    assert keep < 64 * size
    held = torch.empty(free - keep, dtype=torch.uint8, device="cuda")
    try:
        small = build()
        assert small.coarse_operator is None
        xs = small.vcycle_scaled(b)
        ys, ss = small.fgmres(b, tol=1e-10, precision="mixed" if mixed else "fp64")
    finally:
        del held
        torch.cuda.empty_cache()
    # the same V-cycle, level by level: roundings times the coarsest solve's condition
    assert float((x - xs).norm()) <= 1e-9 * float(x.norm())
    assert ss["converged"] and abs(ss["iterations"] - st["iterations"]) <= 1
    assert float((y - ys).norm()) <= 1e-7 * float(y.norm())


def test_a_refused_allocation_is_reported_once():
    """The call that finds no memory says so, and the calls after it work."""
    from impes_b200 import _lib
    from impes_b200.amg import ClassicalAMG
    csr, b = _system(45, 45)
    amg = ClassicalAMG(csr, coarsest_size=60)
    x = amg.vcycle_scaled(b)
    large, _ = _system(1000, 1000)             # its hierarchy takes more than the gigabyte left here
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(_lib.ImpesError) as err:
            ClassicalAMG(large, coarsest_size=60)
        assert err.value.code == _lib.ERR_OOM
        again = amg.vcycle_scaled(b)
    finally:
        del held
        torch.cuda.empty_cache()
    assert torch.equal(again, x)
    _, st = amg.fgmres(b, tol=1e-10)
    assert st["converged"]
