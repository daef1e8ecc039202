"""The device-driven FGMRES of the whole-step graph on the GPU against a plain float64 solve."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _step(nx, ny, nz, restart, precision="fp64"):
    """Pressure of the second step (the first is host-driven, the second runs as a graph) and its system."""
    from impes_b200 import scenarios
    from impes_b200.simulator import build_from_config
    cfg, f = scenarios.two_phase_2d(seed=11, nx=nx, ny=ny, nz=nz)
    cfg["simulation"]["amg"].update({"tol": 1e-12, "restart": restart, "max_iters": 2000, "precision": precision,
                                     "warm_start": False})
    _, fl, _, sim = build_from_config(cfg, f)
    assert sim.run_step(86400.0)
    rowptr, col, val, rhs = sim.assemble(86400.0)
    assert sim.run_step(86400.0)
    assert sim.step_graphs()[0] >= 1 and not sim.step_graphs()[1]
    A = torch.sparse_csr_tensor(rowptr.long(), col.long(), val, size=(rhs.numel(), rhs.numel())).to_dense()
    d = A.diagonal().sqrt()
    ref = torch.linalg.solve(A / d[:, None] / d[None, :], rhs / d) / d
    return fl.pressure.reshape(-1), ref, sim.last_krylov


# basis sizes around the kernels' groups of 8, 16, 32 and 64 vectors, the largest basis, odd and tiny vectors (fewer
# elements than a block holds), in both precisions of the V-cycle
@pytest.mark.parametrize("dims,restart,precision", [
    ((33, 31, 1), 7, "fp64"), ((33, 31, 1), 8, "fp64"), ((33, 31, 1), 9, "mixed"), ((33, 31, 1), 17, "fp64"),
    ((47, 45, 3), 33, "fp64"), ((47, 45, 3), 60, "mixed"), ((64, 64, 4), 65, "fp64"), ((64, 64, 4), 120, "fp64"),
    ((5, 3, 1), 60, "fp64"), ((17, 1, 1), 60, "fp64")])
def test_step_pressure(dims, restart, precision):
    p, ref, st = _step(*dims, restart, precision)
    assert st["converged"]
    # tol 1e-12 of ||D^-1 b||; the pressure follows the scaled residual to a factor of about 1e2 on these grids
    assert float((p - ref).norm() / ref.norm()) < 1e-9
    assert st["iterations"] < 2000
