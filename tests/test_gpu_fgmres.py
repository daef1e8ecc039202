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


# one row, one thread's row each (up to 75,776 rows) and several rows a thread, a limit reached and a limit of none
@pytest.mark.parametrize("dims", [(1, 1, 1), (17, 13, 3), (296, 256, 1), (297, 256, 1), (61, 53, 40)])
def test_pcg_solution(dims):
    import ctypes as C
    from impes_b200 import _lib, scenarios
    from impes_b200.simulator import build_from_config
    cfg, f = scenarios.two_phase_2d(seed=2, nx=dims[0], ny=dims[1], nz=dims[2])
    cfg["wells"] = [dict(cfg["wells"][0], control_value=5.0)]
    _, _, _, sim = build_from_config(cfg, f)
    rowptr, col, val, _ = sim.assemble(3600.0)
    n = rowptr.numel() - 1
    A = torch.sparse_csr_tensor(rowptr.long(), col.long(), val, size=(n, n))
    g = torch.Generator(device="cuda").manual_seed(1)
    ref = torch.randn(n, 1, generator=g, device="cuda", dtype=torch.float64)
    b = (A @ ref).reshape(-1)
    d = torch.zeros(n, device="cuda", dtype=torch.float64)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (rowptr[1:] - rowptr[:-1]).long())
    d[rows[rows == col]] = val[rows == col]
    scale = float(torch.sqrt((b * b / d).sum()))
    x = torch.empty_like(b)
    it, conv, rz = C.c_int(), C.c_int(), C.c_double()

    def solve(tol, limit):
        _lib.check(_lib.lib.impes_pcg_solve(n, _lib.ptr(rowptr), _lib.ptr(col), _lib.ptr(val), _lib.ptr(b), _lib.ptr(x), tol,
                                            limit, C.byref(it), C.byref(conv), C.byref(rz), _lib.stream_of()))
        return it.value, bool(conv.value)

    iters, ok = solve(1e-9 * scale, 5000)
    if float(b @ (b / d)) < 1e-10:        # the reference's start test: nothing to solve
        assert ok and iters == 0
    else:
        assert ok and 0 < iters < 5000
        res = b - (A @ x.reshape(-1, 1)).reshape(-1)
        # the recurrence's r.z against the true residual: equal up to rounding of n eps cond
        assert float(torch.sqrt((res * res / d).sum())) < 2e-9 * scale
        first = x.clone()
        assert solve(1e-9 * scale, 5000) == (iters, True) and torch.equal(first, x)
        assert solve(0.0, 3) == (3, False)
    assert solve(0.0, 0)[0] == 0
