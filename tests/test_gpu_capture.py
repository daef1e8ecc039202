"""V-cycles and value updates captured into a caller's own CUDA graph act on the values of the replay."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _system(dims, precision="fp64"):
    """A hierarchy whose coarse levels are applied as one operator, its values and a right-hand side."""
    from impes_b200 import scenarios
    from impes_b200.amg import ClassicalAMG
    from impes_b200.simulator import build_from_config
    nx, ny, nz = dims
    cfg, f = scenarios.two_phase_2d(seed=5, nx=nx, ny=ny, nz=nz)
    cfg["wells"] = cfg["wells"][:1]
    _, _, _, sim = build_from_config(cfg, f)
    rowptr, col, val, _ = sim.assemble(86400.0)
    n = nx * ny * nz
    levels = 1 if dims == LONG else 10          # one coarsening: a coarsest level of more than 500 rows

    def make():
        return ClassicalAMG((rowptr, col, val, (n, n)), coarsest_size=60, max_levels=levels,
                            mixed_precision=precision == "mixed")
    b = torch.from_numpy(np.random.default_rng(7).standard_normal(n)).cuda()
    return make, val, b


def _scaled(val, top):
    # stays an M-matrix: every value is multiplied by a positive number, the diagonal dominates as before
    return val * torch.linspace(1.0, top, val.numel(), dtype=torch.float64, device=val.device)


def _weakened(val):
    # negative (off-diagonal) values by random factors: an M-matrix whose coarse levels differ from the first's
    g = torch.Generator(device=val.device).manual_seed(3)
    f = torch.rand(val.numel(), generator=g, dtype=torch.float64, device=val.device)
    return torch.where(val < 0, val * f ** 4, val)


def _capture(fn):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = fn()
    return g, out


def _fresh(make, val, b, precision):
    """The V-cycle of a hierarchy that was never captured, at these values (its transfers are those of the first)."""
    amg = make()
    amg.update_values(val)
    return amg.vcycle_scaled(b, precision=precision)


def _close(x, ref, precision):
    # the operator or the levels' sweeps: float64 roundings, or the fp32 level values' through the coarsest solve
    tol = 1e-9 if precision == "fp64" else 2e-3
    return float((x - ref).norm()) <= tol * float(ref.norm())


SHORT, LONG = (45, 45, 1), (40, 44, 1)
CASES = [(SHORT, "fp64"), (SHORT, "mixed"), (LONG, "fp64"), (LONG, "mixed")]


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("dims,precision", CASES)
def test_captured_vcycle_follows_later_values(monkeypatch, dims, precision, graphs):
    if not graphs:
        monkeypatch.setenv("IMPES_NO_GRAPHS", "1")
    make, val, b = _system(dims, precision)
    amg = make()
    amg.vcycle_scaled(b, precision=precision)
    torch.cuda.synchronize()
    g, x = _capture(lambda: amg.vcycle_scaled(b, precision=precision))
    old = _fresh(make, val, b, precision)
    for top in (1.7, 0.4):
        v = _scaled(val, top)
        amg.update_values(v)
        g.replay()
        ref = _fresh(make, v, b, precision)
        assert not _close(old, ref, precision)
        assert _close(x, ref, precision)


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("dims,precision", CASES)
def test_capture_does_not_stand_for_running(monkeypatch, dims, precision, graphs):
    """A V-cycle captured right after an update, never replayed, leaves the next ordinary call right."""
    if not graphs:
        monkeypatch.setenv("IMPES_NO_GRAPHS", "1")
    make, val, b = _system(dims, precision)
    amg = make()
    amg.vcycle_scaled(b, precision=precision)
    v = _scaled(val, 1.7)
    amg.update_values(v)
    torch.cuda.synchronize()
    _capture(lambda: amg.vcycle_scaled(b, precision=precision))
    assert _close(amg.vcycle_scaled(b, precision=precision), _fresh(make, v, b, precision), precision)


@pytest.mark.parametrize("dims,precision", CASES)
def test_failed_capture_leaves_the_solver_usable(dims, precision):
    """A solve cannot be captured (it reads its result on the host): the error leaves the handle as it was."""
    from impes_b200 import _lib
    make, val, b = _system(dims, precision)
    amg = make()
    amg.fgmres(b, tol=1e-10, precision=precision)
    v = _weakened(val)
    amg.update_values(v)
    torch.cuda.synchronize()
    # (by the runtime's own calls: a capture of torch's that fails leaves its allocator on the capture's pool)
    rt = C.CDLL("libcudart.so.12")
    side = torch.cuda.Stream()
    graph = C.c_void_p()
    assert rt.cudaStreamBeginCapture(C.c_void_p(side.cuda_stream), 2) == 0
    try:
        with torch.cuda.stream(side):
            with pytest.raises(_lib.ImpesError):
                amg.fgmres(b, tol=1e-10, precision=precision)
    finally:
        assert rt.cudaStreamEndCapture(C.c_void_p(side.cuda_stream), C.byref(graph)) != 0
        rt.cudaGetLastError()
    torch.cuda.synchronize()
    x, st = amg.fgmres(b, tol=1e-10, precision=precision)
    ref = make()
    ref.update_values(v)
    y, sy = ref.fgmres(b, tol=1e-10, precision=precision)
    assert st["converged"] and st["iterations"] == sy["iterations"]
    # both within the tolerance of ||D^-1 b||, of a system whose solution follows the residual to about 1e2
    assert float((x - y).norm()) <= 1e-7 * float(y.norm())


@pytest.mark.parametrize("dims,precision", CASES)
def test_captured_update_reaches_later_calls(dims, precision):
    """An update replayed from a graph changes what ordinary V-cycles and solves after it use."""
    make, val, b = _system(dims, precision)
    amg = make()
    buf = val.clone()
    amg.update_values(buf)
    amg.vcycle_scaled(b, precision=precision)
    amg.fgmres(b, tol=1e-10, precision=precision)
    torch.cuda.synchronize()
    g, _ = _capture(lambda: amg.update_values(buf))
    assert _close(amg.vcycle_scaled(b, precision=precision), _fresh(make, val, b, precision), precision)
    amg.fgmres(b, tol=1e-10, precision=precision)
    for top in (1.7, 0.4):
        v = _scaled(val, top)
        buf.copy_(v)
        g.replay()
        assert _close(amg.vcycle_scaled(b, precision=precision), _fresh(make, v, b, precision), precision)
        ref = make()
        ref.update_values(v)
        _, st = amg.fgmres(b, tol=1e-10, precision=precision)
        _, sr = ref.fgmres(b, tol=1e-10, precision=precision)
        assert st["converged"] and st["iterations"] == sr["iterations"]


def test_captured_mixed_update_reaches_the_next_fp64_call():
    """A mixed hierarchy's update leaves its fp64 levels to the first fp64 call after it, which forms what that call
    applies; a recorded fp64 V-cycle does not stand for that call."""
    make, val, b = _system(SHORT, "mixed")
    amg = make()
    buf = val.clone()
    amg.update_values(buf)
    amg.vcycle_scaled(b, precision="fp64")
    torch.cuda.synchronize()
    g, _ = _capture(lambda: amg.update_values(buf))
    v = _scaled(val, 1.7)
    buf.copy_(v)
    g.replay()
    torch.cuda.synchronize()
    _capture(lambda: amg.vcycle_scaled(b, precision="fp64"))
    assert _close(amg.vcycle_scaled(b, precision="fp64"), _fresh(make, v, b, "fp64"), "fp64")
    for top in (0.4, 2.5):          # and at every later replay
        v = _scaled(val, top)
        buf.copy_(v)
        g.replay()
        assert _close(amg.vcycle_scaled(b, precision="fp64"), _fresh(make, v, b, "fp64"), "fp64")
        assert _close(amg.vcycle_scaled(b, precision="mixed"), _fresh(make, v, b, "mixed"), "mixed")
