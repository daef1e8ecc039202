"""What a solve that meets a NaN leaves behind: an error, and the caller's vectors as they were."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


# a NaN and an infinity in the right-hand side, a NaN in the first iterate; solves driven by a graph and by the host
@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("where", ["nan_b", "inf_b", "nan_x0"])
def test_fgmres_reports_nan_and_leaves_x(monkeypatch, where, graphs):
    from impes_b200 import _lib, scenarios
    from impes_b200.amg import ClassicalAMG
    from impes_b200.simulator import build_from_config
    if not graphs:
        monkeypatch.setenv("IMPES_NO_GRAPHS", "1")
    cfg, f = scenarios.two_phase_2d(seed=4, nx=33, ny=29, nz=1)
    _, _, _, sim = build_from_config(cfg, f)
    rowptr, col, val, b = sim.assemble(86400.0)
    n = b.numel()
    amg = ClassicalAMG((rowptr, col, val, (n, n)), coarsest_size=60, mixed_precision=False)
    x = torch.linspace(1.0, 2.0, n, dtype=torch.float64, device=b.device)
    b = b.clone()
    use_x0 = 1 if where == "nan_x0" else 0
    if where == "nan_x0":
        x[5] = float("nan")
    else:
        b[n // 2] = float("nan") if where == "nan_b" else float("inf")
    before = x.clone()
    kp = _lib.KrylovParams(1e-8, 30, 100, 1, 0, use_x0)
    st = _lib.KrylovStats()
    for _ in range(2):          # the first call captures, the second replays
        rc = _lib.lib.impes_amg_fgmres(amg.handle, _lib.ptr(b), _lib.ptr(x), C.byref(kp), C.byref(st),
                                       _lib.stream_of(b.device))
        torch.cuda.synchronize()
        assert rc == _lib.ERR_NAN
        assert torch.equal(x.view(torch.int64), before.view(torch.int64))


# a step driven from the host (the first), and one replayed from its graph
@pytest.mark.parametrize("steps", [0, 3])
def test_step_with_nan_leaves_the_state(steps):
    from impes_b200 import _lib, scenarios
    from impes_b200.simulator import build_from_config
    cfg, f = scenarios.two_phase_2d(seed=4, nx=33, ny=29, nz=1)
    _, fl, wm, sim = build_from_config(cfg, f)
    for _ in range(steps):
        assert sim.run_step(86400.0)
    before = [t.clone() for t in (fl.pressure, fl.s_w, fl.s_g)]
    well = wm.get_wells()[0]
    value = well.control_value
    well.control_value = float("nan")
    with pytest.raises(_lib.ImpesError):
        sim.run_step(86400.0)
    torch.cuda.synchronize()
    for t, b in zip((fl.pressure, fl.s_w, fl.s_g), before):
        assert torch.equal(t, b)
    well.control_value = value
    assert sim.run_step(86400.0)
    assert bool(torch.isfinite(fl.pressure).all()) and bool(torch.isfinite(fl.s_w).all())
