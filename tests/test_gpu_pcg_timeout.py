"""The one-launch CG's waits are bounded: a wait that runs out is an error, and the context stays usable."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


# at most one row a thread, and several
@pytest.mark.parametrize("dims", [(17, 13, 3), (61, 53, 40)])
def test_wait_that_runs_out(dims):
    from impes_b200 import _lib, scenarios
    from impes_b200.simulator import build_from_config
    cfg, f = scenarios.two_phase_2d(seed=2, nx=dims[0], ny=dims[1], nz=dims[2])
    cfg["wells"] = cfg["wells"][:1]
    _, _, _, sim = build_from_config(cfg, f)
    rowptr, col, val, b = sim.assemble(3600.0)
    n = b.numel()
    x = torch.full_like(b, 7.0)
    it, conv, rz = C.c_int(), C.c_int(), C.c_double()

    def solve(polls):
        rc = _lib.lib.impes_pcg_solve_bounded(n, _lib.ptr(rowptr), _lib.ptr(col), _lib.ptr(val), _lib.ptr(b), _lib.ptr(x),
                                              1e-3, 2000, polls, C.byref(it), C.byref(conv), C.byref(rz), _lib.stream_of())
        torch.cuda.synchronize()
        return rc

    assert solve(0) == _lib.ERR_TIMEOUT
    assert b"barrier" in _lib.lib.impes_last_error()
    assert solve(1 << 22) == 0 and conv.value == 1 and it.value > 0
    first, its = x.clone(), it.value
    assert solve(0) == _lib.ERR_TIMEOUT
    assert solve(1 << 22) == 0 and it.value == its and torch.equal(x, first)
    assert solve(-1) == _lib.ERR_ARG
