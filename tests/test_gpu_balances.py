"""Balances of the saturation update where the densities are not numbers, against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# an unchanged cell (no flux, no well) whose density the table cannot give: its zero mass times NaN or infinity is NaN,
# in the balances of that phase only
@pytest.mark.parametrize("key,value", [("Bg", float("nan")), ("Bw", float("nan")), ("Bo", float("nan")),
                                       ("Rs_m3m3", float("nan")), ("Rs_m3m3", float("inf")), ("Bw", -1e-12), (None, 0.0)])
def test_balances_of_unchanged_cells(key, value):
    from impes_b200.simulator import build_from_config
    from oracle.impes import Model
    rows = 8
    t = np.linspace(0.0, 1.0, rows)
    table = {"pressure_MPa": list(5.0 + 35.0 * t), "Bo": list(1.3 - 0.2 * t), "Bw": list(1.02 - 0.02 * t),
             "Bg": list(0.02 - 0.015 * t), "mu_o_cP": list(3.0 - 1.5 * t), "mu_w_cP": [0.5] * rows,
             "mu_g_cP": list(0.012 + 0.013 * t), "Rs_m3m3": list(150.0 * t)}
    if key:
        table[key] = table[key][:-2] + [value, value]
    nx, ny = 24, 20
    cfg = {"reservoir": {"dimensions": [nx, ny, 1], "grid_size": [10.0, 10.0, 5.0], "porosity": 0.2,
                         "permeability": 100.0, "k_vertical_fraction": 1.0, "c_rock": 1e-4},
           "fluid": {"pressure": 39.0, "s_w": 0.3, "s_g": 0.1, "rho_oil": 850.0, "rho_water": 1000.0, "rho_gas": 1.0,
                     "c_rock": 1e-4, "pvt": {"table": table},
                     "relative_permeability": {"model": "corey", "nw": 2.0, "no": 2.0, "ng": 2.0, "sw_cr": 0.2,
                                               "so_r": 0.2, "sg_cr": 0.0}},
           "wells": [], "simulation": {"solver_type": "impes", "time_step_days": 1.0}}
    one = np.ones((nx, ny, 1))
    fields = {"kx": 1e-13 * one, "ky": 1e-13 * one, "kz": 1e-13 * one, "poro": 0.2 * one}
    m = Model(cfg, fields["kx"], fields["ky"], fields["kz"], fields["poro"])
    with np.errstate(invalid="ignore", divide="ignore", over="ignore"):
        m.saturation(m.p.copy(), 86400.0)
    _, fl, _, sim = build_from_config(cfg, fields)
    sw = fl.s_w.clone()
    sim.saturation(fl.pressure.clone(), 86400.0)
    assert torch.equal(fl.s_w, sw)
    got = sim.mass_balance
    for ph in ("water", "oil", "gas"):
        for way in ("in", "out"):
            assert np.array_equal(np.float64(got[ph][way]), np.float64(m.mass_balance[ph][way]), equal_nan=True), (ph, way)
