"""Balances of the saturation update where densities are not numbers and where wells are many, against the oracle."""
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


# more wells than blocks: several a warp, every thread of a block at work; the largest number; wells that share a cell
@pytest.mark.parametrize("dims,wells", [((10, 10, 1), 30), ((16, 16, 1), 120), ((40, 40, 2), 256), ((3, 3, 1), 12)])
def test_many_wells_on_small_models(dims, wells):
    from impes_b200.simulator import build_from_config
    from oracle.impes import Model
    rows = 8
    t = np.linspace(0.0, 1.0, rows)
    table = {"pressure_MPa": list(5.0 + 35.0 * t), "Bo": list(1.3 - 0.2 * t), "Bw": list(1.02 - 0.02 * t),
             "Bg": list(0.02 - 0.015 * t), "mu_o_cP": list(3.0 - 1.5 * t), "mu_w_cP": [0.5] * rows,
             "mu_g_cP": list(0.012 + 0.013 * t), "Rs_m3m3": list(150.0 * t)}
    rng = np.random.default_rng(wells)
    ws = []
    for q in range(wells):
        w = {"name": "W%d" % q, "i": int(rng.integers(dims[0])), "j": int(rng.integers(dims[1])), "k": int(rng.integers(dims[2])),
             "radius": 0.1}
        if q % 3 == 0:
            w.update(type="injector", control_type="rate", control_value=2.0, injected_phase="gas" if q % 2 else "water")
        elif q % 3 == 1:
            w.update(type="producer", control_type="bhp", control_value=15.0)
        else:
            w.update(type="producer", control_type="rate", control_value=1.5)
        ws.append(w)
    cfg = {"reservoir": {"dimensions": list(dims), "grid_size": [20.0, 20.0, 5.0], "porosity": 0.2, "permeability": 100.0,
                         "k_vertical_fraction": 0.1, "c_rock": 1e-4},
           "fluid": {"pressure": 20.0, "s_w": 0.3, "s_g": 0.1, "rho_oil": 850.0, "rho_water": 1000.0, "rho_gas": 1.0,
                     "c_rock": 1e-4, "pvt": {"table": table},
                     "relative_permeability": {"model": "corey", "nw": 2.0, "no": 2.0, "ng": 2.0, "sw_cr": 0.2,
                                               "so_r": 0.2, "sg_cr": 0.0}},
           "wells": ws, "simulation": {"solver_type": "impes", "time_step_days": 1.0, "max_substeps": 20}}
    k = 1e-13 * np.exp(0.4 * rng.standard_normal(dims))
    fields = {"kx": k, "ky": k, "kz": 0.1 * k, "poro": np.full(dims, 0.2)}
    m = Model(cfg, fields["kx"], fields["ky"], fields["kz"], fields["poro"])
    n = int(np.prod(dims))
    p = 20e6 * (1.0 + 0.02 * rng.standard_normal(n))
    _, fl, _, sim = build_from_config(cfg, fields)
    for _ in range(2):           # the balances run on
        sub = m.saturation(p.copy(), 86400.0)
        assert sim.saturation(torch.tensor(p, device="cuda").reshape(dims), 86400.0) == sub
    assert sub > 1 or dims == (3, 3, 1)
    assert np.abs(fl.s_w.cpu().numpy().ravel() - m.sw).max() <= 1e-12
    assert np.abs(fl.s_g.cpu().numpy().ravel() - m.sg).max() <= 1e-12
    for got, ref in ((sim.mass_balance, m.mass_balance), (sim.component_balance, m.component_balance)):
        for ph in ref:
            scale = max(abs(v) for v in ref[ph].values())
            for way in ref[ph]:
                # sums of at most a few thousand addends in another order
                assert abs(got[ph][way] - ref[ph][way]) <= 1e-11 * max(scale, 1e-300), (ph, way)
