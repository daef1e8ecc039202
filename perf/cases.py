"""Workloads of the IMPES path for timing and comparison, through the package's public entry points.

A case is a dict of plain values.  ``listed()`` gives the named ones, ``draw(rng)``
one more of the same ranges; ``prepare(case, seed)`` builds what a program holds
before the call (rock, state, wells, the simulator or the hierarchy), ``run(state)``
makes one pass and returns its outputs, ``work(case)`` the bytes and operations a
pass cannot do without, and ``exact(case, seed)`` the same outputs as plain 64-bit
torch computes them.

Kinds of case:

* ``step``        ``Simulator.run_step`` from a given mid-life state
* ``assemble``    ``Simulator.assemble`` (pressure matrix and right-hand side)
* ``saturation``  ``Simulator.saturation`` (explicit saturation update)
* ``apply``       ``ClassicalAMG.apply`` (the preconditioner of a caller's own Krylov method)
* ``refresh``     ``ClassicalAMG.update_values`` and ``fgmres`` (new values on a kept hierarchy)
* ``amg_solve``   ``amg_solve`` on a torch sparse matrix (the reference's drop-in call)
* ``build``       ``ClassicalAMG(A)`` and one ``fgmres`` (a new sparsity pattern)
* ``adjoint``     ``adjoint.misfit_gradient`` (history matching: one gradient)
* ``ensemble``    ``Ensemble.run`` (independent realisations stepped together)

Models, as in the package's scenarios: ``two_phase`` (oil-water, one rate injector
and one BHP producer in opposite corners), ``three_phase`` (constant
compressibilities, two injectors and two producers at given rates), ``black_oil``
(PVT, Stone II, capillarity, gravity, four rate injectors around a BHP producer) and
``gas`` (black oil with correlated rock, nine gas injectors, sixteen BHP producers).
"""
import math
import os
import sys
import time

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oil-simulator-py_b200"))

G = 9.81
MD = 9.869233e-16
DAY = 86400.0
DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def _case(name, kind, model, nx, ny, nz, **kw):
    # solves run to where the explicit saturation update no longer sees the solver: 1e-12 of the right-hand side, and
    # 1e-11 where all wells have given rates and rounding leaves more
    d = {"kind": kind, "model": model, "nx": nx, "ny": ny, "nz": nz,
         "precision": "fp64", "cap": 0, "light": 0.0, "tol": 1e-11 if model == "three_phase" else 1e-12}
    d.update(kw)
    if name:
        d["name"] = name
    return d


def listed():
    return [
        # the smallest earnest run: a 2-D water flood, one step (of a hundred), every setting at its default
        _case("step_two_phase_64x64", "step", "two_phase", 64, 64, 1),
        # a field-scale black-oil five-spot on the reference's own hierarchy
        _case("step_black_oil_100x100x20", "step", "black_oil", 100, 100, 20),
        # the million-cell gas injection as the benchmark runs it: fp32 V-cycle inside fp64 FGMRES, interpolation
        # capped at two entries per row, light sweeps on the coarse levels
        _case("step_gas_200x200x25", "step", "gas", 200, 200, 25, precision="mixed", cap=2, light=0.3),
        # a configuration that names no AMG solver runs Jacobi-preconditioned CG; odd sizes
        _case("step_cg_61x53x11", "step", "three_phase", 61, 53, 11, solver="cg"),
        # the two stencil phases of the step, which callers with their own pressure solver use by themselves
        _case("assemble_gas_200x200x25", "assemble", "gas", 200, 200, 25),
        _case("saturation_gas_200x200x25", "saturation", "gas", 200, 200, 25),
        # the preconditioner inside a caller's own Krylov method
        _case("apply_black_oil_83x97x19", "apply", "black_oil", 83, 97, 19),
        # a nonlinear or time loop that keeps its hierarchy: new values, then a solve with the fp32 V-cycle
        _case("refresh_gas_120x110x25", "refresh", "gas", 120, 110, 25, precision="mixed", cap=2),
        # the reference's drop-in call with a torch matrix: cached hierarchy, stand-alone V-cycles
        _case("amg_solve_64x64x8", "amg_solve", "two_phase", 64, 64, 8, tol=1e-6),
        # a new grid or realisation: the hierarchy is built before it is used once
        _case("build_two_phase_47x39x9", "build", "two_phase", 47, 39, 9),
        # history matching: one gradient of the misfit of producer rates
        _case("adjoint_32x32x4", "adjoint", "two_phase", 32, 32, 4, steps=6),
        # uneven realisations stepped together
        _case("ensemble_12", "ensemble", "two_phase", 64, 48, 8, members=12, steps=2, precision="mixed", cap=2, light=0.3),
    ]


def _dims(rng, cells, flat):
    """A grid of about `cells` cells; nz 1 when flat, otherwise 3 to 25 layers."""
    nz = 1 if flat else rng.randint(3, 25)
    area = max(cells / nz, 100.0)
    ratio = math.exp(rng.uniform(-0.7, 0.7))
    return max(10, round(math.sqrt(area * ratio))), max(10, round(math.sqrt(area / ratio))), nz


def draw(rng):
    def cells(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["step", "step", "step", "cg", "assemble", "saturation", "apply", "refresh", "refresh",
                       "amg_solve", "build", "adjoint", "ensemble"])
    mixed = {"precision": "mixed", "cap": rng.choice([2, 3, 4]), "light": rng.choice([0.0, 0.3])}
    if kind == "step":
        if rng.random() < 0.5:     # the capped hierarchy in either precision, up to the largest grid
            mixed["precision"] = rng.choice(["mixed", "mixed", "fp64"])
            model = rng.choice(["gas", "black_oil"])
            return _case(None, kind, model, *_dims(rng, cells(2e4, 8e5), False), **mixed)
        model = rng.choice(["two_phase", "black_oil", "three_phase"])
        return _case(None, kind, model, *_dims(rng, cells(2e3, 8e4), model != "black_oil" and rng.random() < 0.4),
                     precision=rng.choice(["fp64", "mixed"]))
    if kind == "cg":
        return _case(None, "step", "three_phase", *_dims(rng, cells(2e3, 6e4), False), solver="cg")
    if kind in ("assemble", "saturation"):
        model = rng.choice(["two_phase", "black_oil", "gas", "three_phase"])
        return _case(None, kind, model, *_dims(rng, cells(4e3, 1e6), model in ("two_phase", "three_phase") and rng.random() < 0.4))
    if kind == "apply":
        return _case(None, kind, rng.choice(["two_phase", "black_oil"]), *_dims(rng, cells(4e3, 1.5e5), False),
                     cap=rng.choice([0, 0, 2]))
    if kind == "refresh":
        mixed["precision"] = rng.choice(["fp64", "mixed"])
        return _case(None, kind, rng.choice(["two_phase", "gas"]), *_dims(rng, cells(4e3, 3.3e5), rng.random() < 0.2), **mixed)
    if kind == "amg_solve":
        return _case(None, kind, "two_phase", *_dims(rng, cells(4e3, 6e4), rng.random() < 0.4), tol=1e-6)
    if kind == "build":
        return _case(None, kind, rng.choice(["two_phase", "black_oil"]), *_dims(rng, cells(3e3, 2e4), rng.random() < 0.4),
                     cap=rng.choice([0, 2]))
    if kind == "adjoint":
        return _case(None, kind, "two_phase", *_dims(rng, cells(6e2, 4e3), rng.random() < 0.3), steps=rng.randint(2, 6))
    return _case(None, kind, "two_phase", rng.randint(32, 72), rng.randint(32, 64), rng.randint(4, 8),
                 members=rng.randint(3, 12), steps=rng.randint(1, 2), precision="mixed", cap=2, light=0.3)


# ------------------------------------------------------- rock, wells and state
def _pvt_table(rows=20, lo=5.0, hi=40.0):
    t = [i / (rows - 1) for i in range(rows)]
    p = [lo + (hi - lo) * v for v in t]
    a = (0.02 - 0.003) / (1.0 / lo - 1.0 / hi)
    return {"pressure_MPa": p, "Bo": [1.3 - 0.2 * v for v in t], "Bw": [1.02 - 0.02 * v for v in t],
            "Bg": [a / q + 0.02 - a / lo for q in p], "mu_o_cP": [3.0 - 1.5 * v for v in t], "mu_w_cP": [0.5] * rows,
            "mu_g_cP": [0.012 + 0.013 * v for v in t], "Rs_m3m3": [150.0 * v for v in t]}


def _well(name, typ, i, j, k, control, value, phase="water"):
    w = {"name": name, "type": typ, "i": int(i), "j": int(j), "k": int(k), "radius": 0.1,
         "control_type": control, "control_value": value}
    if typ == "injector":
        w["injected_phase"] = phase
    return w


def _config(case):
    """(configuration, time step in days, mean ln k [mD], its deviation) of the case's model."""
    nx, ny, nz, km = case["nx"], case["ny"], case["nz"], case["nz"] // 2
    amg = {"tol": case["tol"], "theta": 0.25, "max_levels": 10, "coarsest_size": 200, "precision": case["precision"],
           "p_max_elements": case["cap"], "light_sweep_rows": int(case["light"] * nx * ny * nz)}
    sim = {"solver_type": "impes", "pressure_solver": "gmres_amg", "amg": amg}
    if case.get("solver") == "cg":
        sim["pressure_solver"] = "cg"
    corey = {"model": "corey", "nw": 2.0, "no": 2.0, "sw_cr": 0.2, "so_r": 0.2}
    if case["model"] == "two_phase":
        fluid = {"pressure": 20.0, "s_w": 0.2, "s_g": 0.0, "mu_oil": 5.0, "mu_water": 1.0, "c_oil": 1e-4, "c_water": 1e-4,
                 "c_rock": 1e-4, "c_gas": 0.0, "relative_permeability": corey}
        wells = [_well("INJ", "injector", 0, 0, 0, "rate", 50.0), _well("PROD", "producer", nx - 1, ny - 1, 0, "bhp", 15.0)]
        grid, dt, lnk, sig, vert = [10.0, 10.0, 5.0], 1.0, 100.0, 0.5, 1.0
    elif case["model"] == "three_phase":
        fluid = {"pressure": 22.0, "s_w": 0.2, "s_g": 0.04, "mu_oil": 1.8, "mu_water": 0.5, "mu_gas": 0.02,
                 "rho_oil": 840.0, "rho_water": 1000.0, "rho_gas": 1.1, "c_oil": 1e-5, "c_water": 5e-6, "c_gas": 1e-3,
                 "c_rock": 1e-5, "relative_permeability": {"nw": 2.0, "no": 2.0, "ng": 2.5, "sw_cr": 0.15, "so_r": 0.2,
                                                           "sg_cr": 0.02}}
        wells = [_well("GI", "injector", 2, ny // 2, km, "rate", 10.0, "gas"),
                 _well("WI", "injector", nx - 3, ny // 2, km, "rate", 10.0),
                 _well("P1", "producer", nx // 2, 3, km, "rate", 10.0),
                 _well("P2", "producer", nx // 2, ny - 4, km, "rate", 10.0)]
        grid, dt, lnk, sig, vert = [10.0, 10.0, 5.0], 1.0, 120.0, 0.6, 0.1
    else:
        pvt = _pvt_table()
        fluid = {"pressure": 25.0, "s_w": 0.2, "s_g": 0.0, "rho_oil": 850.0, "rho_water": 1000.0, "rho_gas": 1.0,
                 "c_rock": 1e-4, "pvt": {"table": pvt}, "capillary_pressure": {"pc_scale": 5.0e4, "pc_exponent": 0.5},
                 "relative_permeability": {"model": "stone2", "nw": 2.0, "no": 2.0, "ng": 2.5, "sw_cr": 0.2, "so_r": 0.2,
                                           "sg_cr": 0.0}}
        grid, vert = [20.0, 20.0, 2.0], 0.1
        if case["model"] == "black_oil":
            wells = [_well("INJ%d" % n, "injector", i, j, km, "rate", 200.0)
                     for n, (i, j) in enumerate([(0, 0), (nx - 1, 0), (0, ny - 1), (nx - 1, ny - 1)])]
            wells.append(_well("PROD", "producer", nx // 2, ny // 2, km, "bhp", 12.0))
            dt, lnk, sig = 5.0, 200.0, 0.8
        else:
            bg0 = float(_interp(torch.tensor(25.0, dtype=F64), pvt["pressure_MPa"], pvt["Bg"]))
            wells = [_well("GI%d%d" % (a, b), "injector", (a + 0.5) * nx / 3, (b + 0.5) * ny / 3, km, "rate", 2.0e5 * bg0, "gas")
                     for a in range(3) for b in range(3)]
            wells += [_well("P%d%d" % (a, b), "producer", a * (nx - 1) / 3, b * (ny - 1) / 3, km, "bhp", 15.0)
                      for a in range(4) for b in range(4)]
            dt, lnk, sig = 2.0, 150.0, 1.0
            amg.update({"theta": 0.2, "max_levels": 20, "coarsest_size": 120})
            sim.update({"global_rate_scale": 0.05, "max_substeps": 20})
    sim["time_step_days"] = dt
    cfg = {"reservoir": {"dimensions": [nx, ny, nz], "grid_size": grid, "porosity": 0.2, "permeability": lnk,
                         "k_vertical_fraction": vert, "c_rock": fluid["c_rock"]},
           "fluid": fluid, "wells": wells, "simulation": sim}
    return cfg, dt, math.log(lnk), sig


def _rock(case, seed, lnk, sig, vert):
    """kx, ky, kz [m2] and porosity from the seed: log-normal per cell, Gaussian-correlated for the gas model."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    shape = (case["nx"], case["ny"], case["nz"])
    z = torch.randn(shape, generator=g, device=DEV, dtype=F64)
    if case["model"] == "gas":
        r = 5
        for ax in range(3):
            n = shape[ax]
            at = torch.arange(n, device=DEV)
            out = torch.zeros_like(z)
            for o in range(-r, r + 1):
                j = (at + o).remainder(2 * n)
                out += math.exp(-0.5 * (o / 2.5) ** 2) * z.index_select(ax, torch.where(j < n, j, 2 * n - 1 - j))
            z = out
        z = (z - z.mean()) / z.std()
    k = torch.exp(lnk + sig * z) * MD
    poro = 0.15 + 0.1 * torch.rand(shape, generator=g, device=DEV, dtype=F64)
    return k, k.clone(), vert * k, poro


def _state(case, seed, cfg):
    """A mid-life state: swept zones around the injectors (none has reached a producer), a hydrostatic column and
    pressure cones around the wells."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 7919)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    i = torch.arange(nx, device=DEV, dtype=F64)[:, None, None]
    j = torch.arange(ny, device=DEV, dtype=F64)[None, :, None]
    k = torch.arange(nz, device=DEV, dtype=F64)[None, None, :]
    fl = cfg["fluid"]
    radius = min(nx, ny) * {"two_phase": 0.35, "three_phase": 0.2, "black_oil": 0.22, "gas": 0.09}[case["model"]]
    p = fl["pressure"] * 1e6 + 850.0 * G * cfg["reservoir"]["grid_size"][2] * (k - nz / 2)
    sw = torch.full((nx, ny, nz), fl["s_w"], device=DEV, dtype=F64)
    sg = torch.full((nx, ny, nz), fl["s_g"], device=DEV, dtype=F64)
    for w in cfg["wells"]:
        d2 = (i - w["i"]) ** 2 + (j - w["j"]) ** 2 + 0.25 * (k - w["k"]) ** 2
        inj = w["type"] == "injector"
        p = p + (2e5 if inj else -2e5) * torch.exp(-d2 / (0.5 * radius) ** 2)
        if not inj:
            continue
        u = torch.rand((nx, ny, nz), generator=g, device=DEV, dtype=F64)
        swept = torch.clamp(torch.exp(-d2 / (radius * (0.8 + 0.2 * float(u[0, 0, 0]))) ** 2) - 0.05, min=0.0) * (0.9 + 0.1 * u)
        if w["injected_phase"] == "gas":
            sg = torch.maximum(sg, 0.35 * swept)
        else:
            sw = torch.maximum(sw, fl["s_w"] + 0.4 * swept)
    return p.reshape(nx, ny, nz).contiguous(), sw, sg


def _inputs(case, seed):
    cfg, dt, lnk, sig = _config(case)
    rock = _rock(case, seed, lnk, sig, cfg["reservoir"]["k_vertical_fraction"])
    return cfg, dt * DAY, rock, _state(case, seed, cfg)


def _matrix(case, seed):
    """A pressure matrix (CSR, columns sorted), the solution a caller looks for and its right-hand side.  The wells
    are rate wells here, so that the matrix is one that a solver of its own could be given."""
    cfg, dt, rock, (p, sw, sg) = _inputs(case, seed)
    cfg["wells"] = [w for w in cfg["wells"] if w["control_type"] == "rate"]
    m = _Model(cfg, rock)
    s = m.system(p, sw, sg, dt)
    rowptr, col, val = s.csr()
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 104729)
    x = (p + 1e5 * torch.randn(p.shape, generator=g, device=DEV, dtype=F64)).reshape(-1)
    if case["kind"] == "amg_solve":    # stand-alone V-cycles are given the pressure change, not the level
        x = x - x.mean()
    return rowptr, col, val, x, s.apply(x)


# -------------------------------------------------------------------- prepare
def _simulator(cfg, rock):
    from impes_b200.simulator import build_from_config
    return build_from_config(cfg, dict(zip(("kx", "ky", "kz", "poro"), rock)), device=DEV)


def _reset(fluid, state):
    fluid.pressure.copy_(state[0])
    fluid.s_w.copy_(state[1])
    fluid.s_g.copy_(state[2])


def _member(case, n):
    """The n-th realisation of an ensemble: the case's grid with its sides varied."""
    f = (1.0, 0.5, 2.0, 0.75, 1.5, 0.625)
    return dict(case, nx=max(16, int(case["nx"] * f[n % 6])), ny=max(16, int(case["ny"] * f[(n // 2 + 3) % 6])),
                nz=case["nz"] if n % 3 else 2 * case["nz"])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "assemble", "saturation"):
        cfg, dt, rock, state = _inputs(case, seed)
        _, fluid, _, sim = _simulator(cfg, rock)
        _reset(fluid, state)
        st = {"kind": kind, "sim": sim, "fluid": fluid, "state": state, "dt": dt}
        if kind == "step":          # the first step of a run builds the hierarchy that the others keep
            sim.run_step(dt)
        elif kind == "saturation":
            cone = torch.linspace(-1e5, 1e5, case["nx"], device=DEV, dtype=F64)[:, None, None]
            st["p_new"] = (state[0] + cone).contiguous()
        return st
    if kind in ("apply", "refresh"):
        from impes_b200.amg import ClassicalAMG
        rowptr, col, val, x, b = _matrix(case, seed)
        gas = case["model"] == "gas"
        amg = ClassicalAMG((rowptr, col, val, (x.numel(), x.numel())), theta=0.2 if gas else 0.25,
                           max_levels=20 if gas else 10, coarsest_size=120 if gas else 200, device=DEV,
                           mixed_precision=case["precision"] == "mixed", p_max_elements=case["cap"],
                           light_sweep_rows=int(case["light"] * x.numel()))
        return {"kind": kind, "amg": amg, "b": b, "val": val, "tol": case["tol"], "precision": case["precision"]}
    if kind == "amg_solve":
        rowptr, col, val, x, b = _matrix(case, seed)
        A = torch.sparse_csr_tensor(rowptr.long(), col.long(), val, size=(x.numel(), x.numel()))
        return {"kind": kind, "A": A, "b": b, "tol": case["tol"]}
    if kind == "build":
        rowptr, col, val, x, b = _matrix(case, seed)
        return {"kind": kind, "csr": (rowptr, col, val, (x.numel(), x.numel())), "b": b, "cap": case["cap"], "tol": case["tol"]}
    if kind == "adjoint":
        cfg, dt, rock, _ = _inputs(case, seed)
        return {"kind": kind, "cfg": cfg, "rock": dict(zip(("kx", "ky", "kz", "poro"), rock)), "dt": dt,
                "steps": case["steps"], "target": _target(case, seed).numpy(), "tol": case["tol"]}
    from impes_b200.ensemble import Ensemble
    members = [_inputs(_member(case, n), seed * 64 + n) for n in range(case["members"])]
    ens = Ensemble([(cfg, dict(zip(("kx", "ky", "kz", "poro"), rock))) for cfg, _, rock, _ in members], device=DEV)
    states = [m[3] for m in members]
    for sim, s in zip(ens.sims, states):
        _reset(sim.fluid, s)
    ens.run(1, members[0][1])
    return {"kind": kind, "ens": ens, "states": states, "dt": members[0][1], "steps": case["steps"]}


def _target(case, seed):
    g = torch.Generator().manual_seed(int(seed) + 15485863)
    return 30.0 + 10.0 * torch.rand((case["steps"], 1), generator=g, dtype=F64)


# ------------------------------------------------------------------------ run
def run(st):
    kind = st["kind"]
    if kind == "step":
        fl = st["fluid"]
        _reset(fl, st["state"])
        st["sim"].run_step(st["dt"])
        return {"p": fl.pressure, "sw": fl.s_w, "sg": fl.s_g, "so": fl.s_o}
    if kind == "assemble":
        rowptr, col, val, rhs = st["sim"].assemble(st["dt"])
        return {"rowptr": rowptr, "col": col, "val": val, "rhs": rhs}
    if kind == "saturation":
        fl = st["fluid"]
        _reset(fl, st["state"])
        n = st["sim"].saturation(st["p_new"], st["dt"])
        return {"sw": fl.s_w, "sg": fl.s_g, "so": fl.s_o, "substeps": n}
    if kind == "apply":
        return {"z": st["amg"].apply(st["b"], cycles=1)}
    if kind == "refresh":
        st["amg"].update_values(st["val"])
        return {"x": st["amg"].fgmres(st["b"], tol=st["tol"], precision=st["precision"])[0]}
    if kind == "amg_solve":
        from impes_b200.amg import amg_solve
        return {"x": amg_solve(st["A"], st["b"], tol=st["tol"], max_cycles=100)}
    if kind == "build":
        from impes_b200.amg import ClassicalAMG
        amg = ClassicalAMG(st["csr"], coarsest_size=200, device=DEV, mixed_precision=False, p_max_elements=st["cap"])
        x = amg.fgmres(st["b"], tol=st["tol"])[0]
        amg.close()
        return {"x": x}
    if kind == "adjoint":
        from impes_b200.adjoint import misfit_gradient
        r = misfit_gradient(st["cfg"], st["rock"], st["target"], st["steps"], st["dt"], checkpoint_every=3,
                            tol=st["tol"], adjoint_tol=st["tol"], device=DEV)
        return {"J": r["J"], "g_lnk": r["g_lnk"], "g_poro": r["g_poro"], "rates": r["rates"]}
    ens = st["ens"]
    for sim, s in zip(ens.sims, st["states"]):
        _reset(sim.fluid, s)
    ens.run(st["steps"], st["dt"])
    return {"p": [s.fluid.pressure for s in ens.sims], "sw": [s.fluid.s_w for s in ens.sims]}


# ----------------------------------------------------------------------- work
def work(case):
    """Each input read once and each output written once; one operation per matrix entry and a few dozen per cell."""
    n = case["nx"] * case["ny"] * case["nz"]
    faces = 3 * n - case["nx"] * case["ny"] - case["ny"] * case["nz"] - case["nx"] * case["nz"]
    nnz = n + 2 * faces
    kind = case["kind"]
    static = 8 * (faces + n)                        # transmissibilities, pore volume
    step = {"bytes": static + 8 * (3 + 4) * n, "flops": 100 * n + 2 * nnz}
    if kind == "step":
        return step
    if kind == "assemble":
        return {"bytes": static + 8 * (3 + 1) * n + 4 * (n + 1) + 12 * nnz, "flops": 100 * n}
    if kind == "saturation":
        return {"bytes": static + 8 * (3 + 3) * n, "flops": 100 * n}
    if kind in ("apply", "refresh", "amg_solve", "build"):
        return {"bytes": 12 * nnz + 4 * (n + 1) + 16 * n, "flops": 2 * nnz}
    if kind == "adjoint":
        return {"bytes": 8 * (4 + 2) * n + 3 * case["steps"] * step["bytes"], "flops": 3 * case["steps"] * step["flops"]}
    total = {"bytes": 0, "flops": 0}
    for m in range(case["members"]):
        w = work(dict(_member(case, m), kind="step"))
        total = {k: total[k] + case["steps"] * w[k] for k in total}
    return total


# ---------------------------------------------------------------------- exact
def _interp(x, xp, fp):
    """Linear interpolation with flat ends."""
    xp, fp = (torch.as_tensor(v, dtype=F64, device=x.device) for v in (xp, fp))
    at = (torch.searchsorted(xp, x.contiguous(), right=True) - 1).clamp(0, xp.numel() - 2)
    y = fp[at] + (fp[at + 1] - fp[at]) / (xp[at + 1] - xp[at]) * (x - xp[at])
    return torch.where(x < xp[0], fp[0], torch.where(x >= xp[-1], fp[-1], y))


def _between(x, lo, hi):
    """min(max(x, lo), hi); a gradient passes on the bounds too."""
    y = torch.where(x < lo, lo + 0.0 * x, x)
    return torch.where(y > hi, hi + 0.0 * y, y)


class _System:
    """A symmetric seven-point system: face coefficients, diagonal, right-hand side."""

    def __init__(self, shape, faces, diag, rhs):
        self.shape, self.faces, self.diag, self.rhs = shape, faces, diag, rhs

    def apply(self, x):
        X = x.reshape(self.shape)
        y = self.diag.reshape(self.shape) * X
        for ax, c in enumerate(self.faces):
            n = self.shape[ax]
            y = y - torch.cat([c * X.narrow(ax, 1, n - 1), torch.zeros_like(X.narrow(ax, 0, 1))], ax)
            y = y - torch.cat([torch.zeros_like(X.narrow(ax, 0, 1)), c * X.narrow(ax, 0, n - 1)], ax)
        return y.reshape(-1)

    def csr(self):
        n = self.diag.numel()
        idx = torch.arange(n, device=self.diag.device).reshape(self.shape)
        cols, vals = [None] * 7, [None] * 7
        for ax, c in enumerate(self.faces):
            stride = math.prod(self.shape[ax + 1:])
            none = torch.zeros_like(self.diag.reshape(self.shape).narrow(ax, 0, 1))
            up, dn = torch.cat([-c, none], ax), torch.cat([none, -c], ax)
            last = self.shape[ax] - 1
            at = idx.div(stride, rounding_mode="floor").remainder(self.shape[ax])
            cols[ax], vals[ax] = torch.where(at > 0, idx - stride, -1), dn
            cols[6 - ax], vals[6 - ax] = torch.where(at < last, idx + stride, -1), up
        cols[3], vals[3] = idx, self.diag.reshape(self.shape)
        cols = torch.stack([c.reshape(-1) for c in cols], 1)
        vals = torch.stack([v.reshape(-1) for v in vals], 1)
        keep = cols >= 0
        rowptr = torch.zeros(n + 1, dtype=torch.int64, device=cols.device)
        rowptr[1:] = keep.sum(1).cumsum(0)
        return rowptr.int(), cols[keep].int(), vals[keep].contiguous()

    def dense(self):
        n = self.diag.numel()
        idx = torch.arange(n, device=self.diag.device).reshape(self.shape)
        at, v = [], []
        for ax, c in enumerate(self.faces):
            m = self.shape[ax] - 1
            a, b = idx.narrow(ax, 0, m).reshape(-1), idx.narrow(ax, 1, m).reshape(-1)
            at += [a * n + b, b * n + a]
            v += [-c.reshape(-1)] * 2
        at.append(torch.arange(n, device=self.diag.device) * (n + 1))
        v.append(self.diag)
        return torch.zeros(n * n, dtype=F64, device=self.diag.device).index_add(0, torch.cat(at), torch.cat(v)).reshape(n, n)

    def solve(self, limit_s=15.0):
        s = self.diag.abs().sqrt()
        if self.diag.numel() <= 5000:
            A = self.dense() / s[:, None] / s[None, :]
            return torch.linalg.solve(A, self.rhs / s) / s
        # conjugate gradients on the scaled system, restarted from the true residual until it stops falling
        x, best, began = torch.zeros_like(s), math.inf, time.monotonic()
        while time.monotonic() - began < limit_s:
            r = (self.rhs - self.apply(x / s)) / s
            rel = float(r.norm() / (self.rhs / s / s).norm())
            if rel > 0.5 * best:
                return x / s if best < 1e-12 else None
            best = rel
            d, rr = r.clone(), r.dot(r)
            stop = float(rr) * 1e-16
            for it in range(6000):
                q = self.apply(d / s) / s
                a = rr / d.dot(q)
                x = x + a * d
                r = r - a * q
                new = r.dot(r)
                d = r + (new / rr) * d
                rr = new
                if it % 32 == 31 and (float(rr) < stop or time.monotonic() - began > limit_s):
                    break
        return None


class _Model:
    """The IMPES step in plain 64-bit torch: two-point fluxes with upwinding, explicit saturations with clamped substeps."""

    def __init__(self, cfg, rock):
        self.cfg, fl = cfg, cfg["fluid"]
        self.shape = tuple(cfg["reservoir"]["dimensions"])
        self.h = cfg["reservoir"]["grid_size"]
        kx, ky, kz, poro = rock
        hx, hy, hz = self.h
        self.T = [2 * k.narrow(ax, 0, n - 1) * k.narrow(ax, 1, n - 1) / (k.narrow(ax, 0, n - 1) + k.narrow(ax, 1, n - 1) + 1e-15) * a
                  for ax, (k, n, a) in enumerate(zip((kx, ky, kz), self.shape, (hy * hz / hx, hx * hz / hy, hx * hy / hz)))]
        self.pv = hx * hy * hz * poro
        self.rp = rp = fl["relative_permeability"]
        self.swc, self.sor, self.sgc = rp["sw_cr"], rp["so_r"], rp.get("sg_cr", 0.0)
        self.table = fl["pvt"]["table"] if "pvt" in fl else None
        self.gravity = self.shape[2] > 1

    def _pvt(self, key, p):
        return _interp(p / 1e6, self.table["pressure_MPa"], self.table[key])

    def _mobilities(self, p, sw, sg):
        rp, fl, span = self.rp, self.cfg["fluid"], 1 - self.swc - self.sor
        s = _between((sw - self.swc) / span, 0.0, 1.0)
        krw, krg = s ** rp["nw"], _between(sg / (span + 1e-10), 0.0, 1.0) ** rp.get("ng", 2.0)
        if rp.get("model") == "stone2":
            kro = torch.clamp((1 - _between((sw - self.swc) / (span + 1e-12), 0.0, 1.0)) ** rp["no"]
                              + (1 - _between((sg - self.sgc) / (1 - self.sgc - self.sor + 1e-12), 0.0, 1.0)) ** rp["ng"] - 1.0, min=0.0)
        else:
            kro = (1 - s) ** rp["no"]
        if self.table:
            mu = [self._pvt(k, p) * 1e-3 for k in ("mu_w_cP", "mu_o_cP", "mu_g_cP")]
        else:
            mu = [fl["mu_water"] * 1e-3, fl["mu_oil"] * 1e-3, fl.get("mu_gas", 0.02) * 1e-3]
        return krw / mu[0], kro / mu[1], krg / mu[2]

    def _densities(self, p):
        fl = self.cfg["fluid"]
        w, o, g = fl.get("rho_water", 1000.0), fl.get("rho_oil", 850.0), fl.get("rho_gas", 1.0)
        if self.table:
            return (w / (self._pvt("Bw", p) + 1e-12), (o + self._pvt("Rs_m3m3", p) * g) / (self._pvt("Bo", p) + 1e-12),
                    g / (self._pvt("Bg", p) + 1e-12))
        return tuple(r * (1 + c / 1e6 * (p - 1e5)) for r, c in ((w, fl["c_water"]), (o, fl["c_oil"]), (g, fl["c_gas"])))

    def _compressibility(self, p, sw, sg):
        fl = self.cfg["fluid"]
        if not self.table:
            return (fl["c_oil"] + fl["c_water"] + fl["c_gas"] + fl["c_rock"]) / 1e6 / 3 + 0.0 * p
        c = [-((self._pvt(k, p + 1e5) - self._pvt(k, p - 1e5)) / 0.2) / (self._pvt(k, p) + 1e-12) / 1e6 for k in ("Bw", "Bo", "Bg")]
        return fl["c_rock"] / 1e6 + sw * c[0] + (1 - sw - sg) * c[1] + sg * c[2]

    def _up(self, v, dp, ax):
        n = self.shape[ax]
        return torch.where(dp.detach() > 0, v.narrow(ax, 0, n - 1), v.narrow(ax, 1, n - 1))

    def _diff(self, v, ax):
        n = self.shape[ax]
        return v.narrow(ax, 0, n - 1) - v.narrow(ax, 1, n - 1)

    def _net_in(self, f):
        """Sum of the face flows (positive towards the higher index) into each cell."""
        out = 0.0
        for ax, v in enumerate(f):
            none = torch.zeros_like(self.pv.narrow(ax, 0, 1))
            out = out + torch.cat([none, v], ax) - torch.cat([v, none], ax)
        return out

    def _wells(self):
        scale = float(self.cfg["simulation"].get("global_rate_scale", 1.0))
        wi = 2 * math.pi * 100.0 / (math.log(0.28 * math.sqrt(2.0) / 2 / 0.1) + 1e-12)
        for w in self.cfg["wells"]:
            sign = 1.0 if w["type"] == "injector" else -1.0
            yield (w["i"], w["j"], w["k"]), w, sign, wi, sign * w["control_value"] * scale / DAY

    def system(self, p, sw, sg, dt):
        mw, mo, mg = self._mobilities(p, sw, sg)
        mt = mw + mo + mg
        dp = [self._diff(p, ax) for ax in range(3)]
        faces = [t * self._up(mt, d, ax) for ax, (t, d) in enumerate(zip(self.T, dp))]
        self.acc = self.pv * self._compressibility(p, sw, sg) / dt
        diag = self.acc
        for ax, c in enumerate(faces):
            none = torch.zeros_like(self.pv.narrow(ax, 0, 1))
            diag = diag + torch.cat([c, none], ax) + torch.cat([none, c], ax)
        self.buoyancy = torch.zeros_like(self.pv)
        if self.gravity:
            flow = 0.0
            for m, rho in zip((mw, mo, mg), self._densities(p)):
                flow = flow + self._up(m, dp[2], 2) * self._up(rho, dp[2], 2)
            self.buoyancy = self._net_in([torch.zeros_like(self.T[0]), torch.zeros_like(self.T[1]), self.T[2] * G * self.h[2] * flow])
        rhs = self.acc * p + self.buoyancy
        pc = self.cfg["fluid"].get("capillary_pressure")
        if pc:
            s = _between((sw - self.swc) / (1 - self.swc - self.sor), 0.0, 1.0)
            cap = pc["pc_scale"] * (1 - s + 1e-6) ** -pc["pc_exponent"]
            rhs = rhs + self._net_in([-t * self._up(mo, d, ax) * self._diff(cap, ax) for ax, (t, d) in enumerate(zip(self.T, dp))])
        for c, w, _, wi, q in self._wells():
            at = tuple(torch.tensor([v], device=p.device) for v in c)
            if w["control_type"] == "rate":
                rhs = rhs.index_put(at, torch.tensor([q], dtype=F64, device=p.device), accumulate=True)
            else:
                d = (wi * mt[c]).reshape(1)
                diag = diag.index_put(at, d, accumulate=True)
                rhs = rhs.index_put(at, d * (w["control_value"] * 1e6), accumulate=True)
        self.faces, self.fo = faces, mo / (mt + 1e-10)
        return _System(self.shape, faces, diag.reshape(-1), rhs.reshape(-1))

    def oil_rates(self, p_new, p):
        """Producer oil rates [m3/d] from the balance of each producer's cell in the last system."""
        net = self._net_in([c * self._diff(p_new, ax) for ax, c in enumerate(self.faces)])
        q = (net - self.acc * (p_new - p) + self.buoyancy) * self.fo * DAY
        return torch.stack([q[c] for c, w, *_ in self._wells() if w["type"] == "producer"])

    def saturation(self, p, sw, sg, dt):
        prm = self.cfg["simulation"]
        mw, mo, mg = self._mobilities(p, sw, sg)
        mt = mw + mo + mg
        dp = [self._diff(p, ax) for ax in range(3)]
        rw, _, rg = self._densities(p)

        def net(m, rho):
            pot = list(dp)
            if self.gravity:
                n = self.shape[2]
                pot[2] = dp[2] + G * 0.5 * (rho.narrow(2, 0, n - 1) + rho.narrow(2, 1, n - 1)) * self.h[2]
            return self._net_in([t * self._up(m, d, ax) * u for ax, (t, d, u) in enumerate(zip(self.T, dp, pot))])

        qw, qg = net(mw, rw), net(mg, rg)
        for c, w, sign, wi, q in self._wells():
            at = tuple(torch.tensor([v], device=p.device) for v in c)
            gas = w.get("injected_phase") == "gas"
            if w["control_type"] == "rate" and sign > 0:
                s, other = (sg[c], sw[c]) if gas else (sw[c], sg[c])
                room = torch.clamp(1.0 - self.sor - other - s, min=0.0) / torch.clamp(dt / self.pv[c] * q, min=1e-12)
                q = q * torch.clamp(room, 0.0, 1.0) if float(room.detach()) < 1.0 else torch.tensor(q, dtype=F64, device=p.device)
                qw, qg = (qw, qg.index_put(at, q.reshape(1), accumulate=True)) if gas else (qw.index_put(at, q.reshape(1), accumulate=True), qg)
                continue
            if w["control_type"] == "bhp":
                q = -wi * mt[c] * (p[c] - w["control_value"] * 1e6)
            for_w, for_g = q * mw[c] / (mt[c] + 1e-10), q * mg[c] / (mt[c] + 1e-10)
            qw, qg = qw.index_put(at, for_w.reshape(1), accumulate=True), qg.index_put(at, for_g.reshape(1), accumulate=True)
        dw, dg = dt / self.pv * qw, dt / self.pv * qg
        with torch.no_grad():
            up = torch.clamp(1.0 - self.sor - sw - sg, min=0.0)
            worst = 0.0
            for d, down in ((dw, sw - self.swc), (dg, sg - self.sgc)):
                r = torch.where(d > 0, d / torch.clamp(up, min=1e-12), -d / torch.clamp(down, min=1e-12))
                worst = max(worst, float(r.max()), float(d.abs().max()) / prm.get("max_saturation_change", 0.05))
            n = min(max(int(math.ceil(worst)), 1), int(prm.get("max_substeps", 20))) if math.isfinite(worst) else 1
        for _ in range(n):
            sw, sg = sw + dw / n, sg + dg / n
            sw = _between(sw, self.swc, 1.0 - self.sor - sg)
            sg = _between(sg, self.sgc, 1.0 - self.sor - sw)
        return sw, sg, n


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "assemble", "saturation"):
        cfg, dt, rock, (p, sw, sg) = _inputs(case, seed)
        m = _Model(cfg, rock)
        if kind == "saturation":
            cone = torch.linspace(-1e5, 1e5, case["nx"], device=DEV, dtype=F64)[:, None, None]
            sw, sg, _ = m.saturation(p + cone, sw, sg, dt)
            return {"sw": sw, "sg": sg, "so": 1 - sw - sg, "substeps": None}
        s = m.system(p, sw, sg, dt)
        if kind == "assemble":
            return {"rowptr": None, "col": None, "val": s.csr()[2], "rhs": s.rhs}
        x = s.solve()
        if x is None:
            return None
        x = x.reshape(p.shape)
        sw, sg, _ = m.saturation(x, sw, sg, dt)
        return {"p": x, "sw": sw, "sg": sg, "so": 1 - sw - sg}
    if kind == "apply":
        return None                    # a preconditioner's result is what its hierarchy makes it
    if kind in ("refresh", "amg_solve", "build"):
        return {"x": _matrix(case, seed)[3]}
    if kind == "adjoint":
        if case["nx"] * case["ny"] * case["nz"] > 4500:
            return None
        cfg, dt, (kx, ky, kz, poro), _ = _inputs(case, seed)
        lnk = torch.log(kx).requires_grad_(True)
        phi = poro.clone().requires_grad_(True)
        m = _Model(cfg, (torch.exp(lnk), torch.exp(lnk) * (ky / kx), torch.exp(lnk) * (kz / kx), phi))
        p = torch.full(m.shape, cfg["fluid"]["pressure"] * 1e6, dtype=F64, device=DEV)
        sw = torch.full(m.shape, cfg["fluid"]["s_w"], dtype=F64, device=DEV)
        sg, rates = torch.zeros_like(sw), []
        for _ in range(case["steps"]):
            x = m.system(p, sw, sg, dt).solve().reshape(m.shape)
            rates.append(m.oil_rates(x, p))
            sw, p = m.saturation(x, sw, sg, dt)[0], x
        rates = torch.stack(rates)
        J = ((rates - _target(case, seed).to(DEV)) ** 2).sum()
        gl, gp = torch.autograd.grad(J, (lnk, phi))
        return {"J": J.detach(), "g_lnk": gl, "g_poro": gp, "rates": rates.detach()}
    ps, sws = [], []
    for n in range(case["members"]):
        cfg, dt, rock, (p, sw, sg) = _inputs(_member(case, n), seed * 64 + n)
        m = _Model(cfg, rock)
        for _ in range(case["steps"]):
            x = m.system(p, sw, sg, dt).solve(limit_s=1.5)
            if x is None:
                return None
            p = x.reshape(p.shape)
            sw, _, _ = m.saturation(p, sw, sg, dt)
        ps.append(p)
        sws.append(sw)
    return {"p": ps, "sw": sws}
