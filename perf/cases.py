"""Performance cases of the chemistry library.

What a flow solver does with this library each time step: the chemistry step
itself (plain integrator, surrogate with its FP64 fallback, table, on device
fields and through the host arrays), the species predictor, the diffusion
coefficients and the state equation around it, and the training of the
surrogate.  `listed()` gives the cases, `draw()` more of the same ranges,
`prepare()` the device (or host) state of a case, `run()` one pass through
the public entry points, `work()` its algorithmic bytes and flops,
`tolerance()` the agreement two correct implementations show, and `exact()`
a 64-bit torch restatement where one is affordable.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import nrg_b200
from nrg_b200 import surrogate as nrg_surrogate
from nrg_b200.chemistry import ChemicalKineticsSolver, DataManager, mechanism_tables, transport_tables

RG, P_ATM, T_REF = 8.31446261815324, 101325.0, 298.15
DEV = "cuda:0"
RADICALS = {"H2": ["H", "O", "OH", "HO2", "H2O2"], "C2H2": ["H", "O", "OH", "HO2", "HCO", "CH3", "HCCO"]}


# --------------------------------------------------------------------- cases
def listed() -> list:
    return [
        # the smallest block a solver hands over at once: 64 x 64 burning cells
        dict(name="step_small", kind="step", mech="KEROMNES", mode="fast", field="random", nx=64, ny=64, nz=1,
             dt=1e-6, launch="default"),
        # the headline field: a premixed flame on 2048 x 2048 cells, launch shape as the autotuner picks it there
        dict(name="step_flame", kind="step", mech="KEROMNES", mode="fast", field="flame", nx=2048, ny=2048, nz=1,
             dt=1e-6, launch="autotuned"),
        # ignition: long steps, a fifth of the cells near the temperature that ignites within the step
        dict(name="step_ignition", kind="step", mech="KEROMNES", mode="fast", field="ignition", nx=512, ny=512, nz=1,
             dt=1e-5, launch="autotuned"),
        # reference mode (the Fortran's finite-difference Jacobian and roundings) on a ragged
        # block of wide-range states with pressures of 0.5 to 5 atm
        dict(name="step_reference", kind="step", mech="KEROMNES", mode="reference", field="wide", nx=181, ny=113,
             nz=1, dt=1e-6, launch="default"),
        # a larger H2/air mechanism (13 species, 71 reactions) on an ordinary flame block
        dict(name="step_konnov", kind="step", mech="KONNOV", mode="fast", field="flame", nx=512, ny=384, nz=1,
             dt=1e-6, launch="default"),
        # networks, gate and FP64 fallback on the headline field
        dict(name="surrogate_flame", kind="step", mech="KEROMNES", mode="surrogate", field="flame", nx=2048, ny=2048,
             nz=1, dt=1e-6, launch="autotuned"),
        # the drop-in call on the solver's own Fortran-layout host arrays, ghost layer and odd extents
        dict(name="host_block", kind="host", mech="KEROMNES", mode="surrogate", field="flame", nx=1021, ny=1023,
             nz=1, dt=1e-6, launch="default"),
        # table_approximated mode: the streaming step of a tabulated flame
        dict(name="table_flame", kind="table", mech="KEROMNES", field="flame", nx=2048, ny=2048, nz=1, dt=1e-6,
             rows=1134),
        # chemistry sources into the state, then the state equation, over the field
        dict(name="state_flame", kind="state", mech="KEROMNES", field="flame", nx=2048, ny=2048, nz=1, dt=1e-6,
             dims=2),
        # convective species predictor of the low-Mach solver on a 2-D block
        dict(name="predictor_2d", kind="predictor", mech="KEROMNES", nx=2048, ny=2048, nz=1, dt=1e-7),
        # mixture-averaged diffusion coefficients over the field
        dict(name="diffusivity_flame", kind="diffusivity", mech="KEROMNES", field="flame", nx=2048, ny=2048, nz=1),
        # training: forward, backward and Adam over 32 batches
        dict(name="train", kind="train", mech="KEROMNES", n=131072, batch=4096),
    ]


def _log_int(rng, lo: float, hi: float) -> int:
    return max(int(lo), min(int(hi), int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["step", "step", "step", "step", "surrogate", "host", "table", "state", "predictor",
                       "diffusivity", "train"])
    if kind == "train":
        batch = rng.choice([1024, 2048, 4096])
        return dict(kind="train", mech="KEROMNES", n=batch * rng.randint(4, 24) + rng.randint(0, 500), batch=batch)
    # cells of the block, log-uniform up to the largest that costs what the listed cases cost
    mech = rng.choice(["KEROMNES", "KEROMNES", "KEROMNES", "ZHANG", "TEREZA", "KONNOV", "ACETYLENE"])
    field = rng.choice(["flame", "flame", "random", "ignition", "wide"])
    mode = rng.choice(["fast", "fast", "fast", "fast", "mixed", "reference"])
    if kind in ("surrogate", "host", "table"):
        mech, field, mode = "KEROMNES", "flame", "surrogate"
    if kind == "host":
        mode = rng.choice(["surrogate", "fast"])
    if mode == "mixed":
        mech = "KEROMNES"
    if mech == "ACETYLENE" and (field == "ignition" or kind == "diffusivity"):
        mech = "ZHANG"
    if kind == "predictor" and mech == "ACETYLENE":
        mech = "TEREZA"
    top = 3.0e6
    if kind == "step":
        top = {"flame": 1.0e6, "random": 4e5, "ignition": 6e4, "wide": 6e4}[field]
        top /= {"KEROMNES": 1.0, "ZHANG": 1.2, "TEREZA": 2.5, "KONNOV": 6.0, "ACETYLENE": 5.0}[mech]
        top /= {"fast": 1.0, "mixed": 1.5, "reference": 8.0}[mode]
    elif kind == "host":
        top = 6e5
    n = _log_int(rng, 700.0 if kind in ("step", "surrogate", "host") else 2.0e4, top)
    nz = rng.choice([1, 1, 1, 5, 12])
    nx = max(3, int(round(math.sqrt(n / nz) * rng.uniform(0.6, 1.6))))
    ny = max(2, n // (nx * nz))
    case = dict(kind="step" if kind == "surrogate" else kind, mech=mech, nx=nx, ny=ny, nz=nz)
    if kind != "predictor":
        case["field"] = field
    if kind in ("step", "surrogate", "host"):
        case.update(mode=mode, launch=rng.choice(["default", "autotuned"]))
    if kind == "table":
        case["rows"] = _log_int(rng, 40, 4000)
    if kind == "state":
        case["dims"] = rng.choice([1, 2, 3])
    if kind != "diffusivity":
        long_step = kind == "step" and (field == "ignition" or (field == "wide" and mode != "reference"))
        case["dt"] = 1e-7 if kind == "predictor" else 1e-5 if long_step else 1e-6
    return case


# -------------------------------------------------------------------- fields
_TABLES: dict = {}


def _tables(mech: str) -> dict:
    """Constants of the mechanism's input decks."""
    if mech not in _TABLES:
        t = mechanism_tables(*nrg_b200.mechanism_paths(mech), 1.0, nrg_b200.eact_units(mech))
        t["names"] = _solver(mech).species_names
        _TABLES[mech] = t
    return _TABLES[mech]


_SOLVERS: dict = {}


def _solver(mech: str, use: str = "") -> ChemicalKineticsSolver:
    """The handle a program keeps for a mechanism and a use of it."""
    key = (mech, use)
    if key not in _SOLVERS:
        s = ChemicalKineticsSolver(None, *nrg_b200.mechanism_paths(mech), E_act_units=nrg_b200.eact_units(mech),
                                   mode="fast")
        if use == "surrogate":
            nrg_surrogate.load_default(s)
        if use.startswith("table"):
            s.set_table(*(a.cpu().numpy() for a in _chem_table(mech, int(use[5:]))))
            s.set_mode("table")
        if use == "diffusivity":
            s.load_transport(nrg_b200.transport_path(mech))
        _SOLVERS[key] = s
    return _SOLVERS[key]


def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEV)
    g.manual_seed(0x5EED + 7919 * int(seed))
    return g


def _uniform(g, shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, generator=g, dtype=torch.float64, device=DEV)


def _mixture(mech: str):
    """Mass fractions of the stoichiometric reactants and of their products."""
    t = _tables(mech)
    W, idx = torch.tensor(t["molar_mass"], device=DEV), {s: i for i, s in enumerate(t["names"])}
    if mech == "ACETYLENE":
        re, pr, rad = {"C2H2": 2.0, "O2": 5.0, "AR": 16.33}, {"CO2": 4.0, "H2O": 2.0, "AR": 16.33}, RADICALS["C2H2"]
    else:
        re, pr, rad = {"H2": 2.0, "O2": 1.0, "N2": 3.762}, {"H2O": 2.0, "N2": 3.762}, RADICALS["H2"]
    Y = []
    for mix in (re, pr):
        x = torch.zeros(len(W), dtype=torch.float64, device=DEV)
        for s, v in mix.items():
            x[idx[s]] = v * W[idx[s]]
        Y.append(x / x.sum())
    return W, Y[0], Y[1], [idx[s] for s in rad]


def _field(case: dict, seed: int):
    """(T, p, rho, Y[N, n]) of a case's cells, i along x fastest."""
    g = _generator(seed)
    W, Yr, Yp, rad = _mixture(case["mech"])
    nx, rows = case["nx"], case["ny"] * case["nz"]
    n = nx * rows
    peak = 1e-4 if case["mech"] == "ACETYLENE" else 1e-3
    if case["field"] == "flame":
        # tanh front of 0.5 mm on 10 um cells, 300 to 2400 K, wrinkled by 8 sinusoids of 0.2 mm
        dx, delta = 10e-6, 0.5e-3
        modes = torch.randint(1, 17, (8, 1), generator=g, device=DEV).to(torch.float64)
        phase = _uniform(g, (8, 1), 0.0, 2.0 * math.pi)
        y = (torch.arange(rows, dtype=torch.float64, device=DEV) + 0.5) / rows
        xf = 0.5 * nx * dx + 0.2e-3 * torch.sin(2.0 * math.pi * modes * y[None, :] + phase).sum(0)
        s = ((torch.arange(nx, dtype=torch.float64, device=DEV) + 0.5) * dx - xf[:, None]).reshape(-1) / delta
        c = 0.5 * (1.0 + torch.tanh(s))
        T = 300.0 + 2100.0 * c
        p = torch.full((n,), P_ATM, dtype=torch.float64, device=DEV)
        radical = [peak * torch.exp(-0.5 * s * s)] * len(rad)
    else:
        lo, hi = (800.0, 2600.0) if case["field"] == "wide" else (1000.0, 2400.0)
        T, c = _uniform(g, n, lo, hi), _uniform(g, n)
        if case["field"] == "ignition":
            # a fifth of the cells within 50 K of the temperature whose ignition delay is 1e-5 s
            T = torch.where(_uniform(g, n) < 0.2, 1586.9 + _uniform(g, n, -50.0, 50.0), T)
        p = P_ATM * (_uniform(g, n, 0.5, 5.0) if case["field"] == "wide" else torch.ones(n, dtype=torch.float64,
                                                                                        device=DEV))
        radical = [peak * 10.0 ** _uniform(g, n, -5.0, 0.0) for _ in rad]
    Y = (1.0 - c)[None, :] * Yr[:, None] + c[None, :] * Yp[:, None]
    for k, v in zip(rad, radical):
        Y[k] = v
    Y = (Y / Y.sum(0, keepdim=True)).contiguous()
    rho = p / (RG * T * (Y / W[:, None]).sum(0))
    return T.contiguous(), p, rho.contiguous(), Y


def _energy(mech: str, T, Y):
    """E_f [J/kg] whose state equation gives T back, and the mean molar mass."""
    W = torch.tensor(_tables(mech)["molar_mass"], device=DEV)
    avg = 1.0 / (Y / W[:, None]).sum(0)
    X = Y / W[:, None] * avg
    e = (_enthalpy(mech, T) * X).sum(0) - RG * T - (_enthalpy(mech, torch.full_like(T[:1], T_REF)) * X).sum(0)
    return e / avg, avg


def _nasa(mech: str, T):
    a = torch.tensor(_tables(mech)["a_coeffs"], device=T.device)
    hot = (T >= 1000.0)[None, :]
    return [torch.where(hot, a[:, 1, i, None], a[:, 0, i, None]) for i in range(7)]


def _enthalpy(mech: str, T):
    a, t = _nasa(mech, T.clamp(max=6000.0)), T.clamp(max=6000.0)
    return ((((a[4] / 5 * t + a[3] / 4) * t + a[2] / 3) * t + a[1] / 2) * t + a[0]) * t + a[5]


def _cp(mech: str, T):
    a, t = _nasa(mech, T.clamp(max=6000.0)), T.clamp(max=6000.0)
    return (((a[4] * t + a[3]) * t + a[2]) * t + a[1]) * t + a[0]


def _configure(solver, case: dict) -> None:
    """Mode and launch of the case: the default launch, or the shape the
    library's autotuner picks on such a field."""
    shape = (32, False) if case["launch"] == "default" else (
        (64, case["mech"] == "KONNOV") if case["field"] == "flame" else (32, True))
    if getattr(solver, "configured", None) != (case["mode"], shape):
        solver.set_mode(case["mode"])
        solver.set_launch(kernel="thread", block=shape[0], lu_rolled=shape[1])
        solver.configured = (case["mode"], shape)


# ------------------------------------------------------------------- prepare
def prepare(case: dict, seed: int) -> dict:
    return _PREPARE[case["kind"]](case, seed)


def _new(*shape):
    return torch.zeros(shape, dtype=torch.float64, device=DEV)


def _prepare_step(case, seed):
    T, _, rho, Y = _field(case, seed)
    n, N = T.numel(), Y.shape[0]
    s = _solver(case["mech"], "surrogate" if case["mode"] == "surrogate" else "")
    return dict(case=case, solver=s, T=T, rho=rho, Y=Y, Y_prod=_new(N, n), Y_prod2=_new(N, n), E=_new(n),
                T_after=_new(n), status=torch.zeros(n, dtype=torch.uint8, device=DEV))


def _run_step(st):
    case, s = st["case"], st["solver"]
    _configure(s, case)
    s.step_device(case["dt"], st["T"], st["rho"], st["Y"], st["Y_prod"], st["Y_prod2"], st["E"],
                  T_after=st["T_after"], status=st["status"])
    return {k: st[k] for k in ("Y_prod", "Y_prod2", "E", "T_after", "status")}


def _prepare_host(case, seed):
    T, p, rho, Y = (a.cpu().numpy() for a in _field(case, seed))
    m = DataManager.block(case["nx"], case["ny"], case["nz"])
    shape = (case["nx"], case["ny"], case["nz"])

    def put(values, a):
        m.interior(a)[...] = values.reshape(shape[::-1]).transpose(2, 1, 0)

    for name, v in (("temperature", T), ("density", rho), ("pressure", p)):
        put(v, m.create_scalar_field(name))
    for k, a in enumerate(m.create_vector_field("specie_mass_fraction", Y.shape[0])):
        put(Y[k], a)
    m.fields["bc_markers"] = np.zeros(m.shape, np.int8, order="F")
    m.create_scalar_field("energy_production_chemistry")
    m.create_vector_field("specie_production_chemistry", Y.shape[0])
    m.create_vector_field("specie_production_chemistry2", Y.shape[0])
    return dict(case=case, solver=_solver(case["mech"], "surrogate"), manager=m)


def _run_host(st):
    case, s, m = st["case"], st["solver"], st["manager"]
    _configure(s, case)
    s.manager = m
    s.solve_chemical_kinetics(case["dt"])
    f = m.fields
    return dict(E=f["energy_production_chemistry"], Y_prod=f["specie_production_chemistry"],
                Y_prod2=f["specie_production_chemistry2"])


def _chem_table(mech: str, rows: int):
    """A table over a flame's temperatures: mass fractions along the front, moved by a smooth increment."""
    T, _, _, Y = _field(dict(mech=mech, field="flame", nx=rows, ny=1, nz=1), 0)
    T, order = torch.sort(T)
    return T, (Y[:, order] * (1.0 + 1e-3 * _uniform(_generator(17), (Y.shape[0], 1)))).contiguous()


def _prepare_table(case, seed):
    T, _, rho, Y = _field(case, seed)
    n, N = T.numel(), Y.shape[0]
    return dict(case=case, solver=_solver(case["mech"], f"table{case['rows']}"), T=T, rho=rho, Y=Y,
                Y_prod=_new(N, n), Y_prod2=_new(N, n), E=_new(n))


def _run_table(st):
    st["solver"].step_device(st["case"]["dt"], st["T"], st["rho"], st["Y"], st["Y_prod"], st["Y_prod2"], st["E"])
    return {k: st[k] for k in ("Y_prod", "Y_prod2", "E")}


def _state_inputs(case, seed):
    g = _generator(seed + 5)
    T, _, rho, Y = _field(case, seed)
    n, N = T.numel(), Y.shape[0]
    v = _uniform(g, (case["dims"], n), -30.0, 30.0)
    E, _ = _energy(case["mech"], T, Y)
    # sources of the size a step produces, without a net change of mass; none in cold cells
    W = torch.tensor(_tables(case["mech"])["molar_mass"], device=DEV)
    dY = 2e-3 * (_uniform(g, (N, n)) - 0.5) * Y * (T > 305.0)
    dY = dY - Y * dY.sum(0, keepdim=True)
    Y_prod = dY * rho / case["dt"]
    h0 = _enthalpy(case["mech"], torch.full((1,), T_REF, dtype=torch.float64, device=DEV))
    E_prod = -(h0 * Y_prod / W[:, None]).sum(0)
    return T, rho, Y, E + 0.5 * (v * v).sum(0), v, Y_prod.contiguous(), E_prod


def _prepare_state(case, seed):
    T, rho, Y, E, v, Y_prod, E_prod = _state_inputs(case, seed)
    n = T.numel()
    st = dict(case=case, solver=_solver(case["mech"]), T0=T, Y0=Y, E0=E, rho=rho, v=v, Y_prod=Y_prod, E_prod=E_prod,
              T=T.clone(), Y=Y.clone(), E=E.clone(), status=torch.zeros(n, dtype=torch.uint8, device=DEV))
    st.update({k: _new(n) for k in ("p", "gamma", "cp_mass", "h_s", "h_full", "v_s", "mix")})
    return st


def _run_state(st):
    # the state before the step is kept, as a solver keeps it for its corrector
    st["T"].copy_(st["T0"])
    st["Y"].copy_(st["Y0"])
    st["E"].copy_(st["E0"])
    st["solver"].apply_state_device(st["rho"], st["Y"], st["E"], st["T"], st["p"], st["gamma"], v=st["v"],
                                    time_step=st["case"]["dt"], Y_prod=st["Y_prod"], E_f_prod=st["E_prod"],
                                    cp_mass=st["cp_mass"], h_s=st["h_s"], h_full=st["h_full"], v_s=st["v_s"],
                                    mix_mol_mass=st["mix"], status=st["status"])
    return {k: st[k] for k in ("T", "Y", "E", "p", "gamma", "cp_mass", "h_s", "h_full", "v_s", "mix", "status")}


def _predictor_inputs(case, seed):
    g = _generator(seed + 3)
    n = [case["nx"], case["ny"], case["nz"]]
    dims = 3 if n[2] > 1 else 2
    e = [n[d] + 2 if d < dims else 1 for d in range(3)]
    _, _, rho, Y = _field(dict(case, field="flame", nx=e[0], ny=e[1], nz=e[2]), seed)
    ld, N = rho.numel(), Y.shape[0]
    faces = dims * (e[0] + 1) * (e[1] + 1) * (e[2] + 1 if dims == 3 else 1)
    v_f = []
    for _ in range(dims):
        v = _uniform(g, faces, -6.0, 10.0)
        v_f.append(torch.where(_uniform(g, faces) < 0.05, torch.zeros_like(v), v))
    diff = 50.0 * torch.randn((N, ld), generator=g, dtype=torch.float64, device=DEV)
    chem = 200.0 * torch.randn((N, ld), generator=g, dtype=torch.float64, device=DEV) * (Y > 1e-8)
    return dims, n[:dims], e, rho, Y, v_f, diff, chem


def _prepare_predictor(case, seed):
    dims, n, _, rho, Y, v_f, diff, chem = _predictor_inputs(case, seed)
    ld, N = rho.numel(), Y.shape[0]
    return dict(case=case, solver=_solver(case["mech"]), dims=dims, n=n, rho0=rho, Y0=Y, v_f=v_f, diff=diff,
                chem=chem, rho=rho.clone(), Y=Y.clone(), rho_old=_new(ld), Y_old=_new(N, ld), rho_int=_new(ld),
                Y_int=_new(N, ld))


def _run_predictor(st):
    # rho and Y before the step are kept, as a solver keeps them for its corrector
    st["rho"].copy_(st["rho0"])
    st["Y"].copy_(st["Y0"])
    st["solver"].species_predictor_device(st["case"]["dt"], st["dims"], st["n"], 10e-6, st["v_f"], st["rho"],
                                          st["Y"], st["rho_old"], st["Y_old"], st["rho_int"], st["Y_int"],
                                          Y_prod_diff=st["diff"], Y_prod_chem=st["chem"])
    return {k: st[k] for k in ("rho", "Y", "rho_old", "Y_old", "rho_int", "Y_int")}


def _prepare_diffusivity(case, seed):
    T, p, _, Y = _field(case, seed)
    W = torch.tensor(_tables(case["mech"])["molar_mass"], device=DEV)
    return dict(case=case, solver=_solver(case["mech"], "diffusivity"), T=T, p=p, Y=Y,
                mm=1.0 / (Y / W[:, None]).sum(0), D=torch.zeros_like(Y))


def _run_diffusivity(st):
    st["solver"].mixture_diffusivity_device(st["T"], st["p"], st["Y"], st["mm"], st["D"])
    return st["D"]


def _prepare_train(case, seed):
    """Standardised features and targets of a smooth map with the pairs' heavy-tailed outputs."""
    g = _generator(seed)
    n = case["n"]
    x = torch.randn((n, 16), generator=g, device=DEV)
    x[:, 12:] = 0.0
    x = x.to(torch.bfloat16)
    A = torch.randn((12, 10), generator=g, device=DEV) / math.sqrt(12.0)
    z = x[:, :12].float() @ A
    y = (torch.tanh(z) + 0.3 * z * z * torch.sign(z)).contiguous()
    return dict(case=case, net=nrg_surrogate.Surrogate(_solver(case["mech"], "train")), x=x, y=y)


def _run_train(st):
    net, case = st["net"], st["case"]
    net.init(seed=1)
    losses = net.train(st["x"], st["y"], epochs=1, batch=case["batch"], lr=1e-3, seed=2)
    return dict(params=net.params(), losses=losses)


_PREPARE = dict(step=_prepare_step, host=_prepare_host, table=_prepare_table, state=_prepare_state,
                predictor=_prepare_predictor, diffusivity=_prepare_diffusivity, train=_prepare_train)
_RUN = dict(step=_run_step, host=_run_host, table=_run_table, state=_run_state, predictor=_run_predictor,
            diffusivity=_run_diffusivity, train=_run_train)


def run(state: dict):
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------------- work
SPECIES = dict(KEROMNES=9, ZHANG=9, TEREZA=10, KONNOV=13, ACETYLENE=17)
# algorithmic flops of one integrated cell with the KEROMNES mechanism, in
# thousands, from the library's event counts on these fields: 270 per BDF step,
# 269 per right-hand side, 1,092 per iteration matrix with its factors, 207 per
# solve, 1,080 for the set-up (a flame's cold cells take none)
CELL_KFLOP = dict(flame=65.0, random=134.0, ignition=300.0, wide=200.0)
STEP_COST = dict(KEROMNES=1.0, ZHANG=1.1, TEREZA=1.4, KONNOV=3.2, ACETYLENE=2.6)


def work(case: dict) -> dict:
    if case["kind"] == "train":
        # three products per weight and pair; parameters, moments and gradients per batch
        weights, steps = 16 * 128 + 3 * 128 * 128 + 128 * 16, case["n"] // case["batch"]
        return dict(bytes=case["n"] * (32 + 40) + steps * 7 * 4 * (weights + 528),
                    flops=6 * weights * steps * case["batch"])
    N, n = SPECIES[case["mech"]], case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind in ("step", "host"):
        cost = CELL_KFLOP[case["field"]] * STEP_COST[case["mech"]] * 1e3
        cost *= 0.1 if case["mode"] == "surrogate" else 1.25 if case["mode"] == "reference" else 1.0
        return dict(bytes=n * (8 * (3 * N + 4) + 2), flops=n * cost)
    if kind == "table":
        return dict(bytes=n * 8 * (3 * N + 2) + case["rows"] * 8 * (N + 1), flops=n * 10 * N)
    if kind == "state":
        # reads T, rho, E, v, Y, the sources; writes T, E, Y, p, gamma and five more properties, a status
        return dict(bytes=n * (8 * (3 * N + 4 + case["dims"] + 9) + 1), flops=n * (40 * N + 300))
    if kind == "predictor":
        dims = 3 if case["nz"] > 1 else 2
        # reads rho, Y, two source arrays, the face velocities; writes rho, Y three times
        return dict(bytes=n * 8 * (1 + 3 * N + dims + 3 * (1 + N)), flops=n * dims * (N + 1) * 25)
    return dict(bytes=n * 8 * (3 + 2 * N), flops=n * (N * (N - 1) // 2 * 12 + 17 * 40))


# ----------------------------------------------------------------- tolerance
def tolerance(case: dict):
    """About four times what two implementations were seen to differ by."""
    kind = case["kind"]
    if kind in ("step", "host"):
        if case["mode"] == "surrogate":
            # the networks' parameters moved by one ulp: 4.9e-5, 1.4e-2 and 2.3e-5 of the gate's decisions
            return dict(rel=2e-4, max=6e-2, differ=1e-4)
        # analytic against finite-difference Jacobian: 2.1e-10 and 2.2e-8 (both are 4e-9 from the exact solution)
        return dict(rel=8e-10, max=1e-7)
    if kind == "train":
        # two runs (split sums added by atomics): 3.4e-6 and 5.0e-5
        return dict(rel=2e-5, max=3e-4)
    if kind == "table":
        return dict(rel=5e-13, max=4e-12)  # against the other order of the interpolation: 1.0e-13 and 8.4e-13
    if kind == "predictor":
        return dict(rel=5e-16, max=4e-15)  # against torch's order of the sums: 1.2e-16 and 8.5e-16
    if kind == "state":
        return dict(rel=5e-11, max=2e-10)  # against the converged temperature: 1.2e-11 and 3.8e-11 (h_full)
    return dict(rel=1e-15, max=6e-15)  # diffusivity, against the pairs summed per species: 1.9e-16 and 1.4e-15


# --------------------------------------------------------------------- exact
def exact(case: dict, seed: int):
    fn = dict(step=_exact_step, table=_exact_table, state=_exact_state, predictor=_exact_predictor,
              diffusivity=_exact_diffusivity).get(case["kind"])
    return fn(case, seed) if fn else None


def _rates(mech: str, T, C):
    """Forward and reverse rate constants [R, n] of frozen T and third bodies, third-body sums folded in."""
    t = _tables(mech)
    N, R = t["n_species"], t["n_reactions"]
    names = ("A", "beta", "E", "A_low", "beta_low", "E_low")
    arr = {k: torch.tensor(t["arrhenius"][:, i], device=DEV)[:, None] for i, k in enumerate(names)}
    a, lnT = _nasa(mech, T), torch.log(T)
    h = _enthalpy(mech, T)
    s = (((a[4] / 4 * T + a[3] / 3) * T + a[2] / 2) * T + a[1]) * T + a[6] + a[0] * lnT
    M = torch.tensor(t["eff"], device=DEV) @ C
    kinf = arr["A"] * torch.exp(arr["beta"] * lnT - arr["E"] / (RG * T))
    k0 = arr["A_low"] * torch.exp(arr["beta_low"] * lnT - arr["E_low"] / (RG * T))
    kf, kr = kinf.clone(), torch.zeros_like(kinf)
    sides = torch.full((2, R, 3), N, dtype=torch.long)
    S = torch.zeros((N, R), dtype=torch.float64)
    for r in range(R):
        typ = int(t["reaction_type"][r])
        left = [int(x) for x in t["coeffs"][0, r, 1:1 + t["coeffs"][0, r, 0]]]
        right = [int(x) for x in t["coeffs"][1, r, 1:1 + t["coeffs"][1, r, 0]]]
        if typ in (2, 3, 7):
            pr = k0[r] * M[r] / kinf[r]
            kf[r] = kinf[r] * pr / (1.0 + pr)
            if typ == 3:
                al, T3, T1 = (float(x) for x in t["arrhenius"][r, 6:9])
                F = torch.log10((1 - al) * torch.exp(-T / T3) + al * torch.exp(-T / T1)
                                + torch.exp(-float(t["troe3"][r]) / T))
                lp = torch.log10(torch.where(pr > 0, pr, torch.ones_like(pr)))
                c, nn = -0.4 - 0.67 * F, 0.75 - 1.27 * F
                x = (lp + c) / (nn - 0.14 * (lp + c))
                kf[r] = kf[r] * 10.0 ** (F * torch.where(pr > 0, 1.0 / (1.0 + x * x), torch.full_like(x, -1 / 0.14)))
        if typ < 5:
            ds = sum(s[i - 1] for i in right if i <= N) - sum(s[i - 1] for i in left if i <= N)
            dh = sum(h[i - 1] for i in right if i <= N) - sum(h[i - 1] for i in left if i <= N)
            kr[r] = kf[r] * torch.exp(dh / (RG * T) - ds / RG - (len(right) - len(left)) * torch.log(P_ATM / (RG * T)))
        if N + 1 in left:
            kf[r] = kf[r] * M[r]
        if N + 1 in right:
            kr[r] = kr[r] * M[r]
        for side, ids, sgn in ((0, left, -1.0), (1, right, 1.0)):
            for p, i in enumerate(i for i in ids if i <= N):
                sides[side, r, p] = i - 1
                S[i - 1, r] += sgn
    return kf, kr, sides.to(DEV), S.to(DEV)


def _rhs(kf, kr, sides, S, C, jac: bool = False):
    """dC/dt [N, n] of mass-action kinetics, or its Jacobian [n, N, N]; `sides` indexes C with a row of ones added."""
    Cp = torch.cat([C, torch.ones_like(C[:1])])
    if not jac:
        return S @ (kf * Cp[sides[0]].prod(1) - kr * Cp[sides[1]].prod(1))
    J = 0.0
    for k, side in ((kf, sides[0]), (-kr, sides[1])):
        x = Cp[side]
        for p in range(3):
            others = k * x[:, (p + 1) % 3] * x[:, (p + 2) % 3]
            hot = torch.nn.functional.one_hot(side[:, p], C.shape[0] + 1)[:, :-1].to(C.dtype)
            J = J + torch.einsum("kr,rn,rl->nkl", S, others, hot)
    return J


def _exact_step(case, seed):
    """Radau IIA (three stages) on steps that grow from 1e-7 of the interval; frozen T and third bodies."""
    n = case["nx"] * case["ny"] * case["nz"]
    if case["mode"] == "surrogate" or n * case["dt"] > 0.025 or case["mech"] in ("KONNOV", "ACETYLENE"):
        return None
    T, _, rho, Y = _field(case, seed)
    W = torch.tensor(_tables(case["mech"])["molar_mass"], device=DEV)[:, None]
    N, dt = Y.shape[0], case["dt"]
    live = T >= 305.0
    C0 = (Y * rho / W)[:, live]
    kf, kr, sides, S = _rates(case["mech"], T[live], C0)
    r6 = math.sqrt(6.0)
    A = torch.tensor([[(88 - 7 * r6) / 360, (296 - 169 * r6) / 1800, (-2 + 3 * r6) / 225],
                      [(296 + 169 * r6) / 1800, (88 + 7 * r6) / 360, (-2 - 3 * r6) / 225],
                      [(16 - r6) / 36, (16 + r6) / 36, 1 / 9]], dtype=torch.float64, device=DEV)
    edges = np.concatenate([[0.0], np.geomspace(dt * 1e-7, dt * 0.02, 70), np.linspace(dt * 0.02, dt, int(60 * max(1.0, dt / 1e-6)))[1:]])
    eye = torch.eye(3 * N, dtype=torch.float64, device=DEV)
    C = C0
    for h in np.diff(edges):
        J = _rhs(kf, kr, sides, S, C, True)
        lu = torch.linalg.lu_factor(eye - h * torch.einsum("ij,nkl->nikjl", A, J).reshape(-1, 3 * N, 3 * N))
        Z = torch.zeros((3, N, C.shape[1]), dtype=torch.float64, device=DEV)
        for _ in range(9):
            F = torch.stack([_rhs(kf, kr, sides, S, C + Z[i]) for i in range(3)])
            res = h * torch.einsum("ij,jkn->ikn", A, F) - Z
            d = torch.linalg.lu_solve(*lu, res.reshape(3 * N, -1).T.unsqueeze(-1)).squeeze(-1).T
            Z = Z + d.reshape(3, N, -1)
            if float(d.abs().max()) < 1e-17 * float(C.abs().max()):
                break
        C = C + Z[2]
    dC = torch.zeros_like(Y)
    dC[:, live] = C - C0
    h0 = _enthalpy(case["mech"], torch.full((1,), T_REF, dtype=torch.float64, device=DEV))
    E = -(h0 * dC).sum(0) / dt
    Y1 = Y + dC * W / rho
    e0, _ = _energy(case["mech"], T, Y)
    T1 = torch.where(live, _solve_T(case["mech"], T, Y1, e0 + E * dt / rho), T)
    return dict(Y_prod=dC * W / dt, Y_prod2=dC, E=E, T_after=T1, status=live.to(torch.uint8))


def _solve_T(mech, T, Y, E):
    for _ in range(60):
        e, avg = _energy(mech, T, Y)
        W = torch.tensor(_tables(mech)["molar_mass"], device=DEV)[:, None]
        T = T + (E - e) * avg / ((_cp(mech, T) * Y / W).sum(0) * avg)
    return T


def _exact_table(case, seed):
    T, _, rho, Y = _field(case, seed)
    T_t, Y_t = _chem_table(case["mech"], case["rows"])
    W = torch.tensor(_tables(case["mech"])["molar_mass"], device=DEV)[:, None]
    iv = (torch.searchsorted(T_t, T, right=True) - 1).clamp(0, T_t.numel() - 2)
    w = ((T - T_t[iv]) / (T_t[iv + 1] - T_t[iv])).clamp(0.0, 1.0)
    q = Y_t[:, iv + 1] * w + Y_t[:, iv] * (1.0 - w)
    q = torch.where(T < T_t[0], torch.zeros_like(q), q)
    live = T >= 305.0
    h0 = _enthalpy(case["mech"], torch.full((1,), T_REF, dtype=torch.float64, device=DEV))
    zero = torch.zeros_like(q)
    return dict(Y_prod=torch.where(live, q * W / case["dt"], zero), Y_prod2=torch.where(live, q - Y, zero),
                E=torch.where(live, -(h0 * q).sum(0) / case["dt"], zero[0]))


def _exact_state(case, seed):
    T, rho, Y, E, v, Y_prod, E_prod = _state_inputs(case, seed)
    mech, dt = case["mech"], case["dt"]
    Y = Y + Y_prod * dt / rho
    E = E + E_prod * dt / rho
    T = _solve_T(mech, T, Y, E - 0.5 * (v * v).sum(0))
    W = torch.tensor(_tables(mech)["molar_mass"], device=DEV)[:, None]
    avg = 1.0 / (Y / W).sum(0)
    X = Y / W * avg
    h, cp = (_enthalpy(mech, T) * X).sum(0), (_cp(mech, T) * X).sum(0)
    h0 = (_enthalpy(mech, torch.full_like(T[:1], T_REF)) * X).sum(0)
    p, gamma = T * rho * RG / avg, cp / (cp - RG)
    return dict(T=T, Y=Y, E=E, p=p, gamma=gamma, cp_mass=cp / avg, h_s=(h - h0) / avg, h_full=h / avg,
                v_s=torch.sqrt(gamma * p / rho), mix=avg, status=torch.ones_like(T, dtype=torch.uint8))


def _exact_predictor(case, seed):
    """CHARM-limited convection of rho Y_k, the most abundant species closing the sum, over the whole block."""
    dims, n, e, rho, Y, v_f, diff, chem = _predictor_inputs(case, seed)
    W = torch.tensor(_tables(case["mech"])["molar_mass"], device=DEV)
    N, dt, dx = Y.shape[0], case["dt"], 10e-6
    shape = e[::-1]
    q = torch.cat([rho * Y, (rho * Y / W[:, None]).sum(0, keepdim=True)]).reshape(N + 1, *shape)
    top = (rho * Y).argmax(0).reshape(shape)
    inner = [slice(1, -1) if 2 - a < dims else slice(None) for a in range(3)]
    rhs = torch.zeros((N, *[n[d] if d < dims else 1 for d in (2, 1, 0)]), dtype=torch.float64, device=DEV)
    for d in range(dims):
        ax = 2 - d
        fs = [x + 1 if 2 - a < dims else 1 for a, x in enumerate(shape)]
        vel = v_f[d].reshape(*fs, dims)[..., d]
        sel = list(inner)
        sel[ax] = slice(1, n[d] + 2)
        vel = vel[tuple(slice(s.start, 1 + n[2 - a]) if (2 - a < dims and a != ax) else s for a, s in enumerate(sel))]

        def at(a, lo, hi):
            s = list(inner)
            s[ax] = slice(lo, hi)
            return a[(Ellipsis, *s)]

        m = n[d]  # faces 0..m; face f lies between cells f and f + 1 of the ghosted axis
        pos = vel > 0
        up = torch.where(pos, at(q, 0, m + 1), at(q, 1, m + 2))
        F = up[:N] * vel
        if m > 1:
            a0, a1, a2, a3 = at(q, 0, m - 1), at(q, 1, m), at(q, 2, m + 1), at(q, 3, m + 2)
            fsel = [slice(None)] * 3
            fsel[ax] = slice(1, m)
            vi, pi = vel[tuple(fsel)], pos[tuple(fsel)]
            loc, ups = a2 - a1, torch.where(pi, a1 - a0, a3 - a2)
            r = torch.where(loc != 0, ups / torch.where(loc != 0, loc, torch.ones_like(loc)), torch.zeros_like(loc))
            s = 1.0 / torch.where(r > 1e-10, r, torch.ones_like(r))
            B = torch.where(r > 1e-10, s * (3 * s + 1) / (s + 1) / (s + 1), torch.zeros_like(s))
            val = torch.where(pi, a1 + B * 0.5 * ups, a2 - B * 0.5 * ups)
            g = torch.where(pi, at(top, 1, m), at(top, 2, m + 1))
            phi = val[:N]
            lead = torch.arange(N, device=DEV).reshape(N, 1, 1, 1) == g
            rest = torch.where(lead, torch.zeros_like(phi), phi / W.reshape(N, 1, 1, 1)).sum(0)
            phi = torch.where(lead, W.reshape(N, 1, 1, 1) * (val[N] - rest), phi)
            F[(slice(None), *fsel)] = phi * vi
        lo, hi = [slice(None)] * 4, [slice(None)] * 4
        lo[ax + 1], hi[ax + 1] = slice(0, m), slice(1, m + 1)
        rhs = rhs - (F[tuple(hi)] - F[tuple(lo)]) / dx
    cells = (slice(None), *inner)
    new = (q[:N][cells] + dt * (rhs + diff.reshape(N, *shape)[cells] + chem.reshape(N, *shape)[cells])).clamp(min=0.0)
    total = new.sum(0)
    out = dict(rho=rho.clone(), Y=Y.clone(), rho_old=torch.zeros_like(rho), Y_old=torch.zeros_like(Y),
               rho_int=torch.zeros_like(rho), Y_int=torch.zeros_like(Y))
    for k, v in (("rho", total), ("rho_int", total), ("rho_old", rho.reshape(shape)[tuple(inner)])):
        out[k].reshape(shape)[tuple(inner)] = v
    for k, v in (("Y", new / total), ("Y_int", new / total), ("Y_old", Y.reshape(N, *shape)[cells])):
        out[k].reshape(N, *shape)[cells] = v
    return out


def _exact_diffusivity(case, seed):
    """Chapman-Enskog binary coefficients with the Neufeld (1,1) collision integral, mixture-averaged."""
    mech = case["mech"]
    if mech == "ACETYLENE":
        return None
    T, p, _, Y = _field(case, seed)
    W = _tables(mech)["molar_mass"]
    mm = 1.0 / (Y / torch.tensor(W, device=DEV)[:, None]).sum(0)
    t = transport_tables(*nrg_b200.mechanism_paths(mech), nrg_b200.transport_path(mech))
    eps, bdc, N = t["well_depth"], t["binary_diffusivity_constant"], len(W)
    acc = torch.zeros_like(Y)
    for i in range(N):
        for j in range(N):
            if i == j or bdc[i, j] <= 0.0 or eps[i] <= 0.0 or eps[j] <= 0.0:
                continue
            x = T / math.sqrt(eps[i] * eps[j])
            om = 1.06036 / x ** 0.15610
            om = om + torch.where(x < 70.0, 0.19300 * torch.exp(-0.47635 * x) + 1.03587 * torch.exp(-1.52996 * x)
                                  + 1.76474 * torch.exp(-3.89411 * x), torch.zeros_like(x))
            D = bdc[i, j] * T ** 1.5 / (p * om)
            acc[i] += ((1.0 - Y[i]) * W[i] / W[j] + Y[i]) * Y[j] / D
    out = torch.zeros_like(Y)
    for i in range(N):
        out[i] = torch.where(acc[i] > 1e-10, (1.0 - Y[i]) * W[i] / (acc[i] * mm), out[i])
    return out
