"""nrg_mixture_diffusivity_device (calculate_diffusivity_coeff,
fickean_diffusion_solver.f90:358-395) against the oracle on the wide-range
state distribution (T ~ U[800, 2600] K, p ~ U[0.5, 5] atm) for the four
reference mechanisms.  Tolerance: 1e-12 relative per coefficient (the device
divides once per species where the reference divides per pair, and its pow and
exp may differ from the host's in the last bit)."""
import numpy as np
import pytest

from nrg_b200 import MECHANISMS, fields, mechanism_paths, transport_path

pytestmark = pytest.mark.gpu

RTOL = 1e-12


@pytest.mark.parametrize("name", MECHANISMS)
def test_diffusivity_matches_oracle(name):
    import torch
    from nrg_b200.chemistry import ChemicalKineticsSolver, mechanism_tables
    from oracle import oracle_py as op
    paths = mechanism_paths(name)
    W = mechanism_tables(*paths)["molar_mass"]
    s = ChemicalKineticsSolver(None, *paths, mode="fast")
    try:
        s.load_transport(transport_path(name))
        W9 = mechanism_tables(*mechanism_paths("KEROMNES"))["molar_mass"]
        base = fields.slice_field(fields.wide_range_field(W9, n_side=128), 8192, stride=2)
        f = fields.state_for_species(base, s.species_names, W)
        mm = 1.0 / np.sum(f.Y / W[:, None], axis=0)
        bc = (np.arange(f.n) % 97 == 5).astype(np.int8)
        om = op.Mechanism(*paths, 1.0, "cal.mol")
        om.load_transport(transport_path(name))
        Do = om.mixture_diffusivity(f.T, f.p, f.Y, mm, bc=bc)
        d = torch.device("cuda")
        t = lambda a: torch.tensor(np.ascontiguousarray(a), device=d)
        D = torch.full(f.Y.shape, -1.0, dtype=torch.float64, device=d)
        s.mixture_diffusivity_device(t(f.T), t(f.p), t(f.Y), t(mm), D, bc=t(bc))
        Dg = D.cpu().numpy()
    finally:
        s.close()
    assert np.all((Dg == 0) == (Do == 0))
    assert np.all(Dg[:, bc != 0] == 0)
    nz = Do != 0
    assert np.max(np.abs(Dg[nz] / Do[nz] - 1.0)) <= RTOL


def test_diffusivity_outside_the_normal_range():
    """Infinite, vanishing, negative and denormal temperatures, pressures, mass
    fractions and mixture molar masses: zero where the reference's terms vanish
    or overflow, its value elsewhere."""
    import torch
    from nrg_b200.chemistry import ChemicalKineticsSolver, mechanism_tables
    from oracle import oracle_py as op
    paths = mechanism_paths("KEROMNES")
    W = mechanism_tables(*paths)["molar_mass"]
    f = fields.slice_field(fields.wide_range_field(W, n_side=64), 40)
    T, p, Y = f.T.copy(), f.p.copy(), f.Y.copy()
    mm = 1.0 / np.sum(Y / W[:, None], axis=0)
    inf, nan = np.inf, np.nan
    p[:8] = inf, 0.0, -1.0, nan, 1e300, 1e-300, 1e-310, 1e308
    T[8:17] = inf, 0.0, nan, 1e300, 1e-100, 1e-310, 5e4, 1e200, 1e-250
    for c, v in enumerate((inf, -inf, nan, 1e300, -0.1)):
        Y[0, 17 + c] = v
    Y[:, 22] = 0.0
    Y[:, 23] = np.arange(9) == 2
    Y[:, 24] *= 1e-300
    Y[:, 25] *= 1e-320
    mm[26:31] = inf, 0.0, 1e-300, 1e300, -1.0
    p[31], T[31], p[32], T[32] = inf, inf, 1e-300, 1e300
    om = op.Mechanism(*paths, 1.0, "cal.mol")
    om.load_transport(transport_path("KEROMNES"))
    with np.errstate(all="ignore"):
        Do = om.mixture_diffusivity(T, p, Y, mm)
    t = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")
    D = torch.full(Y.shape, -1.0, dtype=torch.float64, device="cuda")
    s = ChemicalKineticsSolver(None, *paths, mode="fast")
    try:
        s.load_transport(transport_path("KEROMNES"))
        s.mixture_diffusivity_device(t(T), t(p), t(Y), t(mm), D)
    finally:
        s.close()
    np.testing.assert_allclose(D.cpu().numpy(), Do, rtol=RTOL, atol=0.0)
