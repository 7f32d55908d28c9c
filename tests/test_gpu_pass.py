"""The pass-structured integrator (csrc/chem_pass.cuh) at the sizes where its
launches change: partly filled warps and blocks, the largest field of blocks
whose warps run on their own and the smallest of blocks in lockstep
(37,888 cells), and the work queue.  A cell's arithmetic depends on no other
cell, so every launch gives the same bits; the values are checked against the
oracle at the parity tolerance (|dY| <= 1e-9, |dT|/T <= 1e-6)."""
import numpy as np
import pytest

from nrg_b200 import eact_units, fields, mechanism_paths
from tests.gpu_util import run_device

pytestmark = pytest.mark.gpu

KEYS = ("Y_prod", "Y_prod2", "E_f_prod", "T_after", "status")


def _cells(W, names, n):
    base = fields.ignition_field(fields_W(), n_side=256)
    f = fields.slice_field(base, n, stride=7)
    f = fields.state_for_species(f, names, W)
    f.T[::11] = 301.0  # skipped
    f.dt = 2e-6
    return f


def fields_W():
    from nrg_b200 import keromnes_paths
    from nrg_b200.chemistry import mechanism_tables
    return mechanism_tables(*keromnes_paths())["molar_mass"]


@pytest.mark.parametrize("name,mode,n", [("KEROMNES", "fast", 37889), ("KEROMNES", "mixed", 37888),
                                         ("ZHANG", "fast", 37888 + 129)])
def test_launches_agree_and_match_the_oracle(name, mode, n):
    from nrg_b200.chemistry import ChemicalKineticsSolver, mechanism_tables
    from oracle import oracle_py as op
    paths = mechanism_paths(name)
    W = mechanism_tables(*paths)["molar_mass"]
    s = ChemicalKineticsSolver(None, *paths, E_act_units=eact_units(name), mode=mode)
    try:
        f = _cells(W, s.species_names, n)
        s.set_cell_order(False)
        whole, _ = run_device(s, f, mode, launch=dict(kernel="thread", block=64, grid=0, chunk=1))
        for part in (1, 31, 33, 64, 65, 129, 37887):
            g, _ = run_device(s, fields.slice_field(f, part), mode)
            for k in KEYS:
                np.testing.assert_array_equal(g[k], whole[k][..., :part], err_msg=f"{k} {part}")
        if name == "KEROMNES":
            g, _ = run_device(s, fields.slice_field(f, 1000), mode,
                              launch=dict(kernel="thread_queue", block=64, grid=7, chunk=3))
            for k in KEYS:
                np.testing.assert_array_equal(g[k], whole[k][..., :1000], err_msg=f"{k} queue")
    finally:
        s.close()
    m = 2048
    h = fields.slice_field(f, m)
    om = op.Mechanism(*paths, 1.0, eact_units(name))
    o = om.chem_step(h.dt, h.T, h.rho, h.Y)
    T1 = om.temperature_after(h.dt, h.T, h.rho, h.Y, o["Y_prod"], o["E_f_prod"])
    assert np.max(np.abs(whole["Y_prod"][:, :m] - o["Y_prod"]) * h.dt / h.rho) <= 1e-9
    assert np.max(np.abs(whole["T_after"][:m] - T1) / h.T) <= 1e-6
    np.testing.assert_array_equal(whole["status"][:m] != 0, h.T >= 305.0)
