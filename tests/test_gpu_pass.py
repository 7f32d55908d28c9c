"""The pass-structured integrator (csrc/chem_pass.cuh) at the sizes where its
launches change: partly filled warps and blocks, the largest field of blocks
whose warps run on their own and the smallest of blocks in lockstep, and the
work queue.  A cell's arithmetic depends on no other
cell, so every launch gives the same bits; the values are checked against the
oracle at the parity tolerance (|dY| <= 1e-9, |dT|/T <= 1e-6)."""
import numpy as np
import pytest

from nrg_b200 import eact_units, fields, mechanism_paths
from tests.gpu_util import run_device

pytestmark = pytest.mark.gpu

KEYS = ("Y_prod", "Y_prod2", "E_f_prod", "T_after", "status")


def _cells(name, W, names, n):
    if name == "ACETYLENE":
        f = fields.acetylene_state(names, W, n, seed=5, dt=1e-6)
    else:
        f = fields.slice_field(fields.ignition_field(fields_W(), n_side=256), n, stride=7)
        f = fields.state_for_species(f, names, W)
        f.dt = 2e-6 if names and W.shape[0] == 9 else 1e-6
    f.T[::11] = 301.0  # skipped
    return f


def fields_W():
    from nrg_b200 import keromnes_paths
    from nrg_b200.chemistry import mechanism_tables
    return mechanism_tables(*keromnes_paths())["molar_mass"]


# first: the largest fields whose warps run on their own, or one cell more; with
# `more` cells on top blocks in lockstep and a ragged end (KONNOV, TEREZA: with the
# rate constants in tensor memory)
@pytest.mark.parametrize("name,mode,first,more", [("KEROMNES", "fast", 37888, 1), ("KEROMNES", "mixed", 37888, 0),
                                                  ("ZHANG", "fast", 37888, 129), ("TEREZA", "fast", 148 * 160, 33),
                                                  ("KONNOV", "fast", 148 * 64, 97), ("ACETYLENE", "fast", 148 * 64, 1)])
def test_launches_agree_and_match_the_oracle(name, mode, first, more):
    from nrg_b200.chemistry import ChemicalKineticsSolver, mechanism_tables
    from oracle import oracle_py as op
    paths = mechanism_paths(name)
    W = mechanism_tables(*paths, 1.0, eact_units(name))["molar_mass"]
    s = ChemicalKineticsSolver(None, *paths, E_act_units=eact_units(name), mode=mode)
    try:
        f = _cells(name, W, s.species_names, first + more)
        s.set_cell_order(False)
        whole, _ = run_device(s, f, mode, launch=dict(kernel="thread", block=64, grid=0, chunk=1))
        for part in (1, 31, 33, 64, 65, 129, first - 1):
            g, _ = run_device(s, fields.slice_field(f, part), mode)
            for k in KEYS:
                np.testing.assert_array_equal(g[k], whole[k][..., :part], err_msg=f"{k} {part}")
        s.set_specialised(False)  # the table walk, in blocks of its own at any size
        for part in (129, f.n):
            g, _ = run_device(s, fields.slice_field(f, part), mode)
            for k in KEYS:
                np.testing.assert_array_equal(g[k], whole[k][..., :part], err_msg=f"{k} tables {part}")
        s.set_specialised(True)
        if name == "KEROMNES":
            # grid 1: each warp sets up some sixteen groups in the shared memory of the one before
            for grid, chunk in ((7, 3), (1, 1)):
                g, _ = run_device(s, fields.slice_field(f, 1000), mode,
                                  launch=dict(kernel="thread_queue", block=64, grid=grid, chunk=chunk))
                for k in KEYS:
                    np.testing.assert_array_equal(g[k], whole[k][..., :1000], err_msg=f"{k} queue {grid}")
    finally:
        s.close()
    m = 1024
    h = fields.slice_field(f, m)
    om = op.Mechanism(*paths, 1.0, eact_units(name))
    o = om.chem_step(h.dt, h.T, h.rho, h.Y)
    T1 = om.temperature_after(h.dt, h.T, h.rho, h.Y, o["Y_prod"], o["E_f_prod"])
    assert np.max(np.abs(whole["Y_prod"][:, :m] - o["Y_prod"]) * h.dt / h.rho) <= 1e-9
    assert np.max(np.abs(whole["T_after"][:m] - T1) / h.T) <= 1e-6
    np.testing.assert_array_equal(whole["status"][:m] != 0, h.T >= 305.0)


def test_autotuner_keeps_what_has_no_effect(decks):
    """In the fast mode the block and the LU form of the thread kernels select
    nothing: the autotuner leaves them as they were set, for the reference mode
    after it, and tries both there."""
    import torch
    from nrg_b200.chemistry import ChemicalKineticsSolver
    f = fields.random_field(fields_W())
    T, rho, Y = (torch.tensor(a, device="cuda") for a in (f.T, f.rho, f.Y))
    s = ChemicalKineticsSolver(None, *decks, mode="fast")
    try:
        for block, rolled in ((32, True), (64, False), (64, True), (32, False)):
            s.set_launch(kernel="thread", block=block, lu_rolled=rolled)
            assert s.autotune(f.dt, T, rho, Y, torch.zeros_like(Y), torch.zeros_like(Y), torch.zeros_like(T)) > 0.0
            d = s.get_launch()
            assert d["kernel"] in ("thread", "thread_queue") and d["block"] == block and d["lu_rolled"] is rolled, d
    finally:
        s.close()


@pytest.mark.parametrize("mode,kernel,block", [("fast", "thread_queue", 64), ("reference", "thread_queue", 32),
                                               ("fast", "warp_queue", 256)])
def test_a_queue_of_more_blocks_than_cells(decks, mode, kernel, block):
    """The largest grid that nrg_chem_set_launch takes: blocks without a cell are
    not launched (their reservations would carry the queue head past the end
    of an int), the cells' bits stay."""
    from nrg_b200.chemistry import ChemicalKineticsSolver
    f = fields.slice_field(fields.random_field(fields_W()), 200)
    s = ChemicalKineticsSolver(None, *decks, mode=mode)
    try:
        a, b = (run_device(s, f, mode, launch=dict(kernel=kernel, block=block, grid=grid, chunk=64))[0]
                for grid in (3, 2**31 - 1))
    finally:
        s.close()
    for k in KEYS:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("mode", ["fast", "mixed"])
def test_norms_beyond_the_range_of_their_squares(decks, mode):
    """Densities at which the first weighted norm of dy/dt is above 1e154, so that
    its square overflows: the step size comes from the scaled norm, and the
    cells end as the oracle's do, at the limit of steps with a finite state."""
    from nrg_b200.chemistry import ChemicalKineticsSolver
    from oracle import oracle_py as op
    f = fields.slice_field(fields.random_field(fields_W()), 64)
    f.rho = f.rho * 1e85
    o = op.Mechanism(*decks, 1.0, "cal.mol").chem_step(f.dt, f.T, f.rho, f.Y)
    assert np.all(np.isfinite(o["Y_prod"]))
    s = ChemicalKineticsSolver(None, *decks, mode=mode)
    try:
        g, st = run_device(s, f, mode)
    finally:
        s.close()
    assert np.all(g["status"] == 2) and np.all(np.isfinite(g["Y_prod"]))
    assert st["steps"] == 10000 * f.n
