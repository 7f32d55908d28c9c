"""Which decks use the generated code, and the reference mode's against its
table walk."""
import numpy as np
import pytest

from nrg_b200 import fields
from tests.gpu_util import dY, run_device

pytestmark = pytest.mark.gpu

KEYS = ("Y_prod", "Y_prod2", "E_f_prod", "T_after", "status")


def test_a_deck_that_lists_an_inert_species_elsewhere(decks, oracle_mech, W, tmp_path):
    """KEROMNES with N2 last: the reacting species and the reactions over them
    are the generated code's, so the fast and mixed modes use it (the bits of
    the table walk); the reference mode, which integrates N2 too, walks its
    tables.  The results are the oracle's on the deck as it stands."""
    from nrg_b200.chemistry import ChemicalKineticsSolver
    with open(decks[0], encoding="latin-1") as fh:
        text = fh.read()
    line = "H2    O2      N2      O       H       OH      H2O     HO2     H2O2\n"
    assert text.count(line) == 1
    moved = tmp_path / "n2_last.txt"
    moved.write_text(text.replace(line, "H2    O2      O       H       OH      H2O     HO2     H2O2    N2\n"),
                     encoding="latin-1")
    f = fields.slice_field(fields.random_field(W), 512)
    o = oracle_mech.chem_step(f.dt, f.T, f.rho, f.Y)
    perm = [0, 1, 3, 4, 5, 6, 7, 8, 2]
    g = fields.slice_field(f, f.n)
    g.Y = np.ascontiguousarray(f.Y[perm])
    s = ChemicalKineticsSolver(None, str(moved), *decks[1:], mode="fast")
    try:
        assert s.species_names == [fields.SPECIES[k] for k in perm]
        for mode in ("fast", "mixed", "reference"):
            outs = []
            for spec in (True, False):
                s.set_specialised(spec)
                outs.append(run_device(s, g, mode, launch=dict(kernel="thread", block=32, grid=0, chunk=1))[0])
            for key in KEYS:
                np.testing.assert_array_equal(outs[0][key], outs[1][key], err_msg=f"{mode} {key}")
            assert np.abs(dY(outs[0], g) - dY(o, f)[perm]).max() <= 1e-9
    finally:
        s.close()


@pytest.mark.parametrize("name", ["KEROMNES", "ZHANG", "TEREZA", "KONNOV", "ACETYLENE"])
def test_reference_mode_generated_code_gives_the_table_walk_bits(name):
    """The reference mode's generated right-hand side over all species against
    its own table walk: every output and event count."""
    from nrg_b200 import eact_units, mechanism_paths
    from nrg_b200.chemistry import ChemicalKineticsSolver, mechanism_tables
    paths, units = mechanism_paths(name), eact_units(name)
    Wn = mechanism_tables(*paths, 1.0, units)["molar_mass"]
    s = ChemicalKineticsSolver(None, *paths, E_act_units=units, mode="reference")
    try:
        if name == "ACETYLENE":
            f = fields.acetylene_state(s.species_names, Wn, 300, seed=6)
        else:
            base = fields.ignition_field(mechanism_tables(*mechanism_paths("KEROMNES"))["molar_mass"], n_side=128)
            f = fields.state_for_species(fields.slice_field(base, 300, stride=7), s.species_names, Wn)
            f.dt = 2e-6
        outs = []
        for spec in (True, False):
            s.set_specialised(spec)
            outs.append(run_device(s, f, "reference", launch=dict(kernel="thread", block=32, grid=0, chunk=1)))
    finally:
        s.close()
    (a, sa), (b, sb) = outs
    assert sa["cells_bad"] == 0
    for key in KEYS:
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)
    for key in ("steps", "rhs_evals", "jacobians", "solves"):
        assert sa[key] == sb[key], key
