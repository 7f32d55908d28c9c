"""The training contraction (k_gemm_tc) at the edges of its tiles: batches of
one row, of a 16-row slice, one below and above a 128-row tile, and one whose
weight gradients take more than one 128-row chunk per block, against the
float64 backward pass with the same BF16 rounding points.  Tolerance: five
layers of BF16 roundings of activations and gradients (2^-9 each, not averaged
for a single row), 3e-2 of a tensor's norm."""
import numpy as np
import pytest

from oracle import mlp_ref
from tests.test_gpu_surrogate import rand_batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sur(decks):
    from nrg_b200.chemistry import ChemicalKineticsSolver
    from nrg_b200.surrogate import Surrogate
    s = ChemicalKineticsSolver(None, *decks, mode="fast")
    n = Surrogate(s)
    n.init(seed=7)
    yield n
    s.close()


@pytest.mark.parametrize("B", [1, 16, 127, 129, 148 * 128 + 40])
def test_gradients_at_tile_edges(sur, B):
    xt, yt, x, y = rand_batch(B, 100 + B)
    g, loss = sur.grad(xt, yt)
    loss_ref, g_ref = mlp_ref.loss_and_grad(sur.params(), x, y)
    assert loss == pytest.approx(loss_ref, rel=2e-2)
    off = 0
    for o, i in mlp_ref.SHAPES:
        for n in (o * i, o):
            a, b = g[off:off + n], g_ref[off:off + n]
            off += n
            assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b) + 1e-12, (o, i, n)
