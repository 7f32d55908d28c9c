"""The training contraction (k_gemm_tc) at the edges of its tiles: batches of
one row, of a 16-row slice, one below and above a 128-row tile, and one whose
weight gradients take more than one 128-row chunk per block, against the
float64 backward pass with the same BF16 rounding points.  Tolerance: five
layers of BF16 roundings of activations and gradients (2^-9 each, not averaged
for a single row), 3e-2 of a tensor's norm."""
import ctypes

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


@pytest.mark.parametrize("off", [1, 2, 4])
def test_arrays_off_a_16_byte_boundary(sur, off):
    """Features and results that start inside a caller's larger array (2, 4 and
    8 bytes past a boundary; the results 4, 8 and 16) give the values of
    aligned copies: the forward pass bit for bit, gradients and parameters up
    to the order of the sums over split rows (1e-5 of their norm)."""
    import torch
    from nrg_b200.chemistry import _check, _ptr, lib
    n = 200
    xt, yt, _, _ = rand_batch(n, 40)
    big = torch.zeros(n * 16 + 8, dtype=torch.bfloat16, device="cuda")
    xo = big[off:off + n * 16].view(n, 16)
    xo.copy_(xt)
    ref = sur.forward(xt)
    assert torch.equal(sur.forward(xo), ref)
    out = torch.full((n * 16 + 8,), 7.0, device="cuda")
    torch.cuda.synchronize()
    _check(lib().nrg_surrogate_forward(sur.h, n, _ptr(xo), ctypes.c_void_p(out.data_ptr() + 4 * off)), sur.h)
    assert torch.equal(out[off:off + n * 16].view(n, 16), ref)
    assert torch.all(out[:off] == 7.0) and torch.all(out[off + n * 16:] == 7.0)
    (ga, la), (gb, lb) = sur.grad(xt, yt), sur.grad(xo, yt)
    assert la == pytest.approx(lb, rel=1e-12)
    assert np.linalg.norm(ga - gb) <= 1e-5 * np.linalg.norm(ga)
    res = []
    for x in (xt, xo):
        sur.init(seed=7)
        sur.train(x, yt, epochs=2, batch=64, lr=1e-3, seed=2)
        res.append(sur.params())
    sur.init(seed=7)
    assert np.linalg.norm(res[0] - res[1]) <= 1e-5 * np.linalg.norm(res[0])


def test_sums_repeat_bit_for_bit(sur):
    """Batches of up to two 128-row tiles train to the same parameters and
    losses every time (two tiles' weight gradients add to zero in either order
    alike); bias gradients and the loss repeat at any batch (155 tiles here, 256
    blocks of the loss)."""
    for batch in (64, 128, 192, 256):
        xt, yt, _, _ = rand_batch(4 * batch + 3, 50 + batch)
        runs = []
        for _ in range(4):
            sur.init(seed=7)
            losses = sur.train(xt, yt, epochs=3, batch=batch, lr=1e-3, seed=2)
            runs.append((sur.params(), losses))
        for p, losses in runs[1:]:
            np.testing.assert_array_equal(p, runs[0][0], err_msg=str(batch))
            np.testing.assert_array_equal(losses, runs[0][1], err_msg=str(batch))
    sur.init(seed=7)
    xt, yt, _, _ = rand_batch(154 * 128 + 9, 60)
    runs = [sur.grad(xt, yt) for _ in range(4)]
    off = 0
    for o, i in mlp_ref.SHAPES:
        for g, loss in runs[1:]:
            np.testing.assert_array_equal(g[off + o * i:off + o * i + o], runs[0][0][off + o * i:off + o * i + o])
            assert loss == runs[0][1]
        off += o * i + o
