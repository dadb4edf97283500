"""Row counts at the edges of the tensor-core training pass: one row, a ragged
tile, one row beyond a tile, one tile more than the CTAs of a full grid (a CTA
with two tiles), gradients against the FP64 oracle; and a training step, whose
gradient reduction also applies AdamW, against the separate gradient and AdamW
calls (the same arithmetic: equal bit for bit)."""
import numpy as np
import pytest

from firecore_b200 import learned as L
from firecore_b200.world import World
from oracle import mlp_oracle as M
from test_gpu_mlp import relerr, setup_net

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    return World(0)


@pytest.mark.parametrize("n", [1, 127, 129, 149 * 128, 2 * 148 * 128 + 5])
def test_gradients_at_tile_edges(world, n):
    p, F, mean, std, T, Xo = setup_net(n, max(n, 2))
    F, T, Xo = F[:n], T[:n], Xo[:n]
    prop = L.Proposal()
    prop.set_params(p, mean, std, 0.5)
    loss, g = prop.grad(F, T)
    lo, go = M.loss_and_grads(Xo, (T / np.float32(0.5)).astype(np.float32).astype(np.float64), p, bf=True)
    assert abs(loss - lo) <= 1e-3 * lo, (loss, lo)
    for k in go:                                  # bf16 operands: the bound of the other gradient tests
        assert relerr(g[k], go[k]) < 1e-2, (k, relerr(g[k], go[k]))


@pytest.mark.parametrize("n", [100, 128, 149 * 128 + 3])
def test_training_step_is_gradient_plus_adamw(world, n):
    p, F, mean, std, T, _ = setup_net(3, n)
    prop = L.Proposal()
    prop.set_params(p, mean, std, 0.5)
    for _ in range(2):
        loss, g = prop.grad(F, T)
        prop.adamw(g, lr=1e-3, wd=0.01)
    want = prop.params()
    prop.set_params(p, mean, std, 0.5)
    prop.set_data(F, T)
    losses = prop.train(2, batch_tiles=(n + 127) // 128, lr=1e-3, wd=0.01)
    got = prop.params()
    assert losses[1] == loss
    for k in want:
        assert np.array_equal(want[k], got[k]), k
