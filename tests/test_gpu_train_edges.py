"""The training kernels at the edges of their tiles: batches of less than one block of rows, of a
block and a remainder, and of one and two stages of the gradient sums with a remainder; loss and
gradient against the FP64 oracle within the FP32 bound that the full batch's tests use."""
import numpy as np
import pytest

import test_gpu_learn as ising
import test_gpu_learn_xyz as xyz
import ether_gb300 as eg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

BATCHES = [1, 7, 9, 64, 65, 130]


def check(g, go, blocks):
    for a, b in zip(blocks[:-1], blocks[1:]):
        assert np.linalg.norm(g[a:b] - go[a:b]) <= 1e-3 * np.linalg.norm(go[a:b]) + 1e-9, (a, b)


@pytest.mark.parametrize("B", BATCHES)
def test_ising_gradient_of_ragged_batches(B):
    lat, sw, _ = ising.ising(8, 1, ising.KTC)
    lr = eg.Learned(sw, seed=1, capacity=4096)
    p = ising.random_params(2)
    lr.set_params(p)
    rng = np.random.default_rng(B)
    x = ising.random_inputs(rng, B)
    y = rng.integers(0, 2 ** 32, size=B, dtype=np.uint64).astype(np.uint32)
    loss, g = lr.loss_grad(x, y)
    loss_o, go = po.mlp_loss_grad(p, x, y, quant=True)
    assert loss == pytest.approx(loss_o, rel=1e-5)
    check(g, go, [0, 16384, 16512, 32896, 33024, 37120, 37152])
    lr.close()


@pytest.mark.parametrize("B", BATCHES)
def test_heisenberg_gradient_of_ragged_batches(B):
    lat, sw, _ = xyz.heis(8, 1, xyz.KTC)
    lr = eg.Learned(sw, seed=1, capacity=4096)
    p = xyz.random_params(2)
    lr.set_params(p)
    rng = np.random.default_rng(B)
    x = xyz.random_inputs(rng, B)
    y = rng.normal(size=(B, 32, 3))
    y = (y / np.linalg.norm(y, axis=2, keepdims=True)).reshape(B, 96).astype(np.float32)
    loss, g = lr.loss_grad(x, y)
    loss_o, go = po.xmlp_loss_grad(p, x, y, quant=True)
    assert loss == pytest.approx(loss_o, rel=1e-5)
    check(g, go, [0, 38912, 39040, 55424, 55552, 67840, 67936])
    lr.close()
