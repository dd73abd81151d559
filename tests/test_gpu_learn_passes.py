"""Learned Ising sweeps whose class is more than one pass of patches, and tiles with a remainder:
the oracle replays replicas on both sides of the pass boundary bit for bit, given the logits."""
import numpy as np
import pytest

import ether_gb300 as eg
from oracle import pyoracle as po
from tests.helpers import beta_of
from tests import test_gpu_learn_xyz as xyz
from tests.test_gpu_learn import FM, KTC, random_params, storage_spins

pytestmark = pytest.mark.gpu


# 64^3: 2048 patches of a class per replica, 512 replicas a pass; 8 x 24 x 16: 12 (a last tile of
# 12 R mod 128 rows); 8^3: 4, one tile's rows from 32 replicas
@pytest.mark.parametrize("L,R,look", [(64, 514, (0, 511, 512, 513)), ((8, 24, 16), 33, (0, 10, 11, 32)),
                                      (8, 65, (0, 31, 32, 64))])
def test_passes_and_remainders_replay(L, R, look):
    lat = eg.simple_cubic(L)
    j = eg.couplings(1, FM, [1.0])
    sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), eg.MODEL_ISING, replicas=R, seed=1992)
    kT = np.linspace(0.7 * KTC, 4.0 * KTC, R)
    sw.set_beta([beta_of(k) for k in kT])
    ion = lat.ion.copy()
    ion[:, 3] = np.random.default_rng(3).choice([-1.0, 1.0], size=lat.N)
    sw.set_spins(ion)
    lr = eg.Learned(sw, seed=9, capacity=4096)
    lr.set_params(random_params(5))
    lr.set_dump(True)
    Ls = [L] * 3 if np.isscalar(L) else list(L)
    stream = np.arange(R) + 40
    sw.set_streams(stream=stream.tolist(), step=[0] * R)
    sw.metropolis(1)  # the replicas part
    before = {r: storage_spins(lat, sw, r) for r in look}
    lr.sweep_(1)
    dump, acc = lr.dump(), lr.accepts()
    for r in look:
        sp = before[r]
        a = po.patch_sweep(sp, Ls, -1.0 / kT[r], np.ascontiguousarray(dump[:, r]), 1992, int(stream[r]), 0)
        np.testing.assert_array_equal(sp, storage_spins(lat, sw, r))
        assert a == int(acc[r])
    lr.close()


# the Heisenberg learner's patches: every wrap of every axis, three different extents
@pytest.mark.parametrize("L", [(16, 24, 8), (24, 8, 16)])
def test_heisenberg_patches_replay(L):
    xyz.test_learned_sweep_replays_bit_exact(L)
