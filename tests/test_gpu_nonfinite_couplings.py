"""Couplings that are not finite in FP32 on lattices whose sites have fewer neighbours than others: the
free neighbour slots of the resident sweep would add infinity times zero, so these lattices sweep by
phases, and the spins are those of ETHER_FLAG_NO_RESIDENT."""
import numpy as np
import pytest

import ether_gb300 as eg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jz", [-np.inf, np.inf, 1e42, np.nan, -1.0])
def test_free_slots_add_nothing(jz):
    lat = eg.simple_cubic((7, 5, 9), bc="ooc")
    j = eg.couplings(1, [[(1, 1, (-1.0, -1.0, jz))]], [1.0])
    v = np.random.default_rng(5).normal(size=(lat.N, 3))
    ion = lat.ion.copy()
    ion[:, 1:4] = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)
    out = []
    for flags in (0, eg.FLAG_NO_RESIDENT):
        sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), eg.MODEL_XYZ, replicas=2, seed=7, flags=flags)
        sw.set_beta(1.0 / 1e-3)
        sw.set_spins(ion)
        acc = sw.metropolis(3)
        out.append((acc, np.stack([sw.get_spins(lat.ion, r)[:, 1:4] for r in range(2)])))
        sw.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
