"""The energy of a general XYZ lattice with few and with many couplings (64 fit in the reduction's
shared memory): against the oracle's FP64 sum."""
import numpy as np
import pytest

import ether_gb300 as eg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


# 4 species, one shell: 16 couplings; 6 species, two shells: 72; 8, one shell: 64
@pytest.mark.parametrize("nsp,shells", [(4, (1.0,)), (6, (1.0, 2 ** 0.5)), (8, (1.0,))])
def test_energy_with_many_couplings(nsp, shells):
    cart = np.zeros((nsp, 3))
    cart[:, 0] = np.arange(nsp)
    lat = eg.Lattice(cart, np.arange(1, nsp + 1), np.diag([float(nsp), 1.0, 1.0]), (3, 5, 7), shells)
    rng = np.random.default_rng(nsp)
    J = [[(a + 1, b + 1, tuple(rng.uniform(-1, 1, 3))) for a in range(nsp) for b in range(a, nsp)] for _ in shells]
    j = eg.couplings(nsp, J, [1.0] * nsp)
    s = np.ones(nsp)
    sw = eg.Sweep.from_lattice(lat, j, s, eg.MODEL_XYZ, replicas=3, seed=1)
    osys = po.System.from_lattice(lat, j, s, eg.MODEL_XYZ)
    v = rng.normal(size=(lat.N, 3)).astype(np.float32)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    ion = lat.ion.copy()
    ion[:, 1:4] = v
    sw.set_spins(ion)
    # FP32 fields: deg products and sums of at most 1 meV each, three components, per site
    deg = 6 + (12 if len(shells) > 1 else 0)
    tol = lat.N * deg * 3 * (deg + 4) * 2.0 ** -24 * 1e-3
    assert np.all(np.abs(sw.tot_energy() - osys.tot_energy(ion)) <= tol)
