"""Thousands of replicas of one block each: energies, magnetisations and recorded rows on both sides of
the counts where a row gets a launch of its own (512) and a replica a single block, against small
contexts of the same configurations (whose replicas have several blocks, or other launches)."""
import numpy as np
import pytest

import ether_gb300 as eg

pytestmark = pytest.mark.gpu


def context(lat, model, ions, flags=0):
    j = eg.couplings(1, [[(1, 1, (-1.0, -0.9, -1.1))]], [1.0])
    sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), model, replicas=len(ions), seed=7, flags=flags, zeeman=True,
                               h=(0.0, 0.0, 0.7), g_factor=2.0)
    sw.set_beta(1.0 / 3e-3)
    sw.set_spins_batch(ions)
    return sw


def configurations(lat, model, R):
    rng = np.random.default_rng(R)
    ions = np.empty((R, lat.N, 9))
    ions[:] = lat.ion
    v = rng.normal(size=(R, lat.N, 3))
    ions[:, :, 1:4] = (v / np.linalg.norm(v, axis=2, keepdims=True)).astype(np.float32)
    if model == eg.MODEL_ISING:
        ions[:, :, 1:3] = 0.0
        ions[:, :, 3] = np.sign(v[:, :, 2])
    return ions


# simple cubic and general, both sides of 512 rows; above 608 replicas every one has a single block
@pytest.mark.parametrize("model", [eg.MODEL_ISING, eg.MODEL_XYZ])
@pytest.mark.parametrize("size,R", [((8, 4, 4), 512), ((8, 4, 4), 513), ((8, 4, 4), 3000), ((5, 7, 3), 700),
                                    ((16, 16, 16), 620), ((15, 16, 16), 620)])
def test_sums_and_rows_of_single_blocks(model, size, R):
    lat = eg.simple_cubic(size)
    ions = configurations(lat, model, R)
    big = context(lat, model, ions)
    E, M = big.tot_energy(), big.tot_magnetisation()
    m, e = big.record_series(6, 2, energy=True)
    m2 = big.record_series(5, 1)
    direct = context(lat, model, ions, eg.FLAG_NO_GRAPHS)
    np.testing.assert_array_equal(direct.tot_energy(), E)
    for a, b in zip(direct.record_series(6, 2, energy=True), (m, e)):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(direct.record_series(5, 1), m2)
    M2 = big.tot_magnetisation()
    np.testing.assert_allclose(m2[:, -1], np.linalg.norm(M2, axis=1), rtol=1e-13)
    for r in (0, R // 2, R - 1):  # the same configuration alone: other blocks, the same terms
        one = context(lat, model, ions[r:r + 1])
        np.testing.assert_allclose(one.tot_energy()[0], E[r], rtol=1e-12, atol=1e-15 * lat.N)
        np.testing.assert_allclose(one.tot_magnetisation()[0], M[r], rtol=1e-12, atol=1e-12 * lat.N)
        one.close()
    big.close()
    direct.close()
