"""The simple-cubic XYZ kernel's columns at their edges: with enough replicas for chunks of 8 (and,
as a variant, 4 and 16) planes, which do not divide the lattices' heights; faces in every
direction; with and without field and anisotropy; bit for bit against the oracle's FP32 mirror."""
import numpy as np
import pytest

import ether_gb300 as eg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

OPTIONS = [dict(), dict(zeeman=True, h=(0.3, 0.1, 2.0), g_factor=2.0, sia=True,
                        sia_vec=np.array([[0.1e-3, -0.2e-3, 0.3e-3]]))]
R = 960  # six blocks per SM of one block per replica


@pytest.mark.parametrize("opts", OPTIONS)
@pytest.mark.parametrize("variant", [5011, 5012, 5013])
@pytest.mark.parametrize("L", [(4, 4, 22), (6, 4, 10), (10, 6, 18)])
def test_xyz_columns_match_fp32_mirror(L, variant, opts):
    lat = eg.simple_cubic(L)
    j = eg.couplings(1, [[(1, 1, (-1.0, -1.0, -1.0))]], [1.0])
    sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), eg.MODEL_XYZ, replicas=R, seed=77, **opts)
    osys = po.System.from_lattice(lat, j, np.array([1.0]), eg.MODEL_XYZ, **opts)
    beta = 1.0 / 1.443e-3
    sw.set_beta(beta)
    sw.set_variant(variant)
    v = np.random.default_rng(5).normal(size=(lat.N, 3))
    ion = lat.ion.copy()
    ion[:, 1:4] = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)
    sw.set_spins(ion)
    sw.metropolis(5, accept=False)
    assert sw.info().fast_path == 1
    n, col, rank = osys.colouring()
    for r in (0, R // 2, R - 1):
        g = sw.get_spins(lat.ion, r)
        work = ion.copy()
        sp4 = osys.spin4(work)
        for t in range(5):
            osys.metropolis_colour(work, sp4, 32, beta, 77, r, t, col, rank, n)
        np.testing.assert_array_equal(g[:, 1:4].astype(np.float32), sp4[:, :3], err_msg="replica %d" % r)
