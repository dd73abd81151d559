"""Recorded series of lattices whose sweeps run in shared memory, against the launch-per-phase form:
the same bits row by row, with and without graphs, sweeps left over after the last row included."""
import numpy as np
import pytest

import ether_gb300 as eg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,L", [(eg.MODEL_ISING, (8, 8, 6)), (eg.MODEL_ISING, (7, 9, 6)), (eg.MODEL_XYZ, (6, 8, 4)),
                                     (eg.MODEL_XYZ, (5, 7, 6))])
@pytest.mark.parametrize("sweeps,stride", [(11, 3), (6, 1), (300, 280)])
def test_series_equals_phases(model, L, sweeps, stride):
    lat = eg.simple_cubic(L)
    j = eg.couplings(1, [[(1, 1, (-1.0, -1.0, -1.0))]], [1.0])
    rng = np.random.default_rng(5)
    ion = lat.ion.copy()
    if model == eg.MODEL_XYZ:
        v = rng.normal(size=(lat.N, 3))
        ion[:, 1:4] = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)
    else:
        ion[:, 1:4] = 0.0
        ion[:, 3] = rng.choice([-1.0, 1.0], size=lat.N)
    out = []
    for flags in (0, eg.FLAG_NO_GRAPHS, eg.FLAG_NO_RESIDENT):
        sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), model, replicas=3, seed=7, flags=flags)
        sw.set_beta(1.0 / 2e-3)
        sw.set_spins(ion)
        m, e = sw.record_series(sweeps, stride, energy=True)
        out.append((m, e, sw.accept_counts(), sw.get_spins(lat.ion, 2)[:, 1:4]))
        sw.close()
    for o in out[1:]:
        for a, b in zip(out[0], o):
            np.testing.assert_array_equal(a, b)
