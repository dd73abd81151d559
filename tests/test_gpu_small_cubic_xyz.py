"""Small simple-cubic XYZ lattices, whose sweeps run in shared memory, against the launch-per-phase
form: same draws, so spins, sums, slots and acceptances are the same bits.  One block a replica up
to 14^3, clusters above; overrelaxation, PT, fields and angle proposals between and in the runs."""
import numpy as np
import pytest

import ether_gb300 as eg

pytestmark = pytest.mark.gpu

OPTIONS = [dict(), dict(zeeman=True, h=(0.3, 0.1, 2.0), g_factor=2.0, sia=True,
                        sia_vec=np.array([[0.1e-3, -0.2e-3, 0.3e-3]])), dict(angle=True, dphi=0.6)]


@pytest.mark.parametrize("opts", OPTIONS)
@pytest.mark.parametrize("L,R", [((4, 4, 4), 1), ((8, 6, 10), 3), ((14, 14, 14), 2), ((16, 16, 18), 2)])
def test_resident_run_equals_phases(L, R, opts):
    lat = eg.simple_cubic(L)
    j = eg.couplings(1, [[(1, 1, (-1.0, -1.0, -0.9))]], [1.0])
    v = np.random.default_rng(5).normal(size=(lat.N, 3))
    ion = lat.ion.copy()
    ion[:, 1:4] = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)
    out = []
    for flags in (0, eg.FLAG_NO_RESIDENT):
        sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), eg.MODEL_XYZ, replicas=R, seed=7, flags=flags, **opts)
        if R > 1:
            sw.set_ladder(1.0 / (1e-3 * np.linspace(0.8, 2.0, R)))
        else:
            sw.set_beta(1.0 / 1.443e-3)
        sw.set_spins(ion)
        sw.zero_avg()
        n0 = sw.info().kernel_launches
        acc = [sw.metropolis(n) for n in (1, 5, 300)]
        launches = sw.info().kernel_launches - n0
        sw.mcs(0, 40, 11, 3, ovrr=True, ovrr_para=1.0, ovrr_mcs=5, pt=R > 1, exchange_interval=7)
        out.append((launches, np.stack(acc), sw.sums(), sw.slots(), sw.accept_counts(), sw.tot_energy(),
                    np.stack([sw.get_spins(lat.ion, r)[:, 1:4] for r in range(R)])))
        sw.close()
    assert out[0][0] < 20 < out[1][0]  # runs, not phases
    for a, b in zip(out[0][1:], out[1][1:]):
        np.testing.assert_array_equal(a, b)
