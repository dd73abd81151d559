"""General Ising lattices whose replicas take two blocks each: spins, sums, slots and acceptances are
the phase form's bits; odd colours, a remainder of the pairs' halves, single sweeps and runs."""
import numpy as np
import pytest

import ether_gb300 as eg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,bc,R", [((21, 18, 15), "cco", 2), ((23, 21, 19), "ccc", 3), ((18, 26, 22), "cco", 1)])
def test_two_blocks_equal_phases(L, bc, R):
    lat = eg.simple_cubic(L, bc=bc)
    j = eg.couplings(1, [[(1, 1, (-1.0, -1.0, -1.0))]], [1.0])
    ion = lat.ion.copy()
    ion[:, 1:3] = 0.0
    ion[:, 3] = np.random.default_rng(3).choice([-1.0, 1.0], size=lat.N)
    out = []
    for flags in (0, eg.FLAG_NO_RESIDENT):
        sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), eg.MODEL_ISING, replicas=R, seed=7, flags=flags)
        sw.set_ladder(1.0 / (1e-3 * np.linspace(3.0, 6.0, R))) if R > 1 else sw.set_beta(1.0 / 4.5e-3)
        sw.set_spins(ion)
        sw.zero_avg()
        acc = [sw.metropolis(n) for n in (1, 3, 260)]
        sw.mcs(0, 40, 11, 3, pt=R > 1, exchange_interval=7)
        out.append((np.stack(acc), sw.sums(), sw.slots(), sw.accept_counts(), sw.tot_energy(),
                    np.stack([sw.get_spins(lat.ion, r)[:, 3] for r in range(R)])))
        sw.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
