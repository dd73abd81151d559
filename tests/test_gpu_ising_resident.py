"""Small simple-cubic Ising lattices in shared memory (sweeps, measurements and acceptances in one
launch) against the launch-per-phase form: same draws, so spins, sums, slots and acceptances are
the same bits.  Extents at the edges of the kernel's forms: vectors of 4, 8 and 16 bytes; less than
a warp of them, one per thread, two per thread (with a remainder), and too many (the loop)."""
import numpy as np
import pytest

import ether_gb300 as eg
from tests.helpers import beta_of

pytestmark = pytest.mark.gpu

FM = [[(1, 1, (-1.0, -1.0, -1.0))]]


@pytest.mark.parametrize("L,R,field", [((8, 4, 4), 1, 0.0), ((8, 6, 10), 3, 0.7), ((16, 8, 6), 2, 0.0),
                                       ((32, 32, 32), 1, 0.7), ((24, 24, 18), 2, 0.0), ((16, 32, 34), 2, 0.0),
                                       ((32, 32, 64), 2, 0.0), ((32, 32, 66), 80, 0.0)])
def test_resident_run_equals_phases(L, R, field):
    lat = eg.simple_cubic(L)
    kw = dict(zeeman=True, h=(0.0, 0.0, field), g_factor=2.0) if field else {}
    rng = np.random.default_rng(2)
    ion = lat.ion.copy()
    ion[:, 3] = rng.choice([-1.0, 1.0], size=lat.N)
    out = []
    for flags in (0, eg.FLAG_NO_RESIDENT):
        j = eg.couplings(1, FM, [1.0])
        sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), eg.MODEL_ISING, replicas=R, seed=7, flags=flags, **kw)
        temps = np.linspace(3.0, 6.0, R)
        if R > 1:
            sw.set_ladder([beta_of(k) for k in temps])
        else:
            sw.set_beta([beta_of(4.5)])
        sw.set_spins(ion)
        sw.zero_avg()
        acc = [sw.metropolis(n) for n in (1, 7, 300)]
        sw.mcs(0, 40, 11, 3, pt=R > 1, exchange_interval=7)
        sw.mcs(40, 5, 11, 3)
        out.append((np.stack(acc), sw.sums(), sw.slots(), sw.accept_counts(), sw.tot_energy(),
                    np.stack([sw.get_spins(lat.ion, r)[:, 3] for r in range(min(R, 3))])))
        sw.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
