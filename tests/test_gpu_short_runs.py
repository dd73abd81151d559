"""Short runs of sweeps, which some contexts keep in shared memory and some leave to the phases (by their
length, the replicas' size and whether a graph replays them): series, loops and single calls give
the bits of ETHER_FLAG_NO_RESIDENT whatever is chosen."""
import numpy as np
import pytest

import ether_gb300 as eg

pytestmark = pytest.mark.gpu


# both sides of the rules: many tiny replicas, few large ones, and some between
@pytest.mark.parametrize("model,size,bc,R", [
    (eg.MODEL_ISING, (8, 4, 4), "ccc", 34000), (eg.MODEL_ISING, (16, 16, 16), "ccc", 1060),
    (eg.MODEL_ISING, (29, 27, 25), "ccc", 1), (eg.MODEL_ISING, (21, 18, 15), "cco", 2), (eg.MODEL_ISING, (7, 5, 9), "ccc", 2),
    (eg.MODEL_XYZ, (20, 20, 20), "ccc", 1), (eg.MODEL_XYZ, (16, 16, 16), "ccc", 5), (eg.MODEL_XYZ, (8, 8, 8), "ccc", 3),
    (eg.MODEL_XYZ, (23, 21, 19), "ccc", 1), (eg.MODEL_XYZ, (9, 9, 9), "cco", 2)])
def test_short_runs_equal_phases(model, size, bc, R):
    lat = eg.simple_cubic(size, bc=bc)
    j = eg.couplings(1, [[(1, 1, (-1.0, -0.9, -1.0))]], [1.0])
    v = np.random.default_rng(5).normal(size=(lat.N, 3))
    ion = lat.ion.copy()
    ion[:, 1:4] = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)
    if model == eg.MODEL_ISING:
        ion[:, 1:3] = 0.0
        ion[:, 3] = np.sign(v[:, 2])
    out = []
    for flags in (0, eg.FLAG_NO_RESIDENT):
        sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), model, replicas=R, seed=7, flags=flags)
        if R > 1:
            sw.set_ladder(1.0 / (1e-3 * np.linspace(1.0, 5.0, R)))
        else:
            sw.set_beta(1.0 / 2e-3)
        sw.set_spins(ion)
        sw.zero_avg()
        rows = [sw.record_series(6 * s + 1, s) for s in (1, 2, 3, 5)]
        swaps = 0
        for coa in (1, 2, 4, 9):
            swaps = sw.mcs(0, 24, 3, coa, ovrr=model == eg.MODEL_XYZ, ovrr_para=1.0, ovrr_mcs=5, pt=R > 1,
                           exchange_interval=3, swap_count=swaps)
        acc = [sw.metropolis(n) for n in (1, 2, 3)]
        out.append((*rows, np.stack(acc), swaps, sw.slots(), sw.sums(), sw.accept_counts(),
                    np.stack([sw.get_spins(lat.ion, r)[:, 1:4] for r in sorted({0, R // 2, R - 1})])))
        sw.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
