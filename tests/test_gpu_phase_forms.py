"""The launch-per-phase forms of lattices small enough for the resident sweeps, which take them unless
ETHER_FLAG_NO_RESIDENT says otherwise: the kernels of every common neighbour count, eight sites a
thread, and the replica parts.  Larger lattices and several species always run so."""
import numpy as np
import pytest

import ether_gb300 as eg
from tests.helpers import beta_of, make_pair, random_ising, random_xyz
from tests.test_gpu_sweep import FM, _lattice, ising_replay, xyz_replay

pytestmark = pytest.mark.gpu

NO = eg.FLAG_NO_RESIDENT


@pytest.mark.parametrize("kind", ["bcc", "fcc", "sc2"])
def test_phase_kernels_of_every_width_match_the_oracle(kind):
    lat, shells = _lattice(kind)
    sw, ion, g, ao, ag = ising_replay(lat, shells, 4.0, 12, flags=NO)
    np.testing.assert_array_equal(g[:, 3], ion[:, 3])
    assert ao == pytest.approx(ag, abs=1e-12)
    sw, osys, sp4, ion64, g = xyz_replay(lat, shells, 1.5, 12, flags=NO)
    for k, col in ((1, 0), (2, 1), (3, 2), (5, 3)):
        np.testing.assert_array_equal(g[:, k].astype(np.float32), sp4[:, col])


def test_eight_sites_a_thread_match_the_oracle():
    lat = eg.simple_cubic(32)  # 48 replicas: enough groups of eight to fill the GPU
    sw, osys = make_pair(lat, eg.MODEL_ISING, FM, replicas=48, flags=eg.FLAG_FORCE_GENERAL | NO)
    beta = beta_of(4.511)
    sw.set_beta(beta)
    ncol, col, rank = osys.colouring()
    ion = random_ising(lat, 100)
    sw.set_spins(ion)
    sw.metropolis(3)
    for r in (0, 47):
        work = ion.copy()
        for t in range(3):
            osys.metropolis_colour(work, None, 64, beta, 1992, r, t, col, rank, ncol)
        np.testing.assert_array_equal(sw.get_spins(lat.ion, r)[:, 3], work[:, 3])


@pytest.mark.parametrize("model", [eg.MODEL_XYZ, eg.MODEL_ISING])
@pytest.mark.parametrize("R,parts", [(18, 2), (36, 4)])
def test_replica_parts_equal_single_sweeps(model, R, parts):
    """ether_metropolis(n) and ether_mcs in two or four replica parts against one sweep a call."""
    lat = eg.pyrochlore(2, shells=(2.97243, 5.1484), tol=1e-3)
    shells = [[(1, 1, (1.0, 1.0, 1.0))], [(1, 1, (-0.1, -0.1, -0.1))]]
    ion = random_xyz(lat, 8) if model == eg.MODEL_XYZ else random_ising(lat, 8)
    runs = []
    for whole in (True, False):
        sw, _ = make_pair(lat, model, shells, replicas=R, flags=NO, zeeman=True, h=(0.0, 0.0, 1.0), g_factor=2.0)
        sw.set_ladder([beta_of(0.5 * 1.25 ** k) for k in range(6)])
        sw.set_spins(ion)
        sw.zero_avg()
        ncol = sw.info().n_colours
        if whole:
            n0 = sw.info().kernel_launches
            sw.metropolis(12, accept=False)
            assert sw.info().kernel_launches - n0 == parts * (12 * ncol + 1)
            swap = sw.mcs(0, 40, 6, 5, pt=True, exchange_interval=3)
        else:
            for _ in range(12):
                sw.metropolis(1, accept=False)
            swap = 0
            for step in range(1, 41):
                sw.metropolis(1, accept=False)
                if step % 3 == 0 and step % 5 != 0:
                    swap += 1
                    sw.parallel_tempering(swap)
                sw.observable(step, 6, 5)
        runs.append((swap, sw.slots(), sw.sums(), sw.accept_counts(),
                     np.stack([sw.get_spins(lat.ion, r)[:, [1, 2, 3, 5]] for r in range(R)])))
        sw.close()
    for a, b in zip(*runs):
        np.testing.assert_array_equal(a, b)
