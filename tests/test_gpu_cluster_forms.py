"""The resident sweeps that the other files compare with the phases do run resident, and the Heisenberg
ones on clusters of two and four blocks: sites with fewer neighbours than slots (the free slots
point at a spin of zeros in the site's own block), odd shares of a colour, one and two shells, a
basis.  The phase form is compared with the oracle elsewhere; here every bit equals it."""
import numpy as np
import pytest

import ether_gb300 as eg
from tests.test_gpu_general_resident import sweep

pytestmark = pytest.mark.gpu


def lattice(kind, size, bc):
    if kind == "pyro":
        return eg.pyrochlore(size, shells=(2.97243, 5.1484), tol=1e-3)
    if kind == "two":
        return eg.Lattice([[0.0, 0.0, 0.0]], [1], np.eye(3), size, [1.0, 1.41421356], bc=bc)
    return eg.simple_cubic(size, bc=bc)


def launches_of(sw, call):
    n0 = sw.info().kernel_launches
    out = call()
    return sw.info().kernel_launches - n0, out


# Blocks a replica: 33 x 31 x 45 fits in no fewer than four and 25 x 21 x 31 in no fewer than two;
# the others take them while all replicas still run at once
@pytest.mark.parametrize("opts", [dict(), dict(zeeman=True, h=(0.5, 0.0, 2.0), angle=True, dphi=0.7)])
@pytest.mark.parametrize("kind,size,bc,R", [("one", (21, 18, 15), "cco", 3), ("one", (21, 18, 15), "cco", 40),
                                            ("one", (13, 15, 17), "ccc", 3), ("two", (25, 21, 31), "cco", 50),
                                            ("two", (33, 31, 45), "ooo", 30), ("pyro", 7, "ccc", 2), ("pyro", 9, "ccc", 2)])
def test_clusters_equal_phases(kind, size, bc, R, opts):
    lat = lattice(kind, size, bc)
    out = []
    for flags in (0, eg.FLAG_NO_RESIDENT):
        sw, ions, j = sweep(lat, lat.nsh, eg.MODEL_XYZ, R, flags, **opts)
        n, acc = launches_of(sw, lambda: sw.metropolis(3))
        assert n == 1 if flags == 0 else n > 3 * sw.info().n_colours
        sw.zero_avg()
        swaps = sw.mcs(0, 24, 2, 4, pt=True, exchange_interval=3)
        out.append((sw.get_spins_batch(ions.copy()), acc, swaps, sw.slots(), sw.sums(), sw.slot_accept_counts()))
        sw.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


# what test_gpu_ising_clusters, test_gpu_ising_resident, test_gpu_series_resident and the small cases
# of test_gpu_general_resident compare: a call of five sweeps is one launch, by phases many
@pytest.mark.parametrize("model,kind,size,bc,R", [
    (eg.MODEL_ISING, "one", (21, 18, 15), "cco", 2), (eg.MODEL_ISING, "one", (23, 21, 19), "ccc", 3),
    (eg.MODEL_ISING, "one", (18, 26, 22), "cco", 1), (eg.MODEL_ISING, "one", (8, 4, 4), "ccc", 1),
    (eg.MODEL_ISING, "one", (8, 6, 10), "ccc", 3), (eg.MODEL_ISING, "one", (16, 8, 6), "ccc", 2),
    (eg.MODEL_ISING, "one", (32, 32, 32), "ccc", 1), (eg.MODEL_ISING, "one", (24, 24, 18), "ccc", 2),
    (eg.MODEL_ISING, "one", (16, 32, 34), "ccc", 2), (eg.MODEL_ISING, "one", (32, 32, 64), "ccc", 2),
    (eg.MODEL_ISING, "one", (32, 32, 66), "ccc", 80), (eg.MODEL_ISING, "one", (7, 9, 6), "ccc", 3),
    (eg.MODEL_XYZ, "one", (6, 8, 4), "ccc", 3), (eg.MODEL_XYZ, "one", (5, 7, 6), "ccc", 3),
    (eg.MODEL_ISING, "pyro", (3, 3, 4), "ccc", 3), (eg.MODEL_XYZ, "pyro", (3, 3, 4), "ccc", 3),
    (eg.MODEL_ISING, "one", (7, 5, 9), "ooc", 5), (eg.MODEL_XYZ, "one", (7, 5, 9), "ooc", 5)])
def test_the_compared_lattices_run_resident(model, kind, size, bc, R):
    lat = lattice(kind, size, bc)
    for flags in (0, eg.FLAG_NO_RESIDENT):
        sw, ions, j = sweep(lat, lat.nsh, model, R, flags)
        n, acc = launches_of(sw, lambda: sw.metropolis(5))
        assert n == 1 if flags == 0 else n > 5 * sw.info().n_colours
        sw.close()
