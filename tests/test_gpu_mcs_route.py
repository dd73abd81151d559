"""ether_mcs takes the same route whether or not a kernel variant was named before it, for both
models: a variant names the phase kernel of single calls, and the captured graphs do not depend
on it."""
import numpy as np
import pytest

import ether_gb300 as eg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,variant,L", [(eg.MODEL_ISING, 81, (16, 6, 8)), (eg.MODEL_XYZ, 5011, (8, 6, 10))])
def test_a_named_variant_leaves_the_loop_its_route(model, variant, L):
    lat = eg.simple_cubic(L)
    j = eg.couplings(1, [[(1, 1, (-1.0, -1.0, -1.0))]], [1.0])
    v = np.random.default_rng(5).normal(size=(lat.N, 3))
    ion = lat.ion.copy()
    ion[:, 1:4] = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)
    if model == eg.MODEL_ISING:
        ion[:, 1:4] = np.stack([0 * v[:, 0], 0 * v[:, 0], np.sign(v[:, 2])], axis=1)
    launches, states = [], []
    for name_it in (False, True):
        sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), model, replicas=3, seed=7, flags=eg.FLAG_NO_GRAPHS)
        sw.set_ladder(1.0 / (1e-3 * np.linspace(1.0, 3.0, 3)))
        sw.set_spins(ion)
        sw.zero_avg()
        if name_it:
            sw.set_variant(variant)
        n0 = sw.info().kernel_launches
        sw.mcs(0, 40, 11, 10)
        launches.append(sw.info().kernel_launches - n0)
        n0 = sw.info().kernel_launches
        sw.metropolis(20, accept=False)  # single calls do run the named variant's phases
        launches.append(sw.info().kernel_launches - n0)
        states.append((sw.sums(), sw.accept_counts(), sw.get_spins(lat.ion, 2)[:, 1:4]))
        sw.close()
    assert launches[0] == launches[2]
    assert launches[1] == 1 and launches[3] > 40
    for a, b in zip(*states):
        np.testing.assert_array_equal(a, b)
