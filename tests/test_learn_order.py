"""A learned sweep that follows a training step uses the weights of that step: the kernels of a class
may overlap, and the network's kernel reads its weights before it has waited for the gather."""
import ctypes as C
import os
import re

import numpy as np
import pytest

import ether_gb300 as eg
from ether_gb300 import abi

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ether_gb300", "csrc")


# the kernel before the one that reads weights ahead of its wait
@pytest.mark.parametrize("source,kernel", [("k_learn.cu", "gather_kernel"), ("k_learn_xyz.cu", "xinputs_kernel")])
def test_the_kernel_before_the_network_waits_before_it_releases(source, kernel):
    text = open(os.path.join(CSRC, source)).read()
    body = re.search(r"__global__[^\n]*\b%s\([^{]*\{(.*?)\n\}\n" % kernel, text, re.S).group(1)
    assert 0 <= body.index("after_wait();") < body.index("after_release();")


@pytest.mark.gpu
@pytest.mark.parametrize("model", [eg.MODEL_ISING, eg.MODEL_XYZ])
def test_a_series_after_training_uses_the_new_weights(model):
    lat = eg.simple_cubic((16, 8, 24))
    j = eg.couplings(1, [[(1, 1, (-1.0, -1.0, -1.0))]], [1.0])
    rng = np.random.default_rng(4)
    ion = lat.ion.copy()
    ion[:, 1:4] = 0.0
    if model == eg.MODEL_ISING:
        ion[:, 3] = rng.choice([-1.0, 1.0], size=lat.N)
    else:
        v = rng.normal(size=(lat.N, 3))
        ion[:, 1:4] = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)

    def run(train, wait):
        sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), model, replicas=24, seed=5)
        sw.set_beta(1.0 / (4.511e-3 if model == eg.MODEL_ISING else 1.443e-3))
        sw.set_spins(ion)
        lr = eg.Learned(sw, seed=3, capacity=4096)
        sw.metropolis(20, accept=False)
        lr.collect(64)
        out = []
        for _ in range(4):
            if train:  # no loss asked for: nothing waits
                abi.check(lr.lib.ether_learn_train(lr.h, 3, 256, 0.05, C.POINTER(C.c_double)()))
            if wait:
                lr.params()
                sw.sync()
            out.append(lr.record_series(1, 0, 1, 1))
        out += [lr.accepts(), sw.get_spins(lat.ion, 23)[:, 1:4], lr.params()]
        lr.close()
        sw.close()
        return out

    got, want, untrained = run(True, False), run(True, True), run(False, True)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    assert not np.array_equal(got[0], untrained[0])  # the first step's weights already count
