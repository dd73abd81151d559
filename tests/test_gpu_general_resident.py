"""The general lattices' resident sweep against the launch-per-phase form and the oracle: one block
and clusters of 2 and 4 per replica, sites with fewer neighbours than slots (open boundaries),
classes of odd size, one and two shells, both models, all bit for bit."""
import numpy as np
import pytest

import ether_gb300 as eg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

SHELLS = {1: [[(1, 1, (-1.0, -0.9, -1.1))]], 2: [[(1, 1, (1.0, 0.8, 1.2))], [(1, 1, (-0.1, -0.2, -0.1))]]}


def lattice(name):
    if name == "pyro":
        return eg.pyrochlore((3, 3, 4), shells=(2.97243, 5.1484), tol=1e-3), 2
    sizes, bc = {"open": ((7, 5, 9), "ooc"), "odd": ((9, 5, 7), "ccc"), "two": ((25, 21, 31), "cco"),
                 "four": ((33, 31, 45), "ooo")}[name]
    return eg.simple_cubic(sizes, bc=bc), 1


def sweep(lat, nsh, model, R, flags, **kw):
    j = eg.couplings(1, SHELLS[nsh], [1.0])
    sw = eg.Sweep.from_lattice(lat, j, np.array([1.0]), model, replicas=R, seed=11, flags=flags, **kw)
    sw.set_ladder(1.0 / np.linspace(0.8e-3, 4e-3, R))
    rng = np.random.default_rng(3)
    ions = np.empty((R, lat.N, 9))
    ions[:] = lat.ion
    if model == eg.MODEL_ISING:
        ions[:, :, 1:4] = 0.0
        ions[:, :, 3] = rng.choice([-1.0, 1.0], size=(R, lat.N))
    else:
        v = rng.normal(size=(R, lat.N, 3))
        ions[:, :, 1:4] = (v / np.linalg.norm(v, axis=2, keepdims=True)).astype(np.float32)
    sw.set_spins_batch(ions)
    return sw, ions, j


# "two" (16 275 sites) and "four" (46 035) need clusters of 2 and 4 for the XYZ model
@pytest.mark.parametrize("name,R", [("pyro", 3), ("open", 5), ("odd", 2), ("two", 70), ("four", 36)])
@pytest.mark.parametrize("model,opts", [(eg.MODEL_ISING, dict(zeeman=True, h=(0.0, 0.0, 2.0))),
                                        (eg.MODEL_XYZ, dict()),
                                        (eg.MODEL_XYZ, dict(zeeman=True, h=(0.5, 0.0, 2.0), angle=True, dphi=0.7))])
def test_resident_equals_phases(name, R, model, opts):
    lat, nsh = lattice(name)
    out = []
    for flags in (0, eg.FLAG_NO_RESIDENT):
        sw, ions, j = sweep(lat, nsh, model, R, flags, **opts)
        acc = sw.metropolis(3)
        sw.zero_avg()
        swaps = sw.mcs(0, 24, 2, 4, pt=True, exchange_interval=3)
        got = sw.get_spins_batch(ions.copy())
        out.append((got, acc, swaps, sw.slots(), sw.sums(), sw.slot_accept_counts()))
        sw.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("model", [eg.MODEL_ISING, eg.MODEL_XYZ])
@pytest.mark.parametrize("name", ["pyro", "open", "odd"])
def test_resident_equals_the_oracle(name, model):
    lat, nsh = lattice(name)
    sw, ions, j = sweep(lat, nsh, model, 2, 0)
    osys = po.System.from_lattice(lat, j, np.array([1.0]), model)
    n, col, rank = osys.colouring()
    sw.metropolis(5, accept=False)
    got = sw.get_spins_batch(ions.copy())
    for r, beta in enumerate(1.0 / np.linspace(0.8e-3, 4e-3, 2)):
        work = ions[r].copy()
        sp4 = osys.spin4(work) if model == eg.MODEL_XYZ else None
        for t in range(5):
            osys.metropolis_colour(work, sp4, 32 if model == eg.MODEL_XYZ else 64, beta, 11, r, t, col, rank, n)
        if model == eg.MODEL_XYZ:
            np.testing.assert_array_equal(got[r, :, 1:4].astype(np.float32), sp4[:, :3])
        else:
            np.testing.assert_array_equal(got[r, :, 3], work[:, 3])
