"""The simple-cubic Ising phase kernel's plane pairs at the edges of its tiles: row lengths of one
and several vectors of each width, colour arrays of less and of more than one block with a
remainder, in a field (all 14 thresholds distinct), bit for bit against the oracle's replay."""
import numpy as np
import pytest

import ether_gb300 as eg
from test_gpu_sweep import FM, ising_replay

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [162, 164, 1164, 82, 84, 1084, 42, 44, 1044])
@pytest.mark.parametrize("L", [(8, 4, 4), (16, 10, 6), (24, 18, 10), (32, 4, 4), (64, 20, 18), (96, 12, 8)])
def test_ising_plane_pairs_bit_exact(variant, L):
    width = variant % 1000 // 10
    if L[0] // 2 % width:
        pytest.skip("row length is not a multiple of the vector")
    kw = dict(zeeman=True, h=(0.0, 0.0, 3.0), g_factor=2.0)
    sw, ion, g, ao, ag = ising_replay(eg.simple_cubic(L), FM, 4.511, 6, variant=variant, **kw)
    np.testing.assert_array_equal(g[:, 3], ion[:, 3])
    assert ao == pytest.approx(ag, abs=1e-12)
