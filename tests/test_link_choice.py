"""The way of small record calls (csrc/link_choice.h) on simulated links: the kernel alone on a good
one, the form shared with the host's cores on a slow one, and back when the link recovers."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ether_gb300", "csrc")

# argv: MB per call, ms of sweeps that a call waits for, then (calls, link GB/s) pairs; prints of each the
# total ms without the sweeps, the calls by the kernel alone and those timed on the device
PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "link_choice.h"
int main(int argc, char **argv) {
    ether::LinkChoice link;
    const size_t bytes = (size_t)(atof(argv[1]) * (1 << 20));
    const double sweeps = atof(argv[2]);
    for (int a = 3; a + 1 < argc; a += 2) {
        double total = 0.0;
        int alone = 0, timed = 0;
        for (int k = 0; k < atoi(argv[a]); ++k) {
            const double ms = bytes / (atof(argv[a + 1]) * 1e6);
            if (link.kernel_alone(bytes)) {
                ++alone;
                total += ms;
                const bool t = link.time_it(bytes);
                timed += t;
                link.took(bytes, ms + sweeps, t ? ms : 0.0);
            } else {
                total += ether::LinkChoice::shared_ms(bytes);
            }
        }
        printf("%.6f %d %d\\n", total, alone, timed);
    }
}
"""


@pytest.fixture(scope="module")
def simulate(tmp_path_factory):
    d = tmp_path_factory.mktemp("link")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def run(mb, *phases, sweeps=0.0):
        out = subprocess.run([str(d / "main"), str(mb), str(sweeps), *[str(v) for p in phases for v in p]],
                             capture_output=True, text=True, check=True).stdout
        return [(float(a), int(b), int(t)) for a, b, t in (l.split() for l in out.splitlines())]
    return run


@pytest.mark.parametrize("sweeps", [0.0, 50.0])
@pytest.mark.parametrize("mb", [1, 15.9, 16, 60, 128])
def test_a_good_link_always_takes_the_kernel(simulate, mb, sweeps):
    good = simulate(mb, (1, 20.0), (200, 170.0), sweeps=sweeps)[1]  # a slow first call changes nothing
    assert good[1] == 200
    assert good[2] <= (1 if sweeps == 0.0 else 200 // 32 + 2)  # and hardly a call is timed


@pytest.mark.parametrize("sweeps", [0.0, 50.0])
@pytest.mark.parametrize("mb,gbs", [(128, 27.0), (128, 10.0), (60, 20.0), (128, 45.0)])
def test_a_slow_link_ends_near_the_shared_form(simulate, mb, gbs, sweeps):
    calls = 400
    total, alone, timed = simulate(mb, (calls, gbs), sweeps=sweeps)[0]
    kernel, shared = mb * 2 ** 20 / (gbs * 1e6), 1.2 + mb * 2 ** 20 / 1e8
    assert kernel > shared and alone <= 3 + calls // 32 + 1
    assert total <= calls * shared + alone * (kernel - shared) + 1e-6


def test_calls_too_small_to_share_stay_with_the_kernel(simulate):
    assert simulate(15, (50, 13.0))[0][1] == 50
    assert simulate(30, (50, 27.0))[0][1] == 50  # 1.2 ms by the kernel, 1.5 shared


@pytest.mark.parametrize("sweeps", [0.0, 50.0])
def test_a_link_that_changes_is_followed(simulate, sweeps):
    slow, good, again = simulate(128, (100, 20.0), (100, 170.0), (200, 20.0), sweeps=sweeps)
    assert slow[1] < 8 and good[1] >= 100 - 32
    assert again[1] <= 32 + 3 + 200 // 32 + 1
