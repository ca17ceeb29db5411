"""The rule that sends flocks over 40960 boids a warp per boid or to the cells'
split, at states both sides of which were timed: (what an even flock would have,
what the state has, boids or slots, kind, by a warp per boid)."""
import os
import subprocess

import pytest

from conftest import ROOT

HANDLE, BARE, ENSEMBLE = 0, 1, 2


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    from boidssimulatormpi_gb300 import build as bld
    exe = str(tmp_path_factory.mktemp("crowd_lines") / "crowd_lines")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + bld.CSRC, "-I" + os.path.join(bld.cuda_home(), "include"),
                    os.path.join(ROOT, "tests", "native", "crowd_lines.cpp"), "-o", exe], check=True)

    def get(even, n, kind):
        seen = 14.8 * even  # marun2019's cones: half of the ball
        r = subprocess.run([exe], input="%r %r %r %d\n" % (even, seen, n, kind), capture_output=True, text=True, check=True)
        return tuple(float(x) for x in r.stdout.split())

    return get


@pytest.mark.parametrize("even,pairs,n,kind,by_warp", [
    # the reference's density: uniform, gathering, gathered
    (0.29, 0.30, 65537, HANDLE, False), (0.29, 0.72, 65537, HANDLE, True), (0.29, 3.0, 65537, HANDLE, True),
    (0.29, 0.75, 262143, HANDLE, False), (0.29, 1.3, 262143, HANDLE, True),
    (0.29, 0.30, 300000, BARE, False), (0.29, 2.3, 65537, BARE, True),
    (0.29, 0.30, 65536, ENSEMBLE, False), (0.29, 0.38, 65536, ENSEMBLE, False), (0.29, 0.46, 65536, ENSEMBLE, True),
    (0.29, 0.57, 131072, ENSEMBLE, False), (0.29, 0.79, 131072, ENSEMBLE, True),
    (0.29, 0.37, 262144, ENSEMBLE, False), (0.29, 0.68, 262144, ENSEMBLE, False), (0.29, 1.0, 262144, ENSEMBLE, True),
    (0.29, 0.79, 491520, ENSEMBLE, False), (0.29, 1.34, 491520, ENSEMBLE, True), (0.29, 3.1, 491520, ENSEMBLE, True),
    (0.29, 3.7, 393216, ENSEMBLE, True),
    # a quarter of it
    (0.07, 0.27, 100000, ENSEMBLE, False), (0.07, 0.50, 100000, ENSEMBLE, True),
    (0.07, 0.62, 256000, ENSEMBLE, False), (0.07, 1.15, 256000, ENSEMBLE, True),
    # uniform at twice, 6, 12 and 24 times that, and the same gathered
    (0.58, 0.58, 262144, ENSEMBLE, True), (0.58, 0.58, 393216, ENSEMBLE, True),
    (1.74, 1.74, 65537, HANDLE, False), (1.74, 1.74, 262143, HANDLE, False), (1.74, 3.0, 65537, HANDLE, True),
    (1.74, 1.74, 262143, BARE, False), (2.32, 2.32, 262143, BARE, True),
    (1.74, 1.74, 262144, ENSEMBLE, False), (1.74, 1.74, 65536, ENSEMBLE, True),
    (3.48, 3.48, 131072, HANDLE, True), (4.64, 4.64, 393216, ENSEMBLE, False), (6.96, 6.96, 262143, HANDLE, True), (13.9, 13.9, 41000, HANDLE, True),
    (16.4, 16.4, 131072, HANDLE, False),
    # collapsed
    (0.29, 16.0, 262143, HANDLE, False), (0.29, 8.0, 131072, ENSEMBLE, False), (43.0, 43.0, 65537, HANDLE, False),
])
def test_route_of_timed_states(lines, even, pairs, n, kind, by_warp):
    line, top = lines(even, float(n), kind)
    assert (line <= pairs and (pairs < top or kind == BARE)) == by_warp
