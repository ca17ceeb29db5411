"""The autotuners' choice of a threshold set and of the split, on times of
flocks that have a choice of kernels and of flocks that do not."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    from boidssimulatormpi_gb300 import build as bld
    exe = str(tmp_path_factory.mktemp("tune_rule") / "tune_rule_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + bld.CSRC, "-I" + os.path.join(bld.cuda_home(), "include"),
                    os.path.join(ROOT, "tests", "native", "tune_rule_check.cpp"), "-o", exe], check=True)

    def run(ms, choice, routed):
        line = " ".join(str(x) for x in [*ms, choice, int(routed)])
        r = subprocess.run([exe], input=line, capture_output=True, text=True, check=True)
        return tuple(int(x) for x in r.stdout.split())

    return run


# us a step of (the default set, the other eight, the fastest with the choice of kernels)
UNIFORM = [102.5, 100.8, 101.2, 194.3, 396.1, 106.7, 225.8, 196.4, 97.5]
CLUSTERS = [680.0, 644.7, 983.9, 496.3, 445.9, 606.0, 642.6, 482.1, 3161.2]
COLLAPSED = [339.0, 330.0, 400.0, 320.0, 300.0, 290.0, 280.0, 310.0, 900.0]


@pytest.mark.parametrize("ms,choice,routed,want", [
    (UNIFORM, 102.0, True, (0, 0)),     # a few percent now are no reason to leave the default
    (CLUSTERS, 680.0, True, (4, 1)),    # the split with this set beats a warp per boid
    (COLLAPSED, 281.0, True, (6, 0)),   # the choice of kernels takes the split anyway: it stays
    (UNIFORM, 0.0, False, (8, 1)),      # no choice of kernels: the fastest set
    ([1.0] * 9, 1.0, True, (0, 0)),
])
def test_autotuners_choice(choose, ms, choice, routed, want):
    assert choose(ms, choice, routed) == want
