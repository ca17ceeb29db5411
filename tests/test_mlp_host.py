"""The surrogate's host side on a stand-in for the CUDA runtime whose queued
copies happen as late as the runtime's contract allows
(tests/native/mlp_host_check.cpp, linked with the built boids_mlp.o)."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="session")
def mlp_host(boids_lib, tmp_path_factory):
    from boidssimulatormpi_gb300 import build as bld
    exe = str(tmp_path_factory.mktemp("mlp_host") / "mlp_host_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + bld.INCLUDE, "-I" + os.path.join(bld.cuda_home(), "include"),
                    os.path.join(ROOT, "tests", "native", "mlp_host_check.cpp"),
                    os.path.join(bld.BUILD, "boids_mlp.o"), "-o", exe], check=True)

    def run(*args):
        r = subprocess.run([exe, *[str(a) for a in args]], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        return [int(x) for x in r.stdout.split()]

    return run


@pytest.mark.parametrize("hidden", [256, 32])  # the fused batch, the general path
@pytest.mark.parametrize("epochs", [1, 2, 3, 8])
def test_every_epochs_order_reaches_the_device_as_drawn(mlp_host, hidden, epochs):
    """An epoch's row order stands in host memory until its copy has read it."""
    rc, copies, late, pending, orders, distinct = mlp_host("train", hidden, 1000, 256, epochs)
    assert rc == 0 and copies == 2 + epochs  # the rows, the targets and an order an epoch
    assert late == 0
    assert pending == 0
    assert orders == distinct == epochs


@pytest.mark.parametrize("fail_at", range(1, 31))
def test_a_failed_training_call_leaves_no_copy_of_host_memory(mlp_host, fail_at):
    """Whatever operation fails, nothing queued still reads host memory when the call returns."""
    rc, _, late, pending, orders, _ = mlp_host("train", 256, 1000, 256, 4, fail_at)
    assert rc != 0
    assert late == 0 and pending == 0 and orders >= 0


@pytest.mark.parametrize("fail_at,images", [(0, 0), (1, 1), (2, 1)])
def test_weight_image_is_kept_only_when_it_was_laid_out(mlp_host, fail_at, images):
    """A forward call whose upload or weight image failed leaves no image for
    the next one to take for the present parameters'."""
    rc1, rc2, laid = mlp_host("image", fail_at)
    assert (rc1 != 0) == (fail_at != 0) and rc2 == 0
    assert laid == images
