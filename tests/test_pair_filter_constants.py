"""The all-pairs product filter with the constants that the engine ships
(boids_engine.h, ap_filter), from fields of 400 radii to radii of a million
fields: the two half-precision terms that carry its threshold are finite, and
every pair in reach gets a product with the sign of a pass."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

f16, f32 = np.float16, np.float32


@pytest.fixture(scope="module")
def constants(tmp_path_factory):
    from boidssimulatormpi_gb300 import build as bld
    exe = str(tmp_path_factory.mktemp("ap_filter") / "ap_filter_constants")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-I" + bld.CSRC,
                    "-I" + os.path.join(bld.cuda_home(), "include"),
                    os.path.join(ROOT, "tests", "native", "ap_filter_constants.cpp"), "-o", exe], check=True)

    def get(radius, field):
        r = subprocess.run([exe], input="%r %r\n" % (radius, field), capture_output=True, text=True, check=True)
        return [float(x) for x in r.stdout.split()]

    return get


def embed(x, field, turn):
    """k_ap_embed's cosines and sines of coordinates within 4 F."""
    a = (x * f32(turn)).astype(f32).astype(np.float64) * np.pi
    return np.stack([np.cos(a).astype(f32).astype(f16), np.sin(a).astype(f32).astype(f16)], -1).reshape(len(x), 6)


@pytest.mark.parametrize("radius,field", [(0.05, 1.6), (0.05, 4.0), (0.05, 0.16), (0.1, 0.205), (0.01, 4.0), (2.0, 64.0),
                                          (0.05, 0.02), (1.0, 0.05), (1.0, 0.0172), (1.0, 0.01), (1.0, 1e-6),
                                          (1e30, 1.0), (float("inf"), 1.0), (1.0, 1e-39)])
def test_shipped_filter_keeps_every_pair_in_reach(constants, radius, field):
    rf, turn, least, _, _ = constants(radius, field)
    assert np.isfinite(turn) and -4.0 <= least < 3.0
    w = f16(f32(-least))
    u = f16(f32(-least) - f32(w))
    assert np.isfinite(w) and np.isfinite(u)
    rng = np.random.default_rng(5)
    n = 50000
    with np.errstate(over="ignore", under="ignore"):
        xi = rng.uniform(-4 * field, 4 * field, (n, 3))
        d = rng.standard_normal((n, 3))
        d *= min(rf, 8 * field) * np.where(rng.random((n, 1)) < 0.7, 1.0, rng.random((n, 1))) / \
            np.linalg.norm(d, axis=1)[:, None]
        xj = xi + d
        inside = np.abs(xj).max(1) <= 4 * field
        a, b = embed(xi.astype(f32), field, turn), embed(xj.astype(f32), field, turn)
    s = np.zeros(n, f32)
    for c in range(6):
        s = (s + a[:, c].astype(f32) * b[:, c].astype(f32)).astype(f32)
    s = s + f32(w) + f32(u)
    assert inside.sum() > 50
    assert not np.signbit(s[inside]).any()


@pytest.mark.parametrize("radius,field", [(0.05, 1.6), (0.05, (777 / 16384) ** (1 / 3)), (0.05, (65537 / 16384) ** (1 / 3)),
                                          (0.05, 0.16), (1.0, 0.05), (float("inf"), 1.0)])
def test_rows_and_columns_past_the_end_are_rejected(constants, radius, field):
    """A row or column of padding makes a negative product with every boid's
    vector, one too far outside for its angles included: none of its pairs is
    queued for the exact tests."""
    _, _, least, far, pad = constants(radius, field)
    pad = np.uint16(int(pad)).view(f16)
    w = f32(f16(f32(-least)))
    u = f32(-least) - w
    for extra in (0.0, far):  # a boid's (w, u); the other side's terms are 1, a padding's angles 0
        bw, bu = f32(f16(w + f32(extra))), f32(f16(u + f32(extra)))
        assert f32(pad) + bu < 0 and bw + f32(pad) < 0
    assert f32(pad) + f32(pad) < 0
