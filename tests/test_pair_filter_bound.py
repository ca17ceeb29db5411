"""The all-pairs engine's product filter, checked on the CPU.

k_ap_pairs keeps a pair when the half-precision inner product of the boids'
(cos, sin) of 2 pi x / F over the axes is at least ap_min (boids_capi.cpp,
make_constants, holds the error budget).  That is exact-safe only if every
pair within the filter radius passes.  This restates the arithmetic with
numpy (angles and sums in float32, the vectors rounded to float16) on pairs
at the radius and inside it, for fields from three radii to 400, with boids
up to 4 F outside the field and pairs across its faces.
"""
import numpy as np

f16, f32 = np.float16, np.float32


def embed(x, F):
    turn = (x * f32(2.0 / F)).astype(f32)
    a = turn.astype(np.float64) * np.pi  # sincospi is exact to float32 rounding
    return np.stack([np.cos(a).astype(f32).astype(f16), np.sin(a).astype(f32).astype(f16)], -1).reshape(len(x), 6)


def test_product_filter_keeps_every_pair_in_reach():
    rng = np.random.default_rng(11)
    for R, F in [(0.05, 1.6), (0.05, 4.0), (0.05, 0.16), (0.1, 1.0), (0.1, 0.205), (0.01, 4.0), (2.0, 64.0)]:
        ulp = float(np.nextafter(f32(max(F, 1.0)), f32(np.inf)) - f32(max(F, 1.0)))
        rf = R * (1 + 1e-4) + 8 * ulp
        r = 2 * np.pi * (rf * (1 + 1e-4) + 8 * ulp) / F
        ap_min = f32(3.0 - r * r / 2 - 2.3e-3)
        ap_min = ap_min if float(ap_min) <= 3.0 - r * r / 2 - 2.3e-3 else np.nextafter(ap_min, f32(-np.inf))
        n = 200000
        xi = rng.uniform(0, F, (n, 3))
        xi[: n // 4] = rng.uniform(-4 * F, 4 * F, (n // 4, 3))
        d = rng.standard_normal((n, 3))
        d *= rf * np.where(rng.random((n, 1)) < 0.7, 1.0, rng.random((n, 1))) / np.linalg.norm(d, axis=1)[:, None]
        xj = xi + d
        half = rng.random((n, 3)) < 0.5  # the same point seen across a face
        xj = np.where(half & (xj < 0), xj + F, np.where(half & (xj > F), xj - F, xj))
        inside = np.abs(xj).max(1) <= 4 * F
        a, b = embed(xi.astype(f32), F), embed(xj.astype(f32), F)
        s = np.zeros(n, f32)
        for c in range(6):
            s = (s + a[:, c].astype(f32) * b[:, c].astype(f32)).astype(f32)
        assert (s[inside] >= ap_min).all(), (R, F, float((s[inside] - ap_min).min()))
