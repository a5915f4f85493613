"""The chase's fixed-point rotation (get_rotation form 0) where its rounding is hardest: the
oracle's givensAlgorithm, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -52


def near(rng, base, m):
    """m values within a few ulps of base on either side."""
    return base * (1.0 + rng.integers(-6, 7, m) * ULP / 2)


def pairs(kind, rng, m=4000):
    k = np.ldexp(1.0, rng.integers(-40, 41, m))
    if kind == "square":        # exact square roots and quotients
        t = np.array([(3, 4), (5, 12), (8, 15), (7, 24), (20, 21), (1, 0.75), (0.28, 0.96)])
        p = t[rng.integers(0, len(t), m)]
        return p[:, 0] * k, p[:, 1] * k
    if kind == "power":         # x just off a power of two (the seed's and the fields' edges)
        f = near(rng, 1.0, m) * k
        return f, f * np.ldexp(rng.random(m) + 0.5, rng.integers(-60, -10, m))
    if kind == "equal":         # c and s near sqrt(1/2), x near twice a square
        f = (1.0 + rng.random(m)) * k
        return f, near(rng, 1.0, m) * f
    if kind == "midpoint":      # sqrt(x) within 2^-104 of a rounding midpoint: x = 1 + odd ulps
        return np.sqrt(1.0 + (2 * rng.integers(0, 200, m) + 1) * ULP) * k, near(rng, 1.0, m) * k * 2.0 ** -30
    if kind == "ratio":         # quotients over the whole exponent range of the fixed-point form
        return (1.0 + rng.random(m)) * k, (1.0 + rng.random(m)) * k * np.ldexp(1.0, rng.integers(-402, 403, m))
    if kind == "range":         # magnitudes about the form's limits 2^-450 and 2^450
        e = rng.choice([-452, -451, -450, -449, 448, 449, 450, 451], m)
        return (1.0 + rng.random(m)) * np.ldexp(1.0, e), (1.0 + rng.random(m)) * np.ldexp(1.0, e + rng.integers(-30, 1, m))
    f, g = rng.standard_normal(m), rng.standard_normal(m)   # special values among ordinary ones
    sp = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.0 ** -1030, 2.0 ** 1023, 1.0])
    f[::2] = sp[rng.integers(0, len(sp), len(f[::2]))]
    g[::3] = sp[rng.integers(0, len(sp), len(g[::3]))]
    return f, g


@pytest.mark.parametrize("kind", ["square", "power", "equal", "midpoint", "ratio", "range", "special"])
def test_fixed_point_rotation_matches_oracle(cuda, pkg, oracle, kind):
    rng = np.random.default_rng(11)
    f, g = pairs(kind, rng)
    f = np.where(rng.random(f.size) < 0.5, -f, f)
    g = np.where(rng.random(g.size) < 0.5, -g, g)
    got = np.stack(pkg.get_rotation(f, g), axis=1)
    want = np.array([oracle.givens(float(a), float(b)) for a, b in zip(f, g)])
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(np.where(nan, 0.0, got).view(np.uint64), np.where(nan, 0.0, want).view(np.uint64))
