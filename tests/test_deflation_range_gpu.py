"""The deflation scan at the ends of the FP64 range, where |d_j| + |d_j+1| overflows, an entry is infinite or the
tolerance is: is_offdiagonal_small (src/bulge_chasing.jl:7-8) holds there for every finite off-diagonal, and
the chase has to deflate where the oracle does.  Same bits, for the single and the batched chase."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def problem(kind):
    rng = np.random.default_rng(3)
    n, tol = 12, np.finfo(np.float64).eps
    d, e = rng.standard_normal(n), rng.random(n - 1)
    if kind == "sum":           # finite, but their sum is not
        d[4:6], e[4] = [1.5 * 2.0 ** 1023, -1.75 * 2.0 ** 1023], 2.0 ** 1000
    elif kind == "infinite":
        d[5], e[4], e[5] = np.inf, 2.0 ** 1000, -2.0 ** 1023
    else:                       # an infinite tolerance deflates everything
        d, e, tol = d * 2.0 ** -1000, e * 2.0 ** 30, np.inf
    return d, e, tol


@pytest.mark.parametrize("kind", ["sum", "infinite", "tolerance"])
def test_deflation_at_the_ends_of_the_range(cuda, pkg, oracle, kind):
    d, e, tol = problem(kind)
    n = d.size
    od, oe, oQ = d.copy(), e.copy(), np.asfortranarray(np.eye(n))
    conv_o, it_o, _, _ = oracle.qr_algorithm(od, oe, oQ, tol=tol)
    assert conv_o and np.isfinite(oQ).all()
    for mode in (0, 1, 2):
        H, Q = pkg.SymTridiagonal(d.copy(), e.copy()), np.asfortranarray(np.eye(n))
        _, conv, it = pkg.qr_algorithm_(H, Q, tol=tol, chase_mode=mode)
        assert (conv, it) == (conv_o, it_o), mode
        assert np.array_equal(H.dv, od) and np.array_equal(H.ev, oe) and np.array_equal(Q, oQ), mode
    bd, be, bQ = d.copy(), e.copy(), np.eye(n).ravel()
    conv, it = pkg.qr_algorithm_batched_(bd, be, [n], bQ, tol=tol)
    assert (conv[0], it[0]) == (conv_o, it_o)
    assert np.array_equal(bd, od) and np.array_equal(be, oe) and np.array_equal(bQ.reshape(n, n, order="F"), oQ)
