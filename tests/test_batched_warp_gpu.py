"""The batched chase (one warp per matrix, four to a CTA) against the single-matrix path, bit for
bit: counts that do not fill a CTA, the smallest orders, both rotation placements, layer
buffers of a few layers, and a batch that hits its iteration limit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,exact,max_layers,factor", [
    ([2], True, 128, 100), ([1, 2, 3], True, 128, 100), ([33, 2, 64, 31, 32], True, 128, 100),
    ([40, 41, 97, 5], False, 128, 100), ([65, 130, 17], False, 3, 100), ([65, 130, 17], True, 3, 100),
    ([50, 20, 90], True, 128, 1)])
def test_batched_chase_is_the_single_chase(cuda, pkg, sizes, exact, max_layers, factor):
    rng = np.random.default_rng(len(sizes) + sum(sizes))
    h = pkg.Handle(0)
    ds = [rng.random(n) if k % 2 else rng.standard_normal(n) for k, n in enumerate(sizes)]
    es = [rng.random(n - 1) * (1.0 if k % 3 else 1e-3) for k, n in enumerate(sizes)]
    d, e = np.concatenate(ds), np.concatenate(es)
    Q = np.concatenate([np.eye(n).ravel() for n in sizes])
    h.set_exact_order(exact)
    conv, iters = pkg.qr_algorithm_batched_(d, e, sizes, Q, max_layers=max_layers, maxiter_factor=factor, handle=h)
    h.set_exact_order(True)
    i = j = q = 0
    for k, n in enumerate(sizes):
        H, Q1 = pkg.SymTridiagonal(ds[k].copy(), es[k].copy()), np.asfortranarray(np.eye(n))
        _, c1, it1 = pkg.qr_algorithm_(H, Q1, max_layers=max_layers, maxiter=factor * n, exact_order=exact, handle=h)
        assert (conv[k], iters[k]) == (c1, it1)
        assert np.array_equal(d[i:i + n], H.dv) and np.array_equal(e[j:j + n - 1], H.ev)
        assert np.array_equal(Q[q:q + n * n].reshape(n, n, order="F"), Q1)
        i, j, q = i + n, j + n - 1, q + n * n
    h.close()
