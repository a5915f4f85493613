"""The batched chase four matrices to a CTA (from 153 matrices on; one to a CTA below): every matrix of small
batches about that count and about a full last CTA, bit for bit the single solve's."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [152, 153, 154, 155, 156, 157])
def test_batched_chase_by_four(cuda, pkg, count):
    rng = np.random.default_rng(count)
    sizes = rng.integers(1, 25, size=count)
    ds, es = [rng.standard_normal(n) for n in sizes], [rng.random(n - 1) for n in sizes]
    d, e, Q = np.concatenate(ds), np.concatenate(es), np.concatenate([np.eye(n).ravel() for n in sizes])
    h = pkg.Handle(0)
    conv, iters = pkg.qr_algorithm_batched_(d, e, sizes, Q, handle=h)
    i = j = q = 0
    for k, n in enumerate(sizes):
        H, Q1 = pkg.SymTridiagonal(ds[k].copy(), es[k].copy()), np.asfortranarray(np.eye(n))
        _, c1, it1 = pkg.qr_algorithm_(H, Q1, handle=h)
        assert (conv[k], iters[k]) == (c1, it1), k
        assert np.array_equal(d[i:i + n], H.dv) and np.array_equal(e[j:j + n - 1], H.ev), k
        assert np.array_equal(Q[q:q + n * n].reshape(n, n, order="F"), Q1), k
        i, j, q = i + n, j + n - 1, q + n * n
    h.close()
