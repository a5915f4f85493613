"""The bulges' hand-over in chunks of release_every steps (fetch, sweep and store warps): results
do not depend on the chunk, for blocks of fewer steps than a chunk, one more or less than a
multiple, both placements and batches of two to many bulges."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bulges,rows,exact", [(9, 2, 4, True), (33, 8, 4, True), (34, 8, 4, False),
                                                 (65, 16, 4, True), (129, 2, 16, True), (258, 64, 4, False)])
def test_chunks_do_not_change_the_bits(cuda, pkg, n, bulges, rows, exact):
    rng = np.random.default_rng(n)
    d, e = rng.standard_normal(n), rng.random(n - 1)
    ref = None
    for every in (1, 2, 4, 16, 64):
        h = pkg.Handle(0)
        h.set_multishift(bulges, rows, every)
        H, Q = pkg.SymTridiagonal(d.copy(), e.copy()), np.asfortranarray(np.eye(n))
        _, conv, it = pkg.qr_algorithm_(H, Q, chase_mode=3, exact_order=exact, handle=h)
        assert conv and h.stats()["bulge_batches"] > 0
        got = (it, H.dv, H.ev, Q)
        ref = ref or got
        assert it == ref[0] and all(np.array_equal(a, b) for a, b in zip(got[1:], ref[1:])), every
        h.close()
    eps = np.finfo(np.float64).eps
    T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    lam = np.linalg.eigvalsh(T)
    assert np.max(np.abs(np.sort(ref[1]) - lam)) <= 10 * n * eps * np.max(np.abs(lam))
