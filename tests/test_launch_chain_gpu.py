"""Chains of dependent launches (launch_after.cuh): calls repeated back to back on the same inputs give the same
bits, and the first ones are right, whatever overlaps what."""
from __future__ import annotations

import numpy as np
import pytest

import test_adjoint_blocks_gpu as blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 65, 130, 257, 700])
def test_dense_reduction_repeats(cuda, pkg, n):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, n))
    A0 = cuda.tensor(X + X.T, device="cuda")
    out = []
    for _ in range(6):
        A = A0.clone().T
        d, e, tau = pkg.sytrd_(A)
        out.append([x.cpu().numpy() for x in (d, e, tau, pkg.orgtr(A, tau))])
    d, e, _, Q = out[0]
    T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    assert np.linalg.norm(Q @ T @ Q.T - (X + X.T)) <= 10 * n * 2.0 ** -52 * np.linalg.norm(X + X.T)
    for o in out[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(o, out[0]))


def test_adjoint_groups(cuda, pkg):
    """Four groups of planes with matrices that fall back among them: each has its bits alone."""
    n, count = 512, 160
    gen = cuda.Generator(device="cuda")
    gen.manual_seed(n * 7 + count)
    rnd = lambda *s: cuda.randn(*s, generator=gen, dtype=cuda.float64, device="cuda")  # noqa: E731
    Q, lam, glam, gQ = (rnd(count, n, n) / n ** 0.5).transpose(1, 2), rnd(count, n), rnd(count, n), rnd(count, n, n).transpose(1, 2)
    h = pkg.Handle(0)
    runs = [pkg.eig_adjoint(lam, Q, glam, gQ, handle=h) for _ in range(3)]
    assert 0 < h.adjoint_sliced() < count
    for z in range(count):
        gd, ge = pkg.eig_adjoint(lam[z], Q[z], glam[z], gQ[z], handle=h)
        for bd, be in runs:
            assert cuda.equal(bd[z], gd) and cuda.equal(be[z], ge), z
    h.close()


@pytest.mark.parametrize("n", [256, 257, 300, 513])
def test_adjoint_repeats(cuda, pkg, n):
    rng = np.random.default_rng(n)
    lam, Q, glam, gQ = rng.standard_normal(n), np.linalg.qr(rng.standard_normal((n, n)))[0], rng.standard_normal(n), rng.standard_normal((n, n))
    col = lambda x: cuda.tensor(np.ascontiguousarray(x.T), device="cuda").T  # noqa: E731
    args = cuda.tensor(lam, device="cuda"), col(Q), cuda.tensor(glam, device="cuda"), col(gQ)
    out = [tuple(x.cpu().numpy() for x in pkg.eig_adjoint(*args)) for _ in range(8)]
    rd, re, td, te = blocks.reference(lam, Q, glam, gQ)
    for gd, ge in out:
        assert (np.abs(gd - rd) <= td).all() and (np.abs(ge - re) <= te).all()
        assert np.array_equal(gd, out[0][0]) and np.array_equal(ge, out[0][1])
