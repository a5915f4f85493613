"""The adjoint where zeros of Q meet peaks of gQ or of M: uncoupled and weakly coupled chains (what a zero or
tiny off-diagonal gives), with close eigenvalues across the chains or gradients of other sizes.  Q is spread
out, so that its norms alone do not keep it from the sliced products.

Tolerance: with u = 2^-53, entry by entry, a length-n FP64 product is off by at most n u |A| |B|.  So G = Q^T gQ
is off by n u |Q|^T |gQ|, M by that over the gap plus u |M|, P = Q M by |Q| times M's plus n u |Q| |M|, and
P Q^T by P's times |Q|^T plus n u |P| |Q|^T.  Twice for the two sides, with gradient entries of an off-diagonal the
sum of two."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def toeplitz(n, rng, a, b):
    j, jj = np.arange(1, n + 1), rng.permutation(n) + 1
    Q = np.sin(np.outer(j, jj) * (np.pi / (n + 1))) * np.where(rng.random(n) < 0.5, -1, 1) * np.sqrt(2 / (n + 1))
    return a + 2 * b * np.cos(jj * (np.pi / (n + 1))), Q


def problem(kind, n1, n2, value):
    rng = np.random.default_rng(n1 + n2)
    n = n1 + n2
    if kind == "mirror":        # a weakly disordered chain and its mirror image, couplings of `value` between them
        from scipy.linalg import eigh_tridiagonal
        d = 0.01 * rng.standard_normal(n1)
        lam, Q = eigh_tridiagonal(np.concatenate([d, d[::-1]]),
                                  np.concatenate([np.ones(n1 - 1), [value], np.ones(n1 - 1)]))
    else:
        (l1, q1), (l2, q2) = toeplitz(n1, rng, 0.3, 0.9), toeplitz(n2, rng, 0.3 + (value if kind == "shift" else 0.4), 0.9)
        lam, Q = np.concatenate([l1, l2]), np.zeros((n, n))
        Q[:n1, :n1], Q[n1:, n1:] = q1, q2
    gQ = rng.standard_normal((n, n))
    if kind == "rows":          # the loss sees the second chain's entries more
        gQ[n1:] *= value
    if kind == "columns":       # or its eigenvectors
        gQ[:, n1:] *= value
    return lam, Q, rng.standard_normal(n), gQ


def reference(lam, Q, glam, gQ):
    n = lam.size
    gap = lam[None, :] - lam[:, None]
    np.fill_diagonal(gap, 1.0)
    F = np.where(gap != 0, 1.0 / np.where(gap != 0, gap, 1.0), 0.0)
    M = F * (Q.T @ gQ)
    eM = n * U * np.abs(F) * (np.abs(Q).T @ np.abs(gQ)) + 2 * U * np.abs(M)
    np.fill_diagonal(M, glam)
    np.fill_diagonal(eM, 0.0)
    A = Q @ M @ Q.T
    aP = np.abs(Q) @ np.abs(M)
    eA = 2 * ((np.abs(Q) @ eM + 2 * n * U * aP) @ np.abs(Q).T)
    off = lambda X: np.diag(X, 1) + np.diag(X, -1)  # noqa: E731
    return np.diag(A), off(A), np.diag(eA), off(eA)


@pytest.mark.parametrize("kind,n1,n2,value", [
    ("shift", 150, 150, 1e-6), ("shift", 150, 150, 1e-10), ("shift", 150, 150, 1e-14), ("shift", 128, 129, 1e-12),
    ("shift", 257, 257, 1e-11), ("mirror", 150, 150, 0.0), ("mirror", 150, 150, 1e-9), ("mirror", 200, 200, 1e-13),
    ("rows", 150, 140, 1e6), ("rows", 200, 200, 1e20), ("columns", 150, 140, 1e6), ("columns", 200, 200, 1e20)])
def test_adjoint_of_blocks(cuda, pkg, kind, n1, n2, value):
    lam, Q, glam, gQ = problem(kind, n1, n2, value)
    n = n1 + n2
    assert all((n * (Q * Q).max(ax) <= 36 * (Q * Q).sum(ax)).all() for ax in (0, 1))
    col = lambda x: cuda.tensor(np.ascontiguousarray(x.T), device="cuda").T  # noqa: E731
    gd, ge = pkg.eig_adjoint(cuda.tensor(lam, device="cuda"), col(Q), cuda.tensor(glam, device="cuda"), col(gQ))
    rd, re, td, te = reference(lam, Q, glam, gQ)
    ed, ee = np.abs(gd.cpu().numpy() - rd) / td, np.abs(ge.cpu().numpy() - re) / te
    assert ed.max() <= 1 and ee.max() <= 1, (ed.max(), ee.max())
