"""The adjoint's products by bf16 slices (orders from 256): edges of the 128-wide tiles and of the
64-deep steps, batches beside single matrices, operands that fall back to the FP64 MMA.

Tolerance: with u = 2^-53 a length-n FP64 product x.y is off by at most n u |x| |y| (2-norms) in either
implementation, and the sliced one by less.  So G = Q^T gQ is off by n u |q_i| |g_j|, M by that over the
gap, P = Q M by n u |Q_i| |m_k| plus |Q| times M's, and the gradients by |P's| |Q|^T plus their own
sums of n terms.  Twice for the two sides, twice for the two gradient entries of an off-diagonal."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def problem(n, seed, kind):
    rng = np.random.default_rng(seed)
    if kind == "localized":     # a banded orthogonal factor: n - 1 plane rotations of the identity
        Q = np.eye(n)
        for i in range(n - 1):
            c, s = np.cos(th := rng.random()), np.sin(th)
            Q[:, i:i + 2] = Q[:, i:i + 2] @ np.array([[c, s], [-s, c]])
    else:
        Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    gQ = rng.standard_normal((n, n))
    if kind == "graded":
        gQ *= np.exp(20 * rng.standard_normal(n))[None, :]
        gQ[:, n // 2] = 0.0
    return rng.standard_normal(n), Q, rng.standard_normal(n), gQ


def reference(lam, Q, glam, gQ):
    n = lam.size
    gap = lam[None, :] - lam[:, None]
    np.fill_diagonal(gap, 1.0)
    M = (Q.T @ gQ) / gap
    np.fill_diagonal(M, glam)
    A = Q @ M @ Q.T
    norm = lambda X, axis: np.sqrt((X * X).sum(axis))  # noqa: E731
    eM = n * U * np.outer(norm(Q, 0), norm(gQ, 0)) / np.abs(gap)
    eP = n * U * np.outer(norm(Q, 1), norm(M, 0)) + np.abs(Q) @ eM
    eA = 4 * (eP @ np.abs(Q).T + n * U * np.abs(Q @ M) @ np.abs(Q).T)
    tol_e = np.diag(eA, 1) + np.diag(eA, -1)
    return np.diag(A), np.diag(A, 1) + np.diag(A, -1), np.diag(eA), tol_e


def run(torch, pkg, lam, Q, glam, gQ):
    dev = lambda x: torch.tensor(x, device="cuda")  # noqa: E731
    col = lambda x: dev(np.ascontiguousarray(np.swapaxes(x, -1, -2))).transpose(-1, -2)  # noqa: E731
    gd, ge = pkg.eig_adjoint(dev(lam), col(Q), dev(glam), col(gQ))
    return gd.cpu().numpy(), ge.cpu().numpy()


@pytest.mark.parametrize("n,kind", [(255, "plain"), (256, "plain"), (257, "plain"), (287, "graded"),
                                    (289, "plain"), (320, "localized"), (321, "graded"),
                                    (384, "plain"), (385, "localized"), (511, "graded")])
def test_sliced_adjoint(cuda, pkg, n, kind):
    lam, Q, glam, gQ = problem(n, n, kind)
    gd, ge = run(cuda, pkg, lam, Q, glam, gQ)
    rd, re, td, te = reference(lam, Q, glam, gQ)
    assert (np.abs(gd - rd) <= td).all(), np.max(np.abs(gd - rd) / td)
    assert (np.abs(ge - re) <= te).all(), np.max(np.abs(ge - re) / te)
    # the gradient is linear: exact under a power of two
    sd, se = run(cuda, pkg, lam, Q, glam * 2.0 ** 300, gQ * 2.0 ** 300)
    assert np.array_equal(sd, gd * 2.0 ** 300) and np.array_equal(se, ge * 2.0 ** 300)


@pytest.mark.parametrize("n,bits,signed", [(300, 9, True), (513, 8, True), (1100, 6, True), (700, 4, False)])
def test_sliced_adjoint_integers(cuda, pkg, n, bits, signed):
    """Integer Q and gQ with gaps of 0 and +-1: every product and sum is an integer below 2^53, so the
    gradient is exact, whatever the order of its sums."""
    rng = np.random.default_rng(n)
    top = 2 ** bits
    ints = lambda: rng.integers(-top + 1 if signed else 1, top, (n, n))  # noqa: E731
    Q, gQ, glam = ints(), ints(), rng.integers(-9, 10, n)
    lam = (rng.random(n) < 0.5).astype(np.int64)
    M = (Q.T @ gQ) * (lam[None, :] - lam[:, None])
    np.fill_diagonal(M, glam)
    P = Q @ M
    assert (np.abs(P) @ np.abs(Q).max(axis=0)).max() < 2 ** 52
    f = lambda x: x.astype(np.float64)  # noqa: E731
    gd, ge = run(cuda, pkg, f(lam), f(Q), f(glam), f(gQ))
    assert np.array_equal(gd, (P * Q).sum(1))
    assert np.array_equal(ge, (P[:-1] * Q[1:]).sum(1) + (P[1:] * Q[:-1]).sum(1))


def test_sliced_adjoint_batch(cuda, pkg):
    """Each matrix of a batch takes its own path: the same bits as alone, beside an infinity."""
    n = 300
    ps = [problem(n, 7 + i, k) for i, k in enumerate(["plain", "localized", "plain", "graded"])]
    ps[2][3][5, 9] = np.inf
    gd, ge = run(cuda, pkg, *(np.stack(x) for x in zip(*ps)))
    for i, p in enumerate(ps):
        sd, se = run(cuda, pkg, *p)
        assert np.array_equal(sd, gd[i], equal_nan=True) and np.array_equal(se, ge[i], equal_nan=True)
        assert np.isfinite(sd).all() == (i != 2)
