"""sytrd and orgtr at the edges of their blocks (32-row blocks, 64-column panels, 16-column T
blocks) and where the product's column chunk and the split of the inner sums change (2048 and
4096): the factorisation itself, to the backward-error bound 10 n eps."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 31, 33, 64, 65, 66, 81, 129, 160, 2050, 4100])
def test_factorisation(cuda, pkg, n):
    torch = cuda
    X = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    A = (X + X.T) * 0.5
    W = A.clone().T
    d, e, tau = pkg.sytrd_(W)
    Q = pkg.orgtr(W, tau)
    eps = float(np.finfo(np.float64).eps)
    QT = Q * d[None, :]
    QT[:, :-1] += Q[:, 1:] * e[None, :]
    QT[:, 1:] += Q[:, :-1] * e[None, :]
    assert float(torch.linalg.norm(A @ Q - QT)) <= 10 * n * eps * float(torch.linalg.norm(A))
    G = Q.T @ Q
    G.diagonal().sub_(1.0)
    assert float(torch.linalg.norm(G)) <= 10 * n * eps
    assert torch.equal(W.diagonal(), d) and torch.equal(W.diagonal(-1), e)


def test_repeated_calls_are_identical(cuda, pkg):
    torch = cuda
    X = torch.randn(300, 300, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    A = (X + X.T) * 0.5
    out = []
    for _ in range(2):
        W = A.clone().T
        d, e, tau = pkg.sytrd_(W)
        out.append((d, e, tau, W, pkg.orgtr(W, tau)))
    assert all(torch.equal(a, b) for a, b in zip(*out))
