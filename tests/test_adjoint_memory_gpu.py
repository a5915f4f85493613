"""The planes of the sliced adjoint of a large matrix go back to the device after the call: the handle keeps M and
the partial sums (8 bytes an element and a little), whether the matrix took the slices or not."""
from __future__ import annotations

import math

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("localized", [False, True])
def test_large_planes_are_given_back(cuda, pkg, localized):
    n = 9600
    if cuda.cuda.mem_get_info()[0] < 16 << 30:
        pytest.skip("needs 16 GB of device memory")
    f64 = dict(dtype=cuda.float64, device="cuda")
    j = cuda.arange(1, n + 1, **f64)
    if localized:
        lam, Q = j, cuda.eye(n, **f64)
    else:
        lam, Q = 2 * cuda.cos(j * (math.pi / (n + 1))), cuda.sin(cuda.outer(j, j) * (math.pi / (n + 1))) * math.sqrt(2 / (n + 1))
    glam, gQ = cuda.ones(n, **f64), cuda.ones(n, n, **f64)
    h = pkg.Handle(0)
    cuda.cuda.synchronize()
    cuda.cuda.empty_cache()
    before = cuda.cuda.mem_get_info()[0]
    gd, ge = pkg.eig_adjoint(lam, Q.T, glam, gQ.T, handle=h)
    assert bool(cuda.isfinite(gd).all()) and h.adjoint_sliced() == (0 if localized else 1)
    cuda.cuda.synchronize()
    cuda.cuda.empty_cache()
    assert before - cuda.cuda.mem_get_info()[0] < 1.2 * 8 * n * n
    h.close()
