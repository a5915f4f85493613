"""Which products the adjoint takes (symeig_adjoint_sliced), and what it does when a bounded wait of the sliced
products runs out: the copies stop on purpose (symeig_set_test_stall), the waits give up after about a
second, the FP64 MMA does the work and the call reports SYMEIG_ERR_TIMEOUT.  No GPU fault: every
wait is bounded and nothing else changes."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import test_adjoint_blocks_gpu as blocks
import test_adjoint_sliced_gpu as plain

pytestmark = pytest.mark.gpu

SYMEIG_ERR_TIMEOUT = -3


def chain(n, seed=0):
    rng = np.random.default_rng(n + seed)
    lam, Q = blocks.toeplitz(n, rng, 0.3, 0.9)
    return lam, Q, rng.standard_normal(n), rng.standard_normal((n, n))


def adjoint(cuda, pkg, h, lam, Q, glam, gQ):
    col = lambda x: cuda.tensor(np.ascontiguousarray(np.swapaxes(x, -1, -2)), device="cuda").transpose(-1, -2)  # noqa: E731
    gd, ge = pkg.eig_adjoint(cuda.tensor(lam, device="cuda"), col(Q), cuda.tensor(glam, device="cuda"), col(gQ), handle=h)
    return gd.cpu().numpy(), ge.cpu().numpy()


@pytest.mark.parametrize("problem,sliced", [
    (lambda: chain(255), 0), (lambda: chain(256), 1), (lambda: chain(257), 1), (lambda: chain(512), 1), (lambda: chain(1100), 1),
    (lambda: plain.problem(320, 1, "plain"), 1), (lambda: plain.problem(320, 1, "localized"), 0),
    (lambda: blocks.problem("shift", 150, 150, 1e-10), 0), (lambda: blocks.problem("mirror", 150, 150, 0.0), 0),
    (lambda: blocks.problem("rows", 150, 140, 1e6), 0), (lambda: blocks.problem("rows", 200, 200, 1e20), 0)])
def test_route(cuda, pkg, problem, sliced):
    h = pkg.Handle(0)
    adjoint(cuda, pkg, h, *problem())
    assert h.adjoint_sliced() == sliced
    h.close()


def test_sliced_wait_timeout_is_reported(cuda, pkg):
    lib, h = pkg.load_library(), pkg.Handle(0)
    lam, Q, glam, gQ = chain(300)
    Qf, gf = np.asfortranarray(Q), np.asfortranarray(gQ)
    gd, ge = np.empty(300), np.empty(299)
    args = [ctypes.c_void_p(x.ctypes.data) for x in (lam, Qf, glam, gf, gd, ge)]
    assert lib.symeig_eig_adjoint_f64(h.ptr, 1, 300, *args) == 0 and h.adjoint_sliced() == 1
    assert h.stats()["device_errors"] == 0
    assert lib.symeig_set_test_stall(h.ptr, 3) == 0
    assert lib.symeig_eig_adjoint_f64(h.ptr, 1, 300, *args) == SYMEIG_ERR_TIMEOUT
    assert h.stats()["device_errors"] == 1 and h.adjoint_sliced() == 0
    rd, re, td, te = blocks.reference(lam, Q, glam, gQ)
    assert (np.abs(gd - rd) <= td).all() and (np.abs(ge - re) <= te).all()
    assert lib.symeig_set_test_stall(h.ptr, 0) == 0
    assert lib.symeig_eig_adjoint_f64(h.ptr, 1, 300, *args) == 0 and h.adjoint_sliced() == 1
    assert h.stats()["device_errors"] == 0
    h.close()
