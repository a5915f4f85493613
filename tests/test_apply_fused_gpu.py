"""The fused-wave apply against the oracle, bit for bit: every (layer groups, layers per group) its
rule picks, layers on each side of the padding, passes and rounds of CTAs, and matrices of fewer
columns than the groups' lag."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rotation_grid, to_device_colmajor

pytestmark = pytest.mark.gpu


def check(pkg, oracle, torch, m, n, k, dtype, seed=0):
    rng = np.random.default_rng(seed + m + 7 * n + 13 * k)
    A = np.asfortranarray((rng.random((m, n)) * 2 - 1).astype(dtype))
    A[:, ::5] = 0.0          # signed zeros and an exact identity column are common in a solve
    g = rotation_grid(pkg, rng, n, k, dtype)
    g[::3, ::2] = (1.0, 0.0)
    ref = A.copy(order="F")
    oracle.apply_seq(ref, g)
    dA = to_device_colmajor(torch, A)
    pkg.bulk_wave_order_2x2_rmul_(dA, torch.from_numpy(np.ascontiguousarray(g.transpose(1, 0, 2))).cuda().permute(1, 0, 2))
    got = dA.cpu().numpy()
    assert np.array_equal(got, ref), (m, n, k, dtype, int(np.sum(got != ref)))


# rows of one, a few and many warps per SM, the last ones in two and three rounds of CTAs
@pytest.mark.parametrize("m", [1, 153, 700, 2500, 4200, 6200, 9100, 17000])
@pytest.mark.parametrize("k", [1, 9, 32, 33, 64, 100, 129, 257])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_rows_and_layers(cuda, pkg, oracle, m, k, dtype):
    check(pkg, oracle, cuda, m, 23, k, dtype)


@pytest.mark.parametrize("n", [2, 3, 4, 9, 10, 11, 64, 200, 331])
@pytest.mark.parametrize("k", [2, 20, 48, 128])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_columns(cuda, pkg, oracle, n, k, dtype):
    check(pkg, oracle, cuda, 97, n, k, dtype)


@pytest.mark.parametrize("k", [16, 40, 64])
@pytest.mark.parametrize("m,n", [(4096, 30), (4300, 257), (9000, 65)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_column_segments(cuda, pkg, oracle, m, n, k, dtype):
    """The host-pointer apply, streamed by column segments."""
    rng = np.random.default_rng(m + n + k)
    A = np.asfortranarray((rng.random((m, n)) * 2 - 1).astype(dtype))
    g = rotation_grid(pkg, rng, n, k, dtype)
    ref = A.copy(order="F")
    oracle.apply_seq(ref, g)
    pkg.bulk_wave_order_2x2_rmul_(A, g)
    assert np.array_equal(A, ref)


@pytest.mark.parametrize("m,n,k", [(60, 2500, 40), (301, 97, 128)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_row_rotations(cuda, pkg, oracle, m, n, k, dtype):
    """lmul!: the same tile on the transposed view."""
    rng = np.random.default_rng(m + n + k)
    A = np.asfortranarray((rng.random((m, n)) * 2 - 1).astype(dtype))
    g = rotation_grid(pkg, rng, m, k, dtype)
    ref = np.asfortranarray(A.T.copy())
    oracle.apply_seq(ref, g)
    dA = to_device_colmajor(cuda, A)
    pkg.bulk_wave_order_2x2_lmul_(dA, cuda.from_numpy(np.ascontiguousarray(g.transpose(1, 0, 2))).cuda().permute(1, 0, 2))
    assert np.array_equal(dA.cpu().numpy(), ref.T)
