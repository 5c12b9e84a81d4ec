"""Householder blocks: the small-tile products, Q's leading columns around the 64-reflector
block edges (V^T Q2 taken from V where Q2 is still the identity), reflectors with tau = 0 in
the block T factor, and the split update of the unit-triangular rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (15, 31, 17), (16, 32, 16), (33, 33, 31), (64, 64, 435), (64, 512, 64),
                                   (65, 511, 70), (130, 97, 2), (3, 512, 700)])
def test_few_output_products(gpu, dtype, m, k, n):
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((m, k)).astype(dtype), rng.standard_normal((k, n)).astype(dtype)
    want = a.astype(np.longdouble) @ b.astype(np.longdouble)
    bound = k * np.finfo(dtype).eps * (np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)) + 1e-300
    assert (np.abs(gpu.mat_mul(a, b) - want) <= bound).all()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("m,n,k", [(70, 63, 63), (200, 64, 64), (200, 65, 65), (200, 65, 200), (300, 129, 100),
                                   (300, 129, 300), (130, 200, 130), (700, 320, 320), (900, 500, 900)])
def test_first_k_columns(gpu, dtype, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a = rng.standard_normal((m, n)).astype(dtype)
    a[:, 5] = 0  # a zero column: tau = 0 in the first block
    h = gpu.HouseholderQr.decompose(a)
    q = h.first_k_columns(k).astype(np.float64)
    eps = np.finfo(dtype).eps
    assert np.linalg.norm(q.T @ q - np.eye(k)) <= 4 * m * eps
    full = np.eye(m, dtype=dtype)
    h.q().left_multiply_into(full)  # the same columns through the general application of Q
    assert np.linalg.norm(q - full[:, :k]) <= 4 * m * eps * np.sqrt(k)
    p = min(m, n, k)
    r = np.triu(h.qr)[:p].astype(np.float64)
    if p == min(m, n):
        assert np.linalg.norm(q[:, :p] @ r - a) <= 4 * m * eps * np.linalg.norm(a)
