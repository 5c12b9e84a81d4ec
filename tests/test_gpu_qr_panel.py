"""The one-exchange cluster Householder panel against the cooperative-grid form (which takes
sigma and u in two passes): same reflectors within rounding, for few and many rows per CTA,
partial blocks, zero and already reduced columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 2), (33, 17), (64, 64), (100, 64), (130, 65), (1000, 70), (1201, 130),
                                 (2600, 40), (5000, 33)])
def test_against_cooperative_form(gpu, dtype, m, n):
    from rulinalg_gb300 import _lib as L
    rng = np.random.default_rng(m + n)
    a = rng.standard_normal((m, n)).astype(dtype)
    if n > 20:
        a[:, 3] = 0                       # zero column
        a[:, 9], a[9, 9] = 0, -2          # zero below and above the diagonal
        a[:, 17] = a[:, 16]               # a repeated column: zero below the diagonal up to rounding
    h = gpu.HouseholderQr.decompose(a)
    saved = gpu.tune_get(L.TUNE_PANEL_CLUSTER_MAX)
    try:
        gpu.tune_set(L.TUNE_PANEL_CLUSTER_MAX, 0)
        c = gpu.HouseholderQr.decompose(a)
    finally:
        gpu.tune_set(L.TUNE_PANEL_CLUSTER_MAX, saved)
    eps = np.finfo(dtype).eps
    assert h.tau[3:4].tolist() == [0.0] * len(h.tau[3:4]) if n > 20 else True
    # R up to column 16 is determined to rounding; the whole factorisation by its residual
    k = min(m, n, 17)
    assert np.linalg.norm(np.triu(h.qr)[:k, :k] - np.triu(c.qr)[:k, :k]) <= 8 * m * eps * np.linalg.norm(a)
    t = h.unpack_thin()
    q, r = t.q1.astype(np.float64), t.r1.astype(np.float64)
    assert np.linalg.norm(q @ r - a) <= 2 * np.sqrt(m) * n * eps * np.linalg.norm(a)
    assert np.linalg.norm(q.T @ q - np.eye(q.shape[1])) <= 2 * np.sqrt(m) * n * eps
