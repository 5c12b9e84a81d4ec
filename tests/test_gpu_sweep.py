"""The one-launch triangular sweep (128-row FP32 / 64-row FP64 blocks, solutions polled in
place): every mode (unit lower, lower, upper, transposed lower), block edges, one and several
right-hand sides, groups of 8 and their remainder, the inverted-diagonal form through the
mixed solvers, and NaN and infinity in the right-hand side."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _resid_ok(t, x, b, eps):
    """Componentwise backward error of a substitution, |b - T x| <= 2 n eps |T||x|."""
    n = t.shape[0]
    t, x, b = t.astype(np.longdouble), x.astype(np.longdouble), b.astype(np.longdouble)
    return (np.abs(b - t @ x) <= 2 * n * eps * (np.abs(t) @ np.abs(x)) + 1e-300).all()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,nrhs", [(1, 1), (63, 1), (64, 2), (65, 1), (127, 3), (128, 1), (129, 8), (513, 9),
                                    (641, 1), (1000, 16), (1025, 17), (700, 128)])
def test_lower_and_upper(gpu, dtype, n, nrhs):
    rng = np.random.default_rng(n + nrhs)
    t = (rng.uniform(-1, 1, (n, n)) / np.sqrt(n) + 2 * np.eye(n)).astype(dtype)
    b = rng.standard_normal((n, nrhs)).astype(dtype)
    eps = np.finfo(dtype).eps
    assert _resid_ok(np.tril(t), gpu.solve_l_triangular(t, b), b, eps)
    assert _resid_ok(np.triu(t), gpu.solve_u_triangular(t, b), b, eps)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,nrhs", [(513, 1), (577, 8), (900, 11)])
def test_unit_lower_and_transposed(gpu, dtype, n, nrhs):
    """LU (unit lower, upper) and Cholesky (lower, its transpose) solves: normwise backward
    error of the whole solve within 4 n eps."""
    rng = np.random.default_rng(n)
    eps = np.finfo(dtype).eps
    b = rng.standard_normal((n, nrhs)).astype(dtype)
    a = (rng.uniform(-1, 1, (n, n)) + np.eye(n)).astype(dtype)
    g = rng.standard_normal((n, n))
    s = (g @ g.T / n + np.eye(n)).astype(dtype)
    for m, x in ((a, gpu.PartialPivLu.decompose(a).solve(b)), (s, gpu.Cholesky.decompose(s).solve(b))):
        r = np.abs(b - m.astype(np.float64) @ x.astype(np.float64)).max(axis=0)
        den = np.abs(m).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0)
        assert (r <= 4 * n * eps * den).all()


@pytest.mark.parametrize("n,nrhs", [(513, 1), (640, 3), (769, 1), (1100, 64), (1281, 100)])
def test_inverted_diagonal_form(gpu, n, nrhs):
    rng = np.random.default_rng(n)
    b = rng.standard_normal((n, nrhs))
    a = rng.uniform(-1, 1, (n, n)) + np.eye(n) * 4
    g = rng.standard_normal((n, n))
    s = g @ g.T + n * np.eye(n)
    for m, kind in ((a, "lu"), (s, "cholesky")):
        x, info = gpu.solve_mixed(m, b, kind)
        assert info["path"] == "refinement" and info["berr"] <= 10 * n * 2.0 ** -53
        r = np.abs(b - m @ x).max(axis=0) / (np.abs(m).sum(axis=1).max() * np.abs(x).max(axis=0))
        assert (r <= 10 * n * 2.0 ** -53).all()


def test_lstsq_uses_sweeps(gpu):
    rng = np.random.default_rng(4)
    a, b = rng.standard_normal((1300, 600)), rng.standard_normal(1300)
    x, info = gpu.lstsq_mixed(a, b)
    want = np.linalg.lstsq(a, b, rcond=None)[0]
    assert info["path"] == "refinement" and np.linalg.norm(x - want) <= 1e-12 * np.linalg.norm(want)


def test_non_finite_right_hand_side(gpu):
    """A NaN or infinity reaches the blocks that depend on it and the sweep ends."""
    n = 700
    rng = np.random.default_rng(6)
    t = np.tril(rng.uniform(-1, 1, (n, n))) / n + np.eye(n)
    b = rng.standard_normal((n, 2))
    b[300, 0], b[500, 1] = np.nan, np.inf
    x = gpu.solve_l_triangular(t, b)
    assert np.isfinite(x[:300, 0]).all() and np.isnan(x[300:, 0]).all()
    assert np.isfinite(x[:500, 1]).all() and not np.isfinite(x[500:, 1]).any()
