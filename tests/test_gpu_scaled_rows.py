"""Substitutions scale a diagonal block by its reciprocal diagonal; entries that this would take out
of the normal range (overflow, or subnormal with fewer bits) are substituted as they are. Triangles
whose rows mix scales, in the sweep and in the one-launch solve of up to 64 rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _triangle(n, dtype, kind):
    """Upper triangle with a last column that overflows / underflows against the other rows'
    diagonal, and b = T x for x of ones and a last entry that brings the products back to scale."""
    big, tiny = (1e36, 1e-43) if dtype == np.float32 else (1e305, 1e-320)
    t = np.triu(np.full((n, n), 0.125)) + np.eye(n)
    x = np.ones(n)
    if kind == "overflow":
        t[: n - 1] *= 2.0 ** -20
        t[: n - 1, n - 1] = big
        x[n - 1] = 1.0 / big
    else:  # t_ij / t_ii of about `tiny`
        t[: n - 1] *= 2.0 ** 60
        t[: n - 1, n - 1] = tiny * 2.0 ** 60
        x[n - 1] = 1e300 if dtype == np.float64 else 1e38
        x[: n - 1] = 0
    with np.errstate(over="ignore"):
        t = t.astype(dtype)
        b = (t.astype(np.longdouble) @ x.astype(dtype).astype(np.longdouble)).astype(dtype)
    return t, b


def _ok(t, x, b):
    n, eps = t.shape[0], np.finfo(t.dtype).eps
    t, x, b = t.astype(np.longdouble), x.astype(np.longdouble), b.astype(np.longdouble)
    return np.isfinite(x).all() and (np.abs(b - t @ x) <= 2 * n * eps * (np.abs(t) @ np.abs(x))).all()


@pytest.mark.parametrize("kind", ["overflow", "underflow"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [5, 33, 64, 65, 128, 200])
def test_rows_of_mixed_scale(gpu, kind, dtype, n):
    t, b = _triangle(n, dtype, kind)
    assert _ok(t, gpu.solve_u_triangular(t, b), b)
    many = np.stack([b, 2 * b, b / 2], axis=1)
    x = gpu.solve_u_triangular(t, many)
    for c in range(3):
        assert _ok(t, x[:, c], many[:, c])
    low = np.ascontiguousarray(t[::-1, ::-1])  # the same system from the last unknown on
    assert _ok(low, gpu.solve_l_triangular(low, b[::-1].copy()), b[::-1])
    assert _ok(t, gpu.solve(t, b), b)
