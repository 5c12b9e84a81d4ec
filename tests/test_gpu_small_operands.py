"""Up to 64 rows: a failing solve leaves the caller's buffers as they were, the packed factors satisfy
P A = L U and A = L L^T componentwise, and the largest digits of the FP64 slices come out as meant."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 7, 20, 64])
def test_failing_solve_leaves_a_and_b(gpu, dtype, n):
    rng = np.random.default_rng(n)
    a, b = rng.uniform(-1, 1, (n, n + 3)).astype(dtype), rng.standard_normal(n).astype(dtype)
    a[:, n // 2] = 0  # the column beyond n // 2 is never reached, the rows' tails are not the solve's
    keep_a, keep_b = a.copy(), b.copy()
    fn, ptr = (gpu.lib.rl_smatrix_solve, C.POINTER(C.c_float)) if dtype == np.float32 else \
        (gpu.lib.rl_dmatrix_solve, C.POINTER(C.c_double))
    assert fn(n, a.ctypes.data_as(ptr), n + 3, b.ctypes.data_as(ptr)) != 0
    assert np.array_equal(a, keep_a) and np.array_equal(b, keep_b)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 2, 5, 16, 31, 33, 47, 63, 64])
def test_factors_componentwise(gpu, dtype, n):
    """|P A - L U| <= 2 n u |L||U|: n products, each multiplier and its correction rounded once."""
    rng = np.random.default_rng(n + 100)
    u = np.finfo(dtype).eps / 2
    a = (rng.uniform(-1, 1, (n, n)) * 2.0 ** rng.integers(-10, 10, (n, 1))).astype(dtype)
    parts = gpu.PartialPivLu.decompose(a).unpack()
    l, r = parts.l.astype(np.longdouble), parts.u.astype(np.longdouble)
    pa = np.empty_like(a)
    pa[parts.p.perm.astype(np.int64)] = a
    assert (np.abs(l @ r - pa) <= 2 * n * u * (np.abs(l) @ np.abs(r))).all()
    g = rng.standard_normal((n, n))
    s = (g @ g.T + n * np.eye(n)).astype(dtype)
    s = np.tril(s) + np.tril(s, -1).T
    f = gpu.Cholesky.decompose(s).unpack().astype(np.longdouble)
    assert (np.abs(f @ f.T - s) <= (2 * n + 4) * u * (np.abs(f) @ np.abs(f).T)).all()


def _cut(v):
    """The 8 balanced base-256 digits of v 2^63, |v| < 1, from the last one on."""
    y, out = int(Fraction(v) * 2 ** 63), []
    for _ in range(7):
        d = ((y + 128) & 255) - 128
        out.append(d)
        y = (y - d) >> 8
    return [y] + out[::-1]


@pytest.mark.parametrize("sign_b", [1, -1])
@pytest.mark.parametrize("first,rest", [(-127, -128), (127, 127)])
def test_digits_at_their_ends(gpu, first, rest, sign_b):
    """Every leading digit of every entry at the end of its range, products of one sign: the exact
    accumulators come as near to 5 x 192 x 2^14 as digits can."""
    mant = first * 256 ** 6 + rest * sum(256 ** t for t in range(6))
    v = float(Fraction(mant if rest == -128 else mant >> 2 << 2, 2 ** 55))
    assert abs(v) < 1 and _cut(v)[:6] == [first] + [rest] * 5
    k = 384
    c = gpu.mat_mul(np.full((260, k), v), np.full((k, 90), sign_b * v))
    want = Fraction(v) * Fraction(sign_b * v) * k
    lo, hi = Fraction(float(c.min())), Fraction(float(c.max()))
    assert abs(lo - want) <= abs(want) / 2 ** 52 and abs(hi - want) <= abs(want) / 2 ** 52


def _solution(a, b):
    """The solution to well beyond a's precision: FP64, refined twice with longer residuals."""
    a64, x = a.astype(np.float64), None
    inv = np.linalg.inv(a64)
    x = (inv @ b.astype(np.float64)).astype(np.longdouble)
    for _ in range(3):
        x = x + inv @ (b.astype(np.longdouble) - a.astype(np.longdouble) @ x).astype(np.float64)
    return x


@pytest.mark.parametrize("dtype,n,seeds,blocked", [(np.float64, 47, 40, 3.140e-16), (np.float64, 64, 40, 3.753e-16),
                                                   (np.float32, 47, 60, 1.671e-7), (np.float32, 64, 60, 2.034e-7)])
def test_forward_error_of_the_one_launch_solve(gpu, dtype, n, seeds, blocked):
    """Diagonally weighted systems: the geometric mean of the forward errors within 1.1 of that of the
    32-row blocked substitution (`blocked`, the same systems on the one-CTA kernels)."""
    logs = []
    for s in range(seeds):
        rng = np.random.default_rng(1000 * n + s)
        a = (rng.uniform(-1, 1, (n, n)) + n * np.eye(n)).astype(dtype)
        b = rng.standard_normal(n).astype(dtype)
        want = _solution(a, b)
        d = (gpu.solve(a, b).astype(np.longdouble) - want).astype(np.float64)
        logs.append(np.log(np.linalg.norm(d) / np.linalg.norm(want.astype(np.float64))))
    assert np.exp(np.mean(logs)) <= 1.1 * blocked
