"""FP64 products on the tensor cores as exact BF16 slices (m >= 64, n >= 32, k >= 32 and
m n k >= 6e6), against exact arithmetic: tile and chunk edges, integer operands whose
product must come out exactly (the largest digits too), operands that a row scaling cannot
represent, non-finite and extreme entries, and the blocked factorisations' forms."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _exact(a, b):
    return np.matmul(a.astype(np.longdouble), b.astype(np.longdouble))


def _check(c, a, b):
    """The classical componentwise bound of an FP64 dot product, k u |A||B|."""
    k = a.shape[1]
    bound = k * U * (np.abs(a) @ np.abs(b)) * (1 + 1e-10) + 1e-300
    assert (np.abs(c.astype(np.longdouble) - _exact(a, b)) <= bound).all()


@pytest.mark.parametrize("m,n,k", [(64, 400, 256), (65, 79, 1200), (127, 80, 608), (128, 81, 609), (129, 320, 191),
                                   (200, 161, 192), (1000, 64, 193), (260, 65, 385), (160, 33, 1153), (700, 700, 33)])
def test_product_edges(gpu, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    _check(gpu.mat_mul(a, b), a, b)


def test_split_k(gpu):
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((130, 5000)), rng.standard_normal((5000, 70))
    _check(gpu.mat_mul(a, b), a, b)


@pytest.mark.parametrize("k", [192, 400, 1000])
def test_integer_products_exact(gpu, k):
    """Products of 20-bit integers: every sum is below 2^53, so the result is exact."""
    rng = np.random.default_rng(k)
    a = rng.integers(-2 ** 20, 2 ** 20, (300, k)).astype(np.float64)
    b = rng.integers(-2 ** 20, 2 ** 20, (k, 130)).astype(np.float64)
    want = a.astype(np.int64) @ b.astype(np.int64)
    assert np.array_equal(gpu.mat_mul(a, b).astype(np.int64), want)


@pytest.mark.parametrize("digit", [-128, 127])
def test_largest_digits(gpu, digit):
    """Every digit of every entry at the end of its range and every term of one sign: the
    exact accumulators reach their bound (5 pairs x 192 x 2^14 below 2^24)."""
    k = 384
    mant = sum(digit * 256 ** t for t in range(6, -1, -1))  # 55 bits: 2 too many for one double
    v = float((mant >> 3) / 2.0 ** 52)
    a, b = np.full((260, k), v), np.full((k, 90), v)
    want = np.longdouble(v) * np.longdouble(v) * k
    c = gpu.mat_mul(a, b)
    assert (np.abs(c - want) <= 2 * U * abs(want)).all()


@pytest.mark.parametrize("spread", [8, 40, 300])
def test_graded_operands_keep_componentwise_accuracy(gpu, spread):
    """A D and D^-1 B with D graded over 2^spread: the large entries of a row and of a
    column do not meet, which a per-row scaling alone would lose."""
    rng = np.random.default_rng(spread)
    k = 300
    d = 2.0 ** np.linspace(-spread / 2, spread / 2, k)
    a, b = rng.standard_normal((200, k)) * d, rng.standard_normal((k, 170)) / d[:, None]
    _check(gpu.mat_mul(a, b), a, b)


def test_sparse_and_zero_rows(gpu):
    rng = np.random.default_rng(9)
    a, b = rng.standard_normal((256, 256)), rng.standard_normal((256, 256))
    eye = np.eye(256)
    assert np.array_equal(gpu.mat_mul(eye, b), b) and np.array_equal(gpu.mat_mul(a, eye), a)
    a[3] = 0
    a[200:] = 0
    b[:, 17] = 0
    c = gpu.mat_mul(a, b)
    assert (c[3] == 0).all() and (c[200:] == 0).all() and (c[:, 17] == 0).all()
    _check(c, a, b)


def test_non_finite_and_extreme_entries(gpu):
    rng = np.random.default_rng(11)
    a, b = rng.standard_normal((300, 200)), rng.standard_normal((200, 260))
    a[5, 7], a[6, 0], b[11, 250], a[280, 3], a[281], a[282] = np.nan, np.inf, -np.inf, 5e-324, 1e-310, 1e300
    b[:, 100] *= 1e-200
    with np.errstate(invalid="ignore", over="ignore"):
        want = a @ b
    c = gpu.mat_mul(a, b)
    assert np.array_equal(np.isnan(c), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(c[inf], want[inf])
    ok = np.isfinite(want)
    bound = 200 * U * (np.abs(np.where(np.isfinite(a), a, 0)) @ np.abs(np.where(np.isfinite(b), b, 0))) + 1e-320
    assert (np.abs(c[ok] - want[ok]) <= 2 * bound[ok]).all()


@pytest.mark.parametrize("n", [900, 1100])
def test_factorisations_over_slices(gpu, n):
    """LU, Cholesky (lower-triangle form, one operand on both sides) and QR (transposed
    operand) with FP64 trailing updates on the tensor cores: residuals within c n u."""
    rng = np.random.default_rng(n)
    a = rng.uniform(-1, 1, (n, n)) * 2.0 ** rng.integers(-30, 30, (n, 1))  # badly scaled rows
    lu = gpu.PartialPivLu.decompose(a)
    f, perm, st = O.lu_decompose(a)
    assert st == O.OK and np.array_equal(lu.p.perm, perm)
    parts = lu.unpack()
    pa = np.empty_like(a)
    pa[parts.p.perm.astype(np.int64)] = a
    assert (np.abs(parts.l @ parts.u - pa) <= n * U * (np.abs(parts.l) @ np.abs(parts.u))).all()
    g = rng.standard_normal((n, n))
    s = g @ g.T + n * np.eye(n)
    l = gpu.Cholesky.decompose(s).unpack()
    assert (np.abs(l @ l.T - s) <= 2 * n * U * (np.abs(l) @ np.abs(l).T)).all()
    qr = gpu.HouseholderQr.decompose(g[:, : n // 2]).unpack_thin()
    assert np.linalg.norm(qr.q1 @ qr.r1 - g[:, : n // 2]) <= 4 * n * U * np.linalg.norm(g[:, : n // 2])
    assert np.linalg.norm(qr.q1.T @ qr.q1 - np.eye(n // 2)) <= 4 * n * U
