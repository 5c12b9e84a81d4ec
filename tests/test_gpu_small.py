"""Single matrices on one CTA up to 64 rows (LU, LU + solve in one launch, Cholesky) and the
sizes around which the one-CTA and the blocked forms meet, against the oracle."""
import numpy as np
import pytest

import oracle as O
from comparators import backward_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 47, 63, 64, 65, 88, 89, 240, 241])
def test_lu_solve_cholesky_around_the_edges(gpu, n):
    rng = np.random.default_rng(n)
    a, b = rng.uniform(-1, 1, (n, n)) + 2 * np.eye(n)[rng.permutation(n)], rng.standard_normal(n)
    f, perm, st = O.lu_decompose(a)
    assert st == O.OK
    lu = gpu.PartialPivLu.decompose(a)
    u = 2.0 ** -53
    assert np.array_equal(lu.p.perm, perm)
    scale = np.abs(np.tril(f, -1) + np.eye(n)) @ np.abs(np.triu(f))
    assert (np.abs(lu.lu - f) <= 4 * n * u * (scale.max() * np.abs(np.linalg.inv(np.triu(f))).max() * np.abs(f).max() + 1)).all()
    x = gpu.solve(a, b)
    assert backward_error(a, x, b) <= 4 * n * u
    assert backward_error(a, lu.solve(b), b) <= 4 * n * u
    g = rng.standard_normal((n, n))
    s = g @ g.T + n * np.eye(n)
    l = gpu.Cholesky.decompose(s)
    lt = l.unpack()
    assert np.abs(lt @ lt.T - s).max() <= 4 * n * u * np.abs(s).max()
    assert np.array_equal(np.triu(l.l, 1), np.triu(s, 1))  # the strict upper triangle is not written
    assert backward_error(s, l.solve(b), b) <= 8 * n * u


@pytest.mark.parametrize("n", [7, 64, 100, 256, 257, 448, 449])
def test_f32(gpu, n):
    rng = np.random.default_rng(n)
    a, b = (rng.uniform(-1, 1, (n, n)) + np.eye(n)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    e = 2.0 ** -24
    x = gpu.solve(a, b).astype(np.float64)
    assert backward_error(a.astype(np.float64), x, b.astype(np.float64)) <= 8 * n * e
    g = rng.standard_normal((n, n))
    s = (g @ g.T + n * np.eye(n)).astype(np.float32)
    lt = gpu.Cholesky.decompose(s).unpack().astype(np.float64)
    assert np.abs(lt @ lt.T - s).max() <= 8 * n * e * np.abs(s).max()


@pytest.mark.parametrize("n", [1, 20, 64])
def test_failures_leave_the_operands(gpu, n):
    rng = np.random.default_rng(n)
    a, b = rng.uniform(-1, 1, (n, n)), rng.standard_normal(n)
    a[:, n // 2] = 0
    with pytest.raises(gpu.RulinalgError) as e:
        gpu.solve(a, b)
    assert e.value.kind == "DivByZero"
    s = np.eye(n)
    s[n // 2, n // 2] = -1
    with pytest.raises(gpu.RulinalgError) as e:
        gpu.Cholesky.decompose(s)
    assert e.value.kind == "DecompFailure"
    a[:, n // 2] = np.nan  # no candidate: the diagonal stays the pivot, as in the reference
    f, perm, st = O.lu_decompose(a)
    if st == O.OK:
        assert np.array_equal(gpu.PartialPivLu.decompose(a).p.perm, perm)


def test_many_threads_share_nothing(gpu):
    from concurrent.futures import ThreadPoolExecutor
    rng = np.random.default_rng(8)
    work = [(rng.uniform(-1, 1, (n, n)) + np.eye(n) * n, rng.standard_normal(n)) for n in (5, 33, 64) * 20]
    with ThreadPoolExecutor(6) as ex:
        xs = list(ex.map(lambda w: gpu.solve(*w), work))
    for (a, b), x in zip(work, xs):
        assert backward_error(a, x, b) <= 4 * len(b) * 2.0 ** -53
