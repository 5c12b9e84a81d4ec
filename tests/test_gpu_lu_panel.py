"""The 16-column register form of the cluster LU panel: bit-identical to the column-by-column
look-ahead form (the same operations on every element in the same order) for every thread
layout (rows per CTA <= 64, 128, 256, 512 and more), cluster size and partial block, with
ties, NaN columns and failing pivots at block edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(gpu, a):
    from rulinalg_gb300 import _lib as L
    out = []
    saved = gpu.tune_get(L.TUNE_PANEL_LOOKAHEAD)
    try:
        for la in (0, 1):
            gpu.tune_set(L.TUNE_PANEL_LOOKAHEAD, la)
            try:
                lu = gpu.PartialPivLu.decompose(a)
                out.append((lu.lu, lu.p.perm, None))
            except gpu.RulinalgError as e:
                out.append((None, None, e.kind))
    finally:
        gpu.tune_set(L.TUNE_PANEL_LOOKAHEAD, saved)
    return out


# f64 targets 64 rows a CTA (513..1024: 64; 1500: 94; 3000: 188; 5500: 344), f32 256
# (513: 171..; 3000: 250; 6000: 375; 9000: 563, 16 CTAs); odd sizes end in partial blocks;
# 6552 f64 rows fill 16 CTAs by size but not in whole rows (the first panel is cooperative)
@pytest.mark.parametrize("n,dtype", [(513, np.float64), (529, np.float64), (577, np.float64), (1024, np.float64),
                                     (1500, np.float64), (3000, np.float64), (5500, np.float64), (6552, np.float64),
                                     (513, np.float32),
                                     (545, np.float32), (1000, np.float32), (3001, np.float32), (6000, np.float32),
                                     (9000, np.float32)])
def test_bit_identical_to_lookahead_form(gpu, n, dtype):
    a = np.random.default_rng(n).uniform(-1, 1, (n, n)).astype(dtype)
    (f, p, e), (f2, p2, e2) = _both(gpu, a)
    assert e is None and e2 is None and np.array_equal(p, p2)
    assert np.array_equal(f.view(np.uint8), f2.view(np.uint8))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_ties_pick_the_first_row(gpu, dtype):
    rng = np.random.default_rng(2)
    n = 600
    a = rng.integers(-1, 2, (n, n)).astype(dtype) + 3 * np.eye(n, dtype=dtype)[rng.permutation(n)]
    (f, p, e), (f2, p2, e2) = _both(gpu, a)
    assert e == e2
    if e is None:
        assert np.array_equal(p, p2) and np.array_equal(f.view(np.uint8), f2.view(np.uint8))


@pytest.mark.parametrize("col", [0, 15, 16, 63, 64, 80, 599])
def test_failing_pivot_and_nan_column(gpu, col):
    rng = np.random.default_rng(col)
    a = rng.uniform(-1, 1, (600, 600))
    z = a.copy()
    z[:, col] = 0.0
    (_, _, e), (_, _, e2) = _both(gpu, z)
    assert e == e2 == "DivByZero"
    a[:, col] = np.nan  # no candidate in that column: the diagonal stays the pivot
    (f, p, e), (f2, p2, e2) = _both(gpu, a)
    assert e == e2
    if e is None:
        assert np.array_equal(p, p2) and np.array_equal(np.isnan(f), np.isnan(f2))
        ok = ~np.isnan(f)
        assert np.array_equal(f[ok], f2[ok])


@pytest.mark.parametrize("n", [3071, 3072, 3600])
def test_fp64_outer_blocks(gpu, n):
    """FP64 LU around the size where 512-column outer blocks start: P A = L U on sampled rows
    within n u |L||U|."""
    rng = np.random.default_rng(n)
    a = rng.uniform(-1, 1, (n, n))
    t = gpu.PartialPivLu.decompose(a).unpack()
    rows = rng.permutation(n)[:40]
    pa = np.empty_like(a)
    pa[t.p.perm.astype(np.int64)] = a
    bound = n * 2.0 ** -53 * (np.abs(t.l[rows]) @ np.abs(t.u))
    assert (np.abs(t.l[rows] @ t.u - pa[rows]) <= bound).all()
