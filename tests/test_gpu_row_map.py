"""The pivots' row map (one gather instead of a chain of swaps): the permutation against
the oracle around the 64-pivot block edges, the solvers that gather by it, in place too,
and a size past the map's shared-memory limit."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 512, 513, 575, 576, 577, 1000])
def test_permutation_matches_oracle(gpu, n):
    a = np.random.default_rng(n).uniform(-1, 1, (n, n))
    lu = gpu.PartialPivLu.decompose(a)
    _, perm, st = O.lu_decompose(a)
    assert st == O.OK and np.array_equal(lu.p.perm, perm)


@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("nrhs", [1, 5])
def test_fp64_solve_gathers_rows(gpu, nrhs, in_place):
    torch = pytest.importorskip("torch")
    n = 641
    rng = np.random.default_rng(nrhs)
    a, b = rng.uniform(-1, 1, (n, n)), rng.standard_normal((n, nrhs))
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    tx = tb if in_place else torch.empty_like(tb)
    assert gpu.lib.rl_dsolve_fp64_dev(n, nrhs, 0, ta.data_ptr(), n, tb.data_ptr(), nrhs, tx.data_ptr(), nrhs, None,
                                      None) == 0
    torch.cuda.synchronize()
    x = tx.cpu().numpy()
    # normwise backward error of a stable solve, 10 n u
    res = np.abs(b - a @ x).max(axis=0) / (np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0))
    assert (res <= 10 * n * 2.0 ** -53).all()


def test_row_map_past_shared_memory(gpu):
    """n = 40,033 rows: the map lives in global memory. A = a row permutation of a
    diagonally dominant matrix, so nearly every pivot swaps."""
    torch = pytest.importorskip("torch")
    from rulinalg_gb300._lib import SolveInfo
    import ctypes as C
    n = 40033
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    a = torch.rand(n, n, dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    rows = torch.randperm(n, device="cuda", generator=g)
    a[rows, torch.arange(n, device="cuda")] += float(n)
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    x, info = torch.empty_like(b), SolveInfo()
    assert gpu.lib.rl_dsolve_mixed_dev(n, 1, 0, a.data_ptr(), n, b.data_ptr(), 1, x.data_ptr(), 1, C.byref(info),
                                       None) == 0
    assert info.path == 0 and info.berr <= 10 * n * 2.0 ** -53
