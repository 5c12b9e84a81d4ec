"""FP64 Cholesky of a matrix that is not positive definite: the failure is reported wherever it is,
and a failure in the first block costs a fraction of the factorisation."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,at", [(65, 0), (65, 63), (65, 64), (128, 64), (700, 0), (700, 130), (700, 699), (1300, 1023),
                                  (1300, 1024), (1300, 1299)])
def test_failure_is_reported(gpu, n, at):
    rng = np.random.default_rng(n + at)
    g = rng.standard_normal((n, n))
    a = g @ g.T + n * np.eye(n)
    gpu.Cholesky.decompose(a)
    a[at, at] = -1.0
    with pytest.raises(gpu.RulinalgError):
        gpu.Cholesky.decompose(a)


@pytest.mark.parametrize("n", [1024, 4096])
def test_early_failure_is_cheap(gpu, n):
    import torch
    a = torch.eye(n, dtype=torch.float64, device="cuda") * 4 + 1
    b, x = torch.ones(n, 1, dtype=torch.float64, device="cuda"), torch.empty(n, 1, dtype=torch.float64, device="cuda")

    def once():
        t = time.perf_counter()
        st = gpu.lib.rl_dsolve_fp64_dev(n, 1, 1, a.data_ptr(), n, b.data_ptr(), 1, x.data_ptr(), 1, None, C.c_void_p(None))
        return st, time.perf_counter() - t

    good = [once() for _ in range(5)]
    torch.cuda.synchronize()
    a[3, 3] = -1.0
    torch.cuda.synchronize()
    bad = [once() for _ in range(5)]
    assert all(st == 0 for st, _ in good) and all(st != 0 for st, _ in bad)
    assert sorted(t for _, t in bad)[2] <= 0.3 * sorted(t for _, t in good)[2]


def test_threads_keep_their_own_outcome(gpu):
    from concurrent.futures import ThreadPoolExecutor
    rng = np.random.default_rng(9)
    g = rng.standard_normal((300, 300))
    good = g @ g.T + 300 * np.eye(300)
    bad = good.copy()
    bad[70, 70] = -1.0

    def job(i):
        if i % 3 == 2:
            return np.abs(gpu.mat_mul(good, g) - good @ g).max() <= 300 * 2.0 ** -52 * np.abs(good).max() * np.abs(g).max() * 4
        try:
            l = gpu.Cholesky.decompose(bad if i % 3 else good).unpack()
            return i % 3 == 0 and np.abs(l @ l.T - good).max() <= 300 * 2.0 ** -52 * np.abs(good).max()
        except gpu.RulinalgError as e:
            return i % 3 == 1 and e.kind == "DecompFailure"

    with ThreadPoolExecutor(6) as ex:
        assert all(ex.map(job, range(90)))
