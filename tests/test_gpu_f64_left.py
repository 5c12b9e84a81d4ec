"""FP64 products whose tiles the tensor-core form leaves to the FP64 unit, whole or in part: sparse,
triangular and graded operands at the edges of the tiles, few outputs with a long K, the SYRK form of
a banded Cholesky, and the form a captured stream takes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _check(c, a, b):
    """The componentwise bound of an FP64 dot product, k u |A||B|."""
    want = np.matmul(a.astype(np.longdouble), b.astype(np.longdouble))
    bound = a.shape[1] * U * (np.abs(a) @ np.abs(b)) * (1 + 1e-10) + 1e-300
    assert (np.abs(c.astype(np.longdouble) - want) <= bound).all()


@pytest.mark.parametrize("m,n,k", [(192, 192, 192), (200, 161, 200), (129, 320, 191), (65, 400, 250), (321, 95, 208),
                                   (1000, 64, 193)])
def test_identity_triangle_and_grading(gpu, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    eye = np.eye(m, k)
    assert np.array_equal(gpu.mat_mul(eye, b), eye @ b)
    _check(gpu.mat_mul(np.tril(a), b), np.tril(a), b)
    d = 2.0 ** np.linspace(-40, 40, k)
    _check(gpu.mat_mul(a * d, b / d[:, None]), a * d, b / d[:, None])
    a[m // 2:, : k // 2] = 0  # half of the rows against operands that meet them in half of K
    b[k // 2:, n // 2:] = 0
    _check(gpu.mat_mul(a, b), a, b)


@pytest.mark.parametrize("m,n,k", [(64, 50, 5000), (130, 33, 1031), (65, 130, 3001)])
def test_few_outputs_long_k(gpu, m, n, k):
    rng = np.random.default_rng(k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    a[: m // 2, k // 3:] = 0
    b[: k // 3, : n // 2] = 0
    c = gpu.mat_mul(a, b)
    assert (c[: m // 2, : n // 2] == 0).all()
    _check(c, a, b)


@pytest.mark.parametrize("n,band", [(700, 3), (901, 40)])
def test_banded_cholesky(gpu, n, band):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    s = np.tril(rng.uniform(-1, 1, (n, n)) * (np.abs(i[:, None] - i[None, :]) <= band), -1)
    s = s + s.T + 2 * band * np.eye(n)
    l = gpu.Cholesky.decompose(s).unpack()
    assert (np.abs(l @ l.T - s) <= 2 * n * U * (np.abs(l) @ np.abs(l).T)).all()
    assert (l[i[:, None] - i[None, :] > band] == 0).all()  # no fill outside the band


@pytest.mark.parametrize("m,n,k", [(300, 260, 200), (128, 96, 4000)])
def test_captured_product(gpu, m, n, k):
    """In a stream capture the product takes the FP64 unit; the graph replays it on new inputs."""
    import torch
    a, b = (torch.randn(*s, dtype=torch.float64, device="cuda") for s in ((m, k), (k, n)))
    c = torch.zeros(m, n, dtype=torch.float64, device="cuda")

    def call():
        s = torch.cuda.current_stream().cuda_stream
        return gpu.lib.rl_dgemm_dev(m, k, n, a.data_ptr(), k, b.data_ptr(), n, c.data_ptr(), n, C.c_void_p(s))

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert call() == 0
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        st = call()
    assert st == 0
    for _ in range(2):
        a.normal_()
        g.replay()
        torch.cuda.synchronize()
        _check(c.cpu().numpy(), a.cpu().numpy(), b.cpu().numpy())
