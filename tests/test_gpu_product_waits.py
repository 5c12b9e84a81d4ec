"""A wait that runs out inside an FP64 product on the tensor cores is reported by the call it
belongs to, and by no later one: one tile of each product never announces its accumulators (a
test setting), so the waits for it end by their own limit of 20 ms; no GPU is faulted or hung."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
RL_ERR_TIMEOUT = 35
N = 700


def _calls(gpu):
    rng = np.random.default_rng(5)
    a = rng.uniform(-1, 1, (N, N)) + np.eye(N)
    spd = a @ a.T + N * np.eye(N)
    b = rng.standard_normal((N, 300))
    lu, chol, qr = gpu.PartialPivLu.decompose(a), gpu.Cholesky.decompose(spd), gpu.HouseholderQr.decompose(a)
    return {
        "product": lambda: gpu.mat_mul(a, b),
        "lu": lambda: gpu.PartialPivLu.decompose(a),
        "cholesky": lambda: gpu.Cholesky.decompose(spd),
        "qr": lambda: gpu.HouseholderQr.decompose(a),
        "qr q": lambda: qr.unpack(),
        "lu solve": lambda: lu.solve(b),
        "cholesky solve": lambda: chol.solve(b),
        "triangle": lambda: gpu.solve_l_triangular(np.tril(a) + 4 * np.eye(N), b),
        "inverse": lambda: gpu.inverse(a),
        "mixed": lambda: gpu.solve_mixed(a, b[:, :64], "lu"),
    }


@pytest.fixture
def withheld(gpu):
    from rulinalg_gb300 import _lib as L
    yield lambda tile: (gpu.tune_set(L.TUNE_TEST_WITHHOLD_PRODUCT_TILE, tile),
                        gpu.tune_set(L.TUNE_WAIT_TIMEOUT_NS, 10 ** 9 if tile < 0 else 20_000_000))
    gpu.tune_set(L.TUNE_TEST_WITHHOLD_PRODUCT_TILE, -1)
    gpu.tune_set(L.TUNE_WAIT_TIMEOUT_NS, 10 ** 9)


@pytest.mark.parametrize("name", ["product", "lu", "cholesky", "qr", "qr q", "lu solve", "cholesky solve", "triangle",
                                  "inverse", "mixed"])
def test_the_call_reports_it(gpu, withheld, name):
    call = _calls(gpu)[name]
    withheld(0)
    with pytest.raises(gpu.DeviceError) as e:
        call()
    assert e.value.status == RL_ERR_TIMEOUT
    withheld(-1)
    rng = np.random.default_rng(6)
    for dt in (np.float64, np.float32):  # later products, FP64 and FP32 on the tensor cores, are not blamed
        x, y = rng.standard_normal((300, 300)).astype(dt), rng.standard_normal((300, 300)).astype(dt)
        assert np.abs(gpu.mat_mul(x, y) - x.astype(np.float64) @ y).max() <= 300 * np.finfo(dt).eps * 30
    call()
