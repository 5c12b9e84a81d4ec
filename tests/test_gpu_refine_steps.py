"""The mixed single-system solver at the edge of its stopping test and of its convergence: the
FP32 sweeps of a refinement decide, by their block size and the order of their sums, at which
step a system passes. The systems are products of Hadamard matrices and signs around geometric
singular values, formed by additions alone, so they are the same bits on every machine; the step
counts and solution entries are those of 64-row diagonal blocks with 16-column quarters."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fwht(m):
    """H m, H the +-1 Hadamard matrix of order len(m)."""
    h = 1
    while h < len(m):
        v = m.reshape(len(m) // (2 * h), 2, h, -1)
        m = np.concatenate([v[:, :1] + v[:, 1:], v[:, :1] - v[:, 1:]], axis=1).reshape(len(m), -1)
        h *= 2
    return m


def system(n, seed, ratio):
    """S1 H S2 H diag(sigma) H S3 H S4 / n^2, sigma_i = ratio^i, and an integer right-hand side / 256."""
    rng = np.random.default_rng(seed)
    s = [rng.integers(0, 2, n) * 2.0 - 1.0 for _ in range(4)]
    sigma = [1.0]
    for _ in range(n - 1):
        sigma.append(sigma[-1] * ratio)
    m = np.diag(sigma)
    for left, right in ((s[0], s[1]), (s[2], s[3])):
        m = np.ascontiguousarray(_fwht(np.ascontiguousarray(_fwht(m).T)).T) / n * left[:, None] * right[None, :]
    return m, rng.integers(-1000, 1001, n) / 256.0


# n, seed, ratio, steps, x[0], x[1]
CASES = [
    (1024, 0, 0.98659, 13, "-0x1.38057cd008ad3p+16", "0x1.347deea23de48p+19"),
    (1024, 1, 0.98659, 14, "0x1.6a599f2da5298p+17", "-0x1.7e4ee294684e7p+16"),
    (1024, 2, 0.98659, 10, "-0x1.3da1ed6078511p+17", "-0x1.67abeb890f33fp+17"),
    (1024, 5, 0.98659, 20, "-0x1.cafba2f7b4e50p+16", "0x1.3a8cddee5d65dp+14"),
    (2048, 0, 0.99327, 13, "-0x1.2cf39bcdf8b6fp+18", "-0x1.ec6cdbf0aafd4p+16"),
    (2048, 2, 0.99327, 8, "0x1.f4a3265130d62p+17", "0x1.6185031c5f9edp+16"),
    (2048, 4, 0.99327, 21, "-0x1.63c049f0f5fefp+16", "-0x1.358f0f4041661p+19"),
]


@pytest.mark.parametrize("n,seed,ratio,steps,x0,x1", CASES)
def test_steps_and_solution(gpu, n, seed, ratio, steps, x0, x1):
    a, b = system(n, seed, ratio)
    x, info = gpu.solve_mixed(a, b, "lu")
    assert info["path"] == "refinement" and info["iters"] == steps
    scale = 1e-9 * np.abs(x).max()
    assert abs(x[0] - float.fromhex(x0)) <= scale and abs(x[1] - float.fromhex(x1)) <= scale


@pytest.mark.parametrize("nrhs", [2, 9])
def test_several_right_hand_sides_converge(gpu, nrhs):
    """The same triangle applied to several columns: no fallback, backward error sqrt(n) u."""
    a, b = system(1024, 0, 0.98659)
    bs = np.stack([np.roll(b, 37 * c) for c in range(nrhs)], axis=1)
    x, info = gpu.solve_mixed(a, bs, "lu")
    assert info["path"] == "refinement"
    r = np.abs(bs - a @ x).max(axis=0)
    assert (r <= 4 * np.sqrt(1024) * 2.0 ** -53 * np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0)).all()


@pytest.mark.parametrize("n", [1, 5, 33, 63, 64, 65, 100, 300])
def test_small_orders(gpu, n):
    """Below the sizes with inverted blocks: the substitution sweeps in every mode, one and three columns."""
    rng = np.random.default_rng(n)
    a = rng.uniform(-1, 1, (n, n)) + 3 * np.eye(n)
    g = rng.standard_normal((n, n))
    for m, kind in ((a, "lu"), (g @ g.T + n * np.eye(n), "cholesky")):
        for b in (rng.standard_normal(n), rng.standard_normal((n, 3))):
            x, info = gpu.solve_mixed(m, b, kind)
            assert info["path"] == "refinement"
            assert np.abs(b - m @ x).max() <= 4 * np.sqrt(n) * 2.0 ** -53 * np.abs(m).sum(axis=1).max() * np.abs(x).max()


@pytest.mark.parametrize("kind,nrhs", [("lu", 1), ("cholesky", 1), ("lu", 9)])
def test_withheld_block_is_reported(gpu, kind, nrhs):
    """A block of the refinement's sweeps (and of the FP64 fallback's) is never published: the waits for
    it end by their own limit, the call returns the timeout, and the next one is right."""
    from rulinalg_gb300 import _lib as L
    n = 1000
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n))
    a = g @ g.T + n * np.eye(n) if kind == "cholesky" else g + 40 * np.eye(n)
    b = rng.standard_normal((n, nrhs))
    try:
        gpu.tune_set(L.TUNE_WAIT_TIMEOUT_NS, 20_000_000)
        gpu.tune_set(L.TUNE_TEST_WITHHOLD_SWEEP_BLOCK, 5)
        with pytest.raises(gpu.DeviceError) as e:
            gpu.solve_mixed(a, b, kind)
        assert e.value.status == 35
    finally:
        gpu.tune_set(L.TUNE_TEST_WITHHOLD_SWEEP_BLOCK, -1)
        gpu.tune_set(L.TUNE_WAIT_TIMEOUT_NS, 10 ** 9)
    x, info = gpu.solve_mixed(a, b, kind)
    assert info["path"] == "refinement" and np.abs(b - a @ x).max() <= 1e-11 * np.abs(b).max()
