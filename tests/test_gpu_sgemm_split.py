"""FP32 products on the tensor cores: operand strides and alignments of the splitting pass
(16-byte and single loads), ragged K and tiles, vectorised and scalar stores, strided C."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(128, 256, 128), (129, 257, 131), (130, 300, 127), (256, 1000, 64), (300, 259, 333),
                                   (64, 2050, 400), (512, 288, 516)])
@pytest.mark.parametrize("pad,off", [(0, 0), (3, 0), (4, 0), (4, 1)])
def test_strided_operands(gpu, m, k, n, pad, off):
    rng = np.random.default_rng(m + k + n)
    a = rng.standard_normal((m, k + pad)).astype(np.float32)[:, off:off + k]
    b = rng.standard_normal((k, n + pad)).astype(np.float32)[:, off:off + n]
    c = gpu.mat_mul(a, b)
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    assert (np.abs(c - a64 @ b64) <= 2 * k * 2.0 ** -24 * (np.abs(a64) @ np.abs(b64))).all()


@pytest.mark.parametrize("ldc,off", [(512, 0), (515, 0), (516, 0), (516, 1)])
def test_strided_device_operands_and_result(gpu, ldc, off):
    torch = pytest.importorskip("torch")
    m, k, n, ld = 200, 320, 500, 517
    g = torch.Generator(device="cuda")
    g.manual_seed(ldc + off)
    a = torch.randn(m, ld, device="cuda", generator=g)
    b = torch.randn(k, ld, device="cuda", generator=g)
    c = torch.full((m, ldc + 1), 7.0, device="cuda")
    base = c.view(-1)[off:]
    ldc_used = ldc + 1 if ldc != 516 else 516
    assert gpu.lib.rl_sgemm_dev(m, k, n, a.data_ptr(), ld, b.data_ptr(), ld, base.data_ptr(), ldc_used, None) == 0
    torch.cuda.synchronize()
    got = torch.as_strided(base, (m, n), (ldc_used, 1)).double()
    want = a[:, :k].double() @ b[:, :n].double()
    bound = 2 * k * 2.0 ** -24 * (a[:, :k].double().abs() @ b[:, :n].double().abs())
    assert bool(((got - want).abs() <= bound).all())
    flat = torch.as_strided(base, (m - 1, ldc_used - n), (ldc_used, 1), base.storage_offset() + n)
    assert bool((flat == 7.0).all())  # nothing written between the rows
