"""FP64 products with a long K: the 64-bit accumulators of the tensor-core form hold 2^46 times the
sum of the scaled products, so entries of one sign just below a power of two would wrap them from
131,072 columns per CTA on. Entries are 30 or 31 sixteenths (15/16 and 31/32 of a power of two) and
every partial sum has fewer than 53 bits, so the product is exact in any order."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (1100, 1100, 160_000),   # as many tiles as SMs: K on one CTA
    (1100, 1100, 65_537),    # one column past a CTA's share
    (64, 32, 2_400_003),     # one tile: 16 slices of K at once, and a ragged K
])
def test_one_signed_entries(gpu, m, n, k):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    a = torch.randint(30, 32, (m, k), device="cuda", generator=g).double() / 16
    b = torch.randint(30, 32, (k, n), device="cuda", generator=g).double() / -16
    c = torch.empty(m, n, dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert gpu.lib.rl_dgemm_dev(m, k, n, a.data_ptr(), k, b.data_ptr(), n, c.data_ptr(), n, C.c_void_p(s or None)) == 0
    torch.cuda.synchronize()
    assert torch.equal(c, a @ b)
