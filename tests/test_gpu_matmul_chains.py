"""fp32 matmul of no whole tiles with long sums of one sign, where the truncation of each addition in tensor memory is the largest error:
against 64 bits no further off than the sequential loop."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(3))
@pytest.mark.parametrize("m,n,k", [(118, 1006, 8351), (200, 201, 20_000), (300, 301, 3000)])
def test_sums_of_one_sign(m, n, k, seed):
    from lapis_b200 import device
    g = torch.Generator(device="cuda").manual_seed(seed)
    A, B = torch.rand((m, k), device="cuda", generator=g), torch.rand((k, n), device="cuda", generator=g)
    got = device.bgemm(A, B, torch.zeros((m, n), device="cuda"))
    device.bgemm_status()
    loop = torch.cat([device.bgemm(A[r:r + 60].contiguous(), B, torch.zeros((len(A[r:r + 60]), n), device="cuda")) for r in range(0, m, 60)])
    exact = A.double() @ B.double()
    assert float((got.double() - exact).norm()) <= float((loop.double() - exact).norm())
