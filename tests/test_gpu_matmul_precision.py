"""fp32 matmul from split operands (gemm_split.cu) where single products or a large C decide the error."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("m,n,k", [(128, 128, 1024), (1024, 1536, 1024), (1000, 1501, 777)])
@pytest.mark.parametrize("below", [28, 29, 30])
def test_small_elements_that_decide_the_result(m, n, k, below):
    """The largest element of every row of A and column of B meets a zero; the one product of each element of C is of two
    elements 2^-below to 2^-(below + 1) of those.  A product may lose 2^-19: what the split into truncated TF32 parts, the
    coarsest of the kernels, leaves out."""
    from lapis_b200 import device
    g = _gen(below)
    A, B = torch.zeros((m, k), device="cuda"), torch.zeros((k, n), device="cuda")
    A[:, 0] = 1.0  # meets row 0 of B, which is zero
    B[1, :] = 1.0  # meets column 1 of A, which is zero
    j = 2 + torch.randint(0, k - 2, (m,), device="cuda", generator=g)
    A[torch.arange(m, device="cuda"), j] = (torch.rand(m, device="cuda", generator=g) + 1) * 2.0 ** -(below + 1)
    B[2:] = (torch.rand((k - 2, n), device="cuda", generator=g) + 1) * 2.0 ** -(below + 1)
    got = device.bgemm(A, B, torch.zeros((m, n), device="cuda"))
    device.bgemm_status()
    exact = A.double() @ B.double()
    assert torch.all((got.double() - exact).abs() <= 2.0 ** -19 * exact)
