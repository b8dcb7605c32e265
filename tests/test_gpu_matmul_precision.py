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


def _sequential(A, B):
    """The error of the sequential fp32 loop, k ascending, product and sum rounded: its 2-norm over that of the result."""
    acc = torch.zeros((A.shape[0], B.shape[1]), device="cuda")
    for k in range(A.shape[1]):
        acc = acc + A[:, k:k + 1] * B[k:k + 1]
    exact = A.double() @ B.double()
    return float((acc.double() - exact).norm() / exact.norm())


@pytest.mark.parametrize("m,n,k", [(1000, 1501, 777), (1001, 1504, 776), (129, 4000, 1000), (2100, 1999, 1500)])
def test_selections_are_exact(m, n, k):
    """One 1 in every row of A, or in every column of B, or small whole numbers: the loop makes no error, nor does the product of no
    whole tiles."""
    from lapis_b200 import device
    g = _gen(m)
    dense = lambda *s: torch.rand(s, device="cuda", generator=g) * 2 - 1
    A, B = torch.zeros((m, k), device="cuda"), dense(k, n)
    j = torch.randint(0, k, (m,), device="cuda", generator=g)
    A[torch.arange(m, device="cuda"), j] = 1.0
    assert torch.equal(device.bgemm(A, B, torch.zeros((m, n), device="cuda")), B[j])
    A, B = dense(m, k), torch.zeros((k, n), device="cuda")
    j = torch.randint(0, k, (n,), device="cuda", generator=g)
    B[j, torch.arange(n, device="cuda")] = 1.0
    assert torch.equal(device.bgemm(A, B, torch.zeros((m, n), device="cuda")), A[:, j])
    whole = lambda *s: torch.randint(-8000, 8000, s, device="cuda", generator=g).float()
    A = whole(m, k) * (torch.rand((m, k), device="cuda", generator=g) < 0.5 / k)  # few terms: the sums stay whole numbers
    A[0] = 0.0
    A[0, 0] = 4095.0
    B = whole(k, n).clamp(-4095, 4095)
    exact = A.double() @ B.double()
    ok = (A.double().abs() @ B.double().abs()) < 2 ** 24
    got = device.bgemm(A, B, torch.zeros((m, n), device="cuda"))
    assert torch.equal(got.double()[ok], exact[ok]) and ok.float().mean() > 0.1
    device.bgemm_status()


@pytest.mark.parametrize("kind", ["both signs", "one sign", "1 % nonzeros", "10 % nonzeros", "normal", "wide range"])
@pytest.mark.parametrize("m,n,k", [(1000, 1501, 777), (129, 4000, 1000), (700, 900, 300), (1500, 1501, 130), (301, 300, 8000)])
def test_error_is_no_larger_than_the_loops(m, n, k, kind):
    from lapis_b200 import device
    g = _gen(k)
    make = (lambda *s: torch.randn(s, device="cuda", generator=g)) if kind == "normal" else lambda *s: torch.rand(s, device="cuda", generator=g) * 2 - 1
    A, B = make(m, k), make(k, n)
    if kind == "one sign":
        A, B = A.abs(), B.abs()
    if kind.endswith("nonzeros"):
        A = A * (torch.rand((m, k), device="cuda", generator=g) < (0.01 if kind[1] == " " else 0.1))
    if kind == "wide range":
        A, B = A.sign() * torch.exp(2 * torch.randn((m, k), device="cuda", generator=g)), B.sign() * torch.exp(2 * torch.randn((k, n), device="cuda", generator=g))
    got = device.bgemm(A, B, torch.zeros((m, n), device="cuda"))
    device.bgemm_status()
    exact = A.double() @ B.double()
    assert float((got.double() - exact).norm() / exact.norm()) <= _sequential(A, B)
