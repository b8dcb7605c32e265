"""fp32 matmul of no whole tiles from split operands (gemm_split.cu): C is joined last and once over any number of stretches of K,
groups of stretches and blocks of C, and what the split does not cover comes in the sequential loop's order."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# K in one stretch; in several of one launch; in two groups (operands of 200 MB); in blocks of rows and of columns, two groups each
SHAPES = [(300, 301, 1000), (301, 300, 8000), (2100, 2099, 8000), (70_000, 321, 1300), (200, 140_001, 2000)]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_one_rounding_joins_a_large_c(m, n, k):
    """Whole numbers up to 8: the product is exact in any order, so the result is its sum with C, rounded once."""
    from lapis_b200 import device
    g = _gen(k)
    A, B = (torch.randint(-8, 9, s, device="cuda", generator=g).float() for s in ((m, k), (k, n)))
    C = (torch.rand((m, n), device="cuda", generator=g) * 2 - 1) * 1000
    got = device.bgemm(A, B, C.clone())
    device.bgemm_status()
    for r in range(0, m, 4096):
        exact = A[r:r + 4096].double() @ B.double() + C[r:r + 4096].double()
        assert torch.equal(got[r:r + 4096], exact.float())


@pytest.mark.parametrize("at", [0, -1])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_what_the_split_does_not_cover_keeps_the_loops_order(m, n, k, at):
    """An element 2^-41 in the first or the last stretch of a row of A, an infinity in a column of B."""
    from lapis_b200 import device
    g = _gen(n)
    A, B, C = (torch.rand(s, device="cuda", generator=g) * 2 - 1 for s in ((m, k), (k, n), (m, n)))
    plain = device.bgemm(A, B, C.clone())
    A[m - 3, at], B[at, 140] = 2.0 ** -41, float("inf")
    got = device.bgemm(A, B, C.clone())
    device.bgemm_status()
    first = (m - 3) // 128 * 128
    few = slice(max(first, m - 40), m)  # fewer than 64 rows: the sequential loop's kernel
    assert torch.equal(got[few].nan_to_num(), device.bgemm(A[few].contiguous(), B, C[few].clone()).nan_to_num())
    cols = slice(128, 168)
    want = device.bgemm(A, B[:, cols].contiguous(), C[:, cols].contiguous())
    assert torch.equal(got[:, cols].nan_to_num(), want.nan_to_num())
    assert torch.equal(got[:first, :128], plain[:first, :128]) and torch.equal(got[:first, 256:], plain[:first, 256:])
