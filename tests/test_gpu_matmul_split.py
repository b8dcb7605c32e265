"""fp32 matmul from operands split into fp16 parts (gemm_split.cu): edges of tiles, stretches of K and batches, what the split
does not cover, and the call under capture and on two streams."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(batch, m, n, k, seed=0, make=None):
    g = torch.Generator(device="cuda").manual_seed(seed)
    make = make or (lambda s: torch.rand(s, generator=g, device="cuda") * 2 - 1)
    lead = () if batch == 1 else (batch,)
    return make(lead + (m, k)), make(lead + (k, n)), make(lead + (m, n))


def _check(A, B, C, got):
    """Per element: parts and left-out product 2^-21 of |a| |b|, at most 64 truncated additions of a chain (2^-23 of the partial
    sum each), one rounded addition a chain and stretch, C joined last."""
    exact = C.double() + A.double() @ B.double()
    mag = A.double().abs() @ B.double().abs()
    k = A.shape[-1]
    bound = (2.0 ** -21 + min(k / 16, 64) * 2.0 ** -23 + (k / 128 + 2) * 2.0 ** -24) * mag + 2.0 ** -23 * (C.double().abs() + exact.abs())
    assert torch.all((got.double() - exact).abs() <= bound)


@pytest.mark.parametrize("batch,m,n,k", [
    (1, 1000, 1501, 777), (1, 1001, 1504, 776), (1, 1024, 1536, 128 * 9 + 1), (1, 129, 4000, 1000), (1, 4097, 127, 1025),  # no whole tiles
    (1, 64, 8193, 600), (1, 5000, 3000, 130), (1, 300, 300, 8000), (100, 200, 200, 200), (3, 257, 1500, 1100),
    (1, 128, 128, 1024), (1, 128, 128, 4128), (1, 1024, 1024, 1056), (1, 2048, 2304, 1024), (2, 1024, 1280, 2080)])        # whole tiles
def test_products_of_every_form(batch, m, n, k):
    from lapis_b200 import device
    A, B, C = _operands(batch, m, n, k, m + n + k)
    got = device.bgemm(A, B, C.clone())
    device.bgemm_status()
    _check(A, B, C, got)
    shifted = [torch.empty(t.numel() + 1, device="cuda")[1:].view(t.shape).copy_(t) for t in (A, B, C)]  # 4 bytes off
    off = device.bgemm(*shifted)
    device.bgemm_status()
    _check(A, B, C, off)
    assert torch.equal(got, device.bgemm(A, B, C.clone()))


@pytest.mark.parametrize("m,n,k", [(1000, 1501, 777), (1024, 1536, 1024)])
def test_rows_and_columns_of_any_scale(m, n, k):
    """Rows of A and columns of B from 1e-12 to 1e12: one scale each, nothing is lost."""
    from lapis_b200 import device
    A, B, _ = _operands(1, m, n, k, 3)
    A = A * torch.logspace(-12, 12, m, device="cuda")[:, None]
    B = B * torch.logspace(12, -12, n, device="cuda")[None, :]
    C = torch.zeros((m, n), device="cuda")
    got = device.bgemm(A, B, C.clone())
    device.bgemm_status()
    _check(A, B, C, got)


@pytest.mark.parametrize("m,n,k", [(1000, 1501, 777), (1024, 1536, 1024), (300, 300, 8000)])
def test_what_the_split_does_not_cover(m, n, k):
    """Elements 2^40 below the largest of their row, a huge row, infinities and NaN: the panels of 128 rows or columns that hold
    them come from the kernels on whole operands, the others are not touched by them."""
    from lapis_b200 import device
    A, B, C = _operands(1, m, n, k, 4)
    plain = device.bgemm(A, B, C.clone())
    A[5, 3], A[140, 7] = 2.0 ** -41, 1e25       # panels 0 and 1 of A
    B[9, 270] = float("inf")                    # panel 2 of B
    B[k - 1, 299] = float("nan")
    got = device.bgemm(A, B, C.clone())
    device.bgemm_status()
    assert torch.equal(got[256:, :256], plain[256:, :256])
    if n > 384:
        assert torch.equal(got[256:, 384:], plain[256:, 384:])
    assert torch.isnan(got[:, 299]).all()
    nonfinite = torch.zeros(n, dtype=torch.bool, device="cuda")
    nonfinite[[270, 299]] = True
    assert not torch.isfinite(got[:, 270]).any()
    assert torch.isfinite(got[:, ~nonfinite]).all()
    exact = C.double() + A.double() @ B.double()
    mag = A.double().abs() @ B.double().abs()
    ok = (got.double() - exact).abs()[:, ~nonfinite] <= 1e-5 * mag[:, ~nonfinite]  # also the TF32 split's 2^-19 a product
    assert ok.all()
    if n % 128 != 0 and k <= 1024:
        # the kernel for general shapes, one stretch: the sequential loop's bits, as a product of few rows has them
        few = device.bgemm(A[:40].contiguous(), B, C[:40].clone())
        assert torch.equal(got[:40, ~nonfinite], few[:, ~nonfinite])


def test_graded_operands_are_left_to_the_other_kernel():
    """Columns of A scaled by 2^i, rows of B by 2^-i: every panel is marked, every product is of the same size."""
    from lapis_b200 import device
    m, n, k = 1000, 1100, 300
    A, B, C = _operands(1, m, n, k, 5)
    scale = 2.0 ** torch.linspace(-40, 40, k, device="cuda").round()
    A, B = A * scale[None, :], B / scale[:, None]
    got = device.bgemm(A, B, C.clone())
    _check(A, B, C, got)
    assert torch.equal(got[:40], device.bgemm(A[:40].contiguous(), B, C[:40].clone()))


def test_zeros_and_empty_rows():
    from lapis_b200 import device
    A, B, C = _operands(1, 1000, 1501, 777, 6)
    A[17], B[:, 33], A[40:60, 100:300] = 0.0, 0.0, 0.0
    got = device.bgemm(A, B, C.clone())
    _check(A, B, C, got)
    assert torch.equal(got[17], C[17]) and torch.equal(got[:, 33], C[:, 33])


@pytest.mark.parametrize("m,n,k", [(1000, 1501, 777), (1024, 1536, 2048)])
def test_capture_and_streams(m, n, k):
    from lapis_b200 import device
    sets = [_operands(1, m, n, k, s) for s in range(4)]
    want = [device.bgemm(A, B, C.clone()) for A, B, C in sets]
    A, B, C = sets[0]
    out = C.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        device.bgemm(A, B, out)
    for _ in range(2):
        out.copy_(C)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want[0])
    streams = [torch.cuda.Stream() for _ in sets]
    outs = [C.clone() for _, _, C in sets]
    torch.cuda.synchronize()
    for _ in range(5):
        for st, (A, B, C), o in zip(streams, sets, outs):
            with torch.cuda.stream(st):
                o.copy_(C)
                device.bgemm(A, B, o)
    torch.cuda.synchronize()
    assert all(torch.equal(o, w) for o, w in zip(outs, want))
    device.bgemm_status()
