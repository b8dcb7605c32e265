"""Batched products whose right-hand side is larger than L2, taken in slices of its rows: every form returns the bits of the
sequential row loop, so the slices are compared bit for bit with products of parts that L2 holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _matrix(rows, cols, lens, idx, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    pos = torch.zeros(rows + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(lens, 0, out=pos[1:])
    nnz = int(pos[-1])
    crd = torch.randint(0, cols, (nnz,), device=DEV, generator=g)
    val = torch.rand(nnz, dtype=torch.float64, device=DEV, generator=g) * 2 - 1
    return pos.to(idx), crd.to(idx), val


def _dense(shape, dtype, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.rand(shape, dtype=dtype, device=DEV, generator=g) * 2 - 1


@pytest.mark.parametrize("idx", [torch.int32, torch.int64])
@pytest.mark.parametrize("cols,dh,nh", [(131_072, 64, 8), (131_072, 25, 8), (100_000, 27, 10), (60_000, 71, 7), (300_000, 20, 4), (100_000, 300, 1)])
def test_bspmm_in_slices(cols, dh, nh, idx):
    """B of 96 to 268 MB, fibers of any length: against dh taken a few at a time."""
    from lapis_b200 import device
    rows = 2003
    lens = torch.randint(0, 20, (rows,), device=DEV, generator=torch.Generator(device=DEV).manual_seed(nh))
    pos, crd, val = _matrix(rows, cols, lens, idx, nh)
    val = _dense((crd.numel() * nh,), torch.float32, 4)
    B, C = _dense((cols, dh, nh), torch.float32, 5), _dense((rows, dh, nh), torch.float32, 6)
    got, summed = device.bspmm_csrv(pos, crd, val, B, cols), device.bspmm_csrv(pos, crd, val, B, cols, C.clone())
    step = max(1, 90_000_000 // (4 * cols * nh))
    for d0 in range(0, dh, step):
        part = B[:, d0:d0 + step].contiguous()
        assert torch.equal(got[:, d0:d0 + step], device.bspmm_csrv(pos, crd, val, part, cols))
        assert torch.equal(summed[:, d0:d0 + step], device.bspmm_csrv(pos, crd, val, part, cols, C[:, d0:d0 + step].contiguous()))
