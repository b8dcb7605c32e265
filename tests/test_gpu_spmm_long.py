"""SpMM rows that spmm_long_kernel takes: lengths around its tiles, columns around its panels, more of them than a block notes
at once; bit for bit against the oracle's sequential loop, or against the matrix that has only those rows."""
import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("idx", [np.int32, np.int64])
@pytest.mark.parametrize("k", [1, 2, 7, 16, 31, 33, 63, 64, 65, 128, 129, 200])
def test_lengths_around_the_tiles(k, idx):
    """A tile is 1152 products: rows of one entry less and more than one, two and three tiles, and of 64 and 65 entries."""
    from lapis_b200 import device
    panels = -(-k // 64)
    tile = 1152 // -(-k // panels)
    rng = np.random.default_rng(k)
    lens = rng.integers(0, 9, 400)
    marks = [n for t in (tile, 2 * tile, 3 * tile) for n in (t - 1, t, t + 1)] + [64, 65, 66, 2500]
    lens[rng.choice(400, len(marks), replace=False)] = marks
    pos = np.zeros(401, idx)
    pos[1:] = np.cumsum(lens)
    cols = 300
    crd, val = rng.integers(0, cols, pos[-1]).astype(idx), rng.uniform(-1, 1, pos[-1])
    B, C = rng.uniform(-1, 1, (cols, k)), rng.uniform(-1, 1, (400, k))
    t = lambda a: torch.as_tensor(a).to(DEV)
    A = device.CsrMatrix(t(pos), t(crd), t(val), (400, cols))
    for accumulate in (True, False):
        want = oracle.spmm(pos, crd, val, B, C if accumulate else np.zeros_like(C))
        assert np.array_equal(A.spmm(t(B), t(C), accumulate=accumulate).cpu().numpy(), want)
    number = np.arange(0, 800, 2).astype(idx)
    D = rng.uniform(-1, 1, (800, k))
    want = D.copy()
    got = device.spmm_dcsr(t(number), t(pos), t(crd), t(val), t(B), t(D), cols).cpu().numpy()
    for r in range(400):  # in place, in entry order
        for j in range(pos[r], pos[r + 1]):
            want[number[r]] = want[number[r]] + val[j] * B[crd[j]]
    assert np.array_equal(got, want)


@pytest.mark.parametrize("k", [1, 33, 130])
def test_more_long_rows_than_a_block_notes_at_once(k):
    """900 long rows placed so that one block meets all of them: the result of the matrix that has only those rows."""
    from lapis_b200 import device
    blocks = torch.cuda.get_device_properties(0).multi_processor_count
    chunks = torch.arange(113, device=DEV) * blocks
    long_rows = (chunks[:, None] * 8 + torch.arange(8, device=DEV)).reshape(-1)[:900]
    rows, cols = int(long_rows[-1]) + 5, 5000
    g = torch.Generator(device=DEV).manual_seed(k)
    lens = torch.zeros(rows, dtype=torch.int64, device=DEV)
    lens[long_rows] = torch.randint(200, 300, (900,), device=DEV, generator=g)
    pos = torch.zeros(rows + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(lens, 0, out=pos[1:])
    nnz = int(pos[-1])
    crd = torch.randint(0, cols, (nnz,), device=DEV, generator=g).to(torch.int32)
    val = torch.rand(nnz, dtype=torch.float64, device=DEV, generator=g) * 2 - 1
    B = torch.rand((cols, k), dtype=torch.float64, device=DEV, generator=g) * 2 - 1
    zero = lambda n: torch.zeros((n, k), dtype=torch.float64, device=DEV)
    pos = pos.to(torch.int32)
    got = device.CsrMatrix(pos, crd, val, (rows, cols)).spmm(B, zero(rows), accumulate=False)
    few = torch.cat([pos[:1], pos[1:][long_rows]])
    want = device.CsrMatrix(few, crd, val, (900, cols)).spmm(B, zero(900), accumulate=False)
    assert torch.equal(got[long_rows], want) and int((got != 0).any(1).sum()) == 900
