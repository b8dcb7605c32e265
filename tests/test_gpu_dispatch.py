"""Kernels chosen by size: each one at the edges of the range it is chosen for (needs a B200)."""
import numpy as np
import pytest
import torch

from lapis_b200 import workloads as w
from oracle import oracle

pytestmark = pytest.mark.gpu


def _dev():
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the gpu-marked tests must run on a GPU box")
    return torch.device("cuda:0")


def _csr(rng, lens, ncols, idx):
    pos, crd = w.random_csr_from_lengths(np.asarray(lens), ncols, rng, idx)
    return pos, crd, rng.uniform(-1, 1, crd.size)


@pytest.mark.parametrize("hint", [2, 3, 4], ids=["thread", "block64", "block32"])
@pytest.mark.parametrize("rows", [1, 31, 33, 64, 65, 1000])
def test_short_row_kernels_share_their_bits(rows, hint):
    """Rows of 0 to 32 entries, a block of rows that starts anywhere in the arrays (pos[0] != 0), rows that cross a
    2048-entry boundary: the bits of the chunk kernel, which the oracle tests cover."""
    from lapis_b200._lib import check, load
    from lapis_b200.device import CsrMatrix
    dev, lib = _dev(), load()
    rng = np.random.default_rng(rows)
    ncols, first = 700, 5
    lens = rng.integers(0, 33, rows + first)
    lens[first] = 32
    for idx in (np.int32, np.int64):
        pos, crd, val = (torch.as_tensor(a).to(dev) for a in _csr(rng, lens, ncols, idx))
        A = CsrMatrix(pos[first:], crd, val, (rows, ncols))
        x = torch.as_tensor(rng.uniform(-1, 1, ncols)).to(dev)
        y0 = torch.as_tensor(rng.uniform(-1, 1, rows)).to(dev)
        got, want = [], []
        for kernel, out in ((256, want), (1, got)):
            check(lib.lapis_b200_spmv_select_kernel(kernel, 4 if kernel > 1 else 0, hint if kernel == 1 else 1))
            try:
                out += [A.spmv(x, y0.clone(), accumulate=acc) for acc in (True, False)]
            finally:
                check(lib.lapis_b200_spmv_select_kernel(0, 0, 0))
        got += [A.spmv(x, y0.clone(), accumulate=acc) for acc in (True, False)]  # untuned: the rule's choice
        for g, v in zip(got, want + want):
            assert torch.equal(g, v)


def test_launches_that_overlap_see_each_others_results():
    """Back-to-back calls may start before the call in front has drained; a chain in which every call reads what the
    one before wrote gives the bits of the same chain with a synchronisation between calls."""
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    rng = np.random.default_rng(3)
    for lens in (np.full(3000, 9), np.r_[np.full(3000, 9), 700]):
        n = len(lens)
        pos, crd, val = _csr(rng, lens, n, np.int64)
        A = CsrMatrix.from_host(pos, crd, val / 9, (n, n), dev)
        v = torch.as_tensor(rng.uniform(-1, 1, n)).to(dev)
        ends = []
        for sync in (True, False):
            a, b = v.clone(), torch.zeros_like(v)
            for _ in range(40):
                A.spmv(a, b, accumulate=True)
                if sync:
                    torch.cuda.synchronize()
                a, b = b, a
            ends.append(a)
        assert torch.equal(ends[0], ends[1])
        assert bool(torch.isfinite(ends[0]).all())


@pytest.mark.parametrize("rows,mean,pinned", [(1, 1, False), (900, 4, False), (30_000, 9, False), (300_000, 5, False), (300_000, 5, True)])
def test_host_arrays_travel_in_pieces(rows, mean, pinned):
    """Calls on host arrays from one piece to more than the staging ring holds, pageable and page-locked: the result of
    the resident call, bad indices found wherever they are, and y untouched then."""
    from lapis_b200 import KokkosBackend as KB
    from lapis_b200 import modules as mm
    from lapis_b200._lib import LapisError
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    rng = np.random.default_rng(rows)
    pos, crd, val = _csr(rng, np.full(rows, min(mean, rows)), rows, np.int64)
    x, y = rng.uniform(-1, 1, rows), rng.uniform(-1, 1, rows)
    want = CsrMatrix.from_host(pos, crd, val, (rows, rows), dev).spmv(torch.as_tensor(x).to(dev), torch.as_tensor(y).to(dev)).cpu().numpy()
    module = KB.KokkosBackend(decompose_tensors=True).compile(mm.spmv(mm.CSR64))
    spec = ((rows, rows), (rows + 1, len(crd), len(crd)))
    if pinned:
        pos, crd, val, x, y = (torch.as_tensor(a).pin_memory().numpy() for a in (pos, crd, val, x, y))
    y0 = y.copy()
    module.spmv(pos, crd, val, spec, x, y)
    assert np.array_equal(y, want)
    y[:] = y0
    for at, bad in ((0, rows), (len(crd) // 2, -1), (len(crd) - 1, rows)):
        keep, crd[at] = crd[at], bad
        with pytest.raises(LapisError, match="column index out of range"):
            module.spmv(pos, crd, val, spec, x, y)
        crd[at] = keep
    for at in {1, rows // 2, rows} - {0}:
        keep, pos[at] = pos[at], pos[at - 1] - 1
        with pytest.raises(LapisError, match="pos"):
            module.spmv(pos, crd, val, spec, x, y)
        pos[at] = keep
    assert np.array_equal(y, y0)
