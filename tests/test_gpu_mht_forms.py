"""Hitting-time moments on graphs on either side of the rules that choose between two passes and four launches an iteration, against
the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def _graph(n, half, kind):
    """Symmetric weights: `half` random columns a row and their mirrors, a band, or a band of which every column is moved away in every
    second row."""
    import scipy.sparse as sp
    rng = np.random.default_rng(n + half)
    if kind == "scattered":
        r, c = np.repeat(np.arange(n), half), rng.integers(0, n, n * half)
    else:
        r = np.tile(np.arange(n), half)
        c = (r + np.repeat(np.arange(1, half + 1), n)) % n
        if kind == "moved":
            c = np.where(r % 2 == 0, c, (c + n // 2) % n)
    keep = r != c
    a = sp.coo_matrix((rng.uniform(0.5, 1.5, keep.sum()), (r[keep], c[keep])), shape=(n, n)).tocsr()
    a = (a + a.T).tocsr()
    a.sort_indices()
    return a


@pytest.mark.parametrize("idx", [np.int32, np.int64])
@pytest.mark.parametrize("n,half,kind", [
    (130_000, 2, "scattered"), (131_072, 2, "scattered"), (200_000, 3, "scattered"), (100_000, 4, "scattered"),  # around 2^19 entries, six a row
    (300_000, 2, "scattered"), (300_001, 2, "scattered"),                                                        # most rows
    (300_001, 2, "band"), (100_000, 8, "band"), (320_000, 8, "band"), (320_000, 9, "band"), (150_000, 6, "moved"), (300_001, 1, "moved")])
def test_against_the_oracle(n, half, kind, idx):
    from lapis_b200.device import CsrMatrix
    a = _graph(n, half, kind)
    assert np.diff(a.indptr).max() <= 32
    d = np.asarray(a.sum(axis=1)).ravel() + 1e-3
    mask = np.ones(n)
    mask[np.random.default_rng(1).choice(n, size=n // 100, replace=False)] = 0.0
    pad = half % 3  # offsets that do not start at zero
    A = CsrMatrix.from_host(a.indptr.astype(idx) + idx(pad), np.concatenate([np.zeros(pad), a.indices]).astype(idx),
                            np.concatenate([np.zeros(pad), a.data]), (n, n))
    A.tune()
    args = [torch.as_tensor(t).cuda() for t in (mask, d)]
    m1, m2 = A.mht(*args, 0.95, 1e-9, 60)
    want1, _ = oracle.mht(a.indptr, a.indices, a.data, mask, d, 0.95, 1e-9, 60)
    assert np.linalg.norm(m1.cpu().numpy() - want1) <= 1e-8 * np.linalg.norm(want1)
    n1, n2 = A.mht(*args, 0.95, 1e-9, 60)
    assert torch.equal(m1, n1) and torch.equal(m2, n2)
    assert torch.equal(A.mht(*args, 0.95, 1e-9, 60, info=True)[0], m1)
