"""The one-cluster PCG solver at the edges of its sizes, with rows side by side and, where columns are scattered, one behind the other:
against the launch-per-pass form, which the oracle tests cover."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _passes(A, *args):
    from lapis_b200._lib import check, load
    check(load().lapis_b200_spmv_select_kernel(1, 0, 1))
    try:
        return A.pcg(*args)
    finally:
        check(load().lapis_b200_spmv_select_kernel(0, 0, 0))


def _system(n, per_row, kind):
    """Symmetric, diagonally dominant: `per_row` random columns a row and their mirrors, a band, or scattered columns in every tenth row
    only, between rows that hold just the diagonal."""
    import scipy.sparse as sp
    rng = np.random.default_rng(n + per_row)
    if kind == "band":
        a = sp.diags([rng.uniform(-1, 0, n - d) for d in range(1, per_row + 1)], list(range(1, per_row + 1))).tocsr()
    else:
        rows = np.arange(0, n, 10 if kind == "few" else 1)
        cols = rng.choice(rows, len(rows) * per_row)
        a = sp.coo_matrix((rng.uniform(-1, 0, len(cols)), (np.repeat(rows, per_row), cols)), shape=(n, n)).tocsr()
    a = (a + a.T).tocsr()
    a.setdiag(0)
    a.eliminate_zeros()
    a = (a + sp.diags(np.asarray(abs(a).sum(1)).ravel() + rng.uniform(0.5, 1, n))).tocsr()
    a.sort_indices()
    return a


@pytest.mark.parametrize("idx", [np.int32, np.int64])
@pytest.mark.parametrize("kind,per_row", [("scattered", 1), ("scattered", 2), ("scattered", 3), ("band", 2), ("band", 3), ("few", 7)])
@pytest.mark.parametrize("n", [37, 1024, 1025, 4096, 4097, 8191, 8192, 8193, 12_345, 16_384])
def test_against_the_passes(n, kind, per_row, idx):
    from lapis_b200.device import CsrMatrix
    a = _system(n, per_row, kind)
    assert np.diff(a.indptr).max() <= 32 and a.nnz <= 131_072
    pad = n % 3  # offsets that do not start at zero
    A = CsrMatrix.from_host(a.indptr.astype(idx) + idx(pad), np.concatenate([np.zeros(pad), a.indices]).astype(idx),
                            np.concatenate([np.zeros(pad), a.data]), (n, n))
    rng = np.random.default_rng(1)
    b, dinv = torch.as_tensor(rng.uniform(0, 1, n)).cuda(), torch.as_tensor(1 / a.diagonal()).cuda()
    for tol, maxiter in ((1e-10, 500), (0.0, 1), (0.0, 4)):
        x, it, rel = A.pcg(b, dinv, tol, maxiter)
        again = A.pcg(b, dinv, tol, maxiter)
        x0, it0, rel0 = _passes(A, b, dinv, tol, maxiter)
        assert torch.equal(x, again[0]) and again[1:] == (it, rel)
        assert abs(it - it0) <= 1 and (it != it0 or abs(rel - rel0) <= 1e-6 * rel0)
        assert float((x - x0).norm()) <= (1e-11 if it == it0 else 1e-9) * float(x0.norm())
