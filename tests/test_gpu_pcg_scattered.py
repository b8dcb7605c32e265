"""PCG on small systems with scattered columns, which the one-cluster solver leaves to one cooperative launch, or, where rows are too
long for that on average, to the passes: against the passes, on both sides of the limits."""
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


def _system(n, per_row):
    import scipy.sparse as sp
    rng = np.random.default_rng(n + per_row)
    a = sp.coo_matrix((rng.uniform(-1, 0, per_row * n), (np.repeat(np.arange(n), per_row), rng.integers(0, n, per_row * n))), shape=(n, n)).tocsr()
    a = (a + a.T).tocsr()
    a.setdiag(0)
    a.eliminate_zeros()
    a = (a + sp.diags(np.asarray(abs(a).sum(1)).ravel() + 1)).tocsr()
    a.sort_indices()
    return a


def _far(a):
    """Gathers from another block's slice of p: eight blocks, of 512, 1024 or 2048 rows."""
    n = a.shape[0]
    rows = 512 if n <= 4096 else 1024 if n <= 8192 else 2048
    return int((a.indices // rows != np.repeat(np.arange(n), np.diff(a.indptr)) // rows).sum())


@pytest.mark.parametrize("idx", [np.int32, np.int64])
@pytest.mark.parametrize("n,per_row,form", [
    (3000, 7, "cluster"), (4000, 7, "launch"), (4000, 8, "cluster"), (4000, 9, "passes"), (5500, 2, "cluster"), (5500, 3, "launch"), (8000, 5, "launch"),
    (16_000, 2, "launch")])
def test_against_the_passes(n, per_row, form, idx):
    from lapis_b200.device import CsrMatrix
    a = _system(n, per_row)
    assert np.diff(a.indptr).max() <= 32 and a.nnz <= 131_072
    limit = 60_000 if a.nnz > 16 * n else 36_000 if n <= 4096 else 24_000
    assert (form == "cluster") == (_far(a) <= limit)
    assert (form == "passes") == (form != "cluster" and a.nnz > 16 * n)
    A = CsrMatrix.from_host(a.indptr.astype(idx), a.indices.astype(idx), a.data, (n, n))
    rng = np.random.default_rng(1)
    b, dinv = torch.as_tensor(rng.uniform(0, 1, n)).cuda(), torch.as_tensor(1 / a.diagonal()).cuda()
    for tol, maxiter in ((1e-10, 500), (0.0, 1), (0.0, 9)):
        x, it, rel = A.pcg(b, dinv, tol, maxiter)
        again = A.pcg(b, dinv, tol, maxiter)
        x0, it0, rel0 = _passes(A, b, dinv, tol, maxiter)
        assert torch.equal(x, again[0]) and again[1:] == (it, rel)
        assert it == it0 and abs(rel - rel0) <= 1e-6 * rel0
        assert float((x - x0).norm()) <= 1e-11 * float(x0.norm())
