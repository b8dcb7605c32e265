"""PCG in one cooperative launch (pcg_grid.cu): against the launch-per-pass form, which the oracle tests cover."""
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


def _system(n, per_row, idx, seed, base=0):
    """Diagonally dominant, symmetric pattern not needed for the comparison: `per_row` scattered columns and the diagonal."""
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    half = sp.coo_matrix((rng.uniform(-1, 0, per_row * n), (np.repeat(np.arange(n), per_row), rng.integers(0, n, per_row * n))), shape=(n, n)).tocsr()
    a = (half + half.T).tocsr()
    a -= sp.diags(a.diagonal())
    a = (a + sp.diags(np.asarray(abs(a).sum(1)).ravel() + rng.uniform(0.5, 1, n))).tocsr()
    a.sort_indices()
    return a


@pytest.mark.parametrize("idx", [np.int32, np.int64])
@pytest.mark.parametrize("n,per_row", [(16_385, 2), (20_000, 5), (75_776, 2), (75_777, 1), (151_553, 3), (303_104, 2), (303_105, 2)])
def test_against_the_passes(n, per_row, idx):
    """From the smallest to beyond the largest: one, two and four rows a thread, partly empty blocks; the same bits again."""
    from lapis_b200.device import CsrMatrix
    a = _system(n, per_row, idx, n)
    assert np.diff(a.indptr).max() <= 32
    rng = np.random.default_rng(1)
    A = CsrMatrix.from_host(a.indptr.astype(idx), a.indices.astype(idx), a.data, (n, n))
    b, dinv = torch.as_tensor(rng.uniform(0, 1, n)).cuda(), torch.as_tensor(1 / a.diagonal()).cuda()
    for tol, maxiter in ((1e-8, 1000), (0.0, 1), (0.0, 6)):
        x, it, rel = A.pcg(b, dinv, tol, maxiter)
        again = A.pcg(b, dinv, tol, maxiter)
        x0, it0, rel0 = _passes(A, b, dinv, tol, maxiter)
        assert torch.equal(x, again[0]) and again[1:] == (it, rel)
        assert it == it0 and abs(rel - rel0) <= 1e-6 * rel0
        assert float((x - x0).norm()) <= 1e-11 * float(x0.norm())


def test_over_several_launches_and_offsets():
    """4200 iterations, more than one launch makes, on a matrix whose offsets do not start at zero."""
    from lapis_b200 import workloads
    from lapis_b200.device import CsrMatrix
    d = workloads.pcg_laplacian(150)
    n = 150 * 150
    pad = 7
    A = CsrMatrix.from_host(d["pos"] + pad, np.concatenate([np.zeros(pad, d["crd"].dtype), d["crd"]]), np.concatenate([np.zeros(pad), d["val"]]), (n, n))
    b, dinv = torch.as_tensor(d["b"]).cuda(), torch.as_tensor(d["dinv"]).cuda()
    x, it, rel = A.pcg(b, dinv, 0.0, 4200)
    assert it == 4200 and 0 <= rel < 1e-14
    y, _, _ = A.pcg(b, dinv, 1e-12, 4000)
    assert float((x - y).norm()) <= 1e-8 * float(y.norm())
    z, itz, relz = _passes(A, b, dinv, 1e-12, 4000)
    assert float((z - y).norm()) <= 1e-9 * float(y.norm())


@pytest.mark.parametrize("at,value", [(None, 0.0), (19_999, float("nan")), (5, float("inf")), (0, float("-inf"))])
def test_special_right_hand_sides(at, value):
    import scipy.sparse as sp
    from lapis_b200.device import CsrMatrix
    n = 20_000
    a = sp.diags([-np.ones(n - 1), np.full(n, 2.5), -np.ones(n - 1)], [-1, 0, 1]).tocsr()
    A = CsrMatrix.from_host(a.indptr.astype(np.int32), a.indices.astype(np.int32), a.data, (n, n))
    dinv = torch.full((n,), 0.4, dtype=torch.float64, device="cuda")
    b = torch.full((n,), 0.0 if at is None else 1.0, dtype=torch.float64, device="cuda")
    if at is not None:
        b[at] = value
    (x, it, rel), (x0, it0, rel0) = A.pcg(b, dinv, 1e-8, 50), _passes(A, b, dinv, 1e-8, 50)
    assert it == it0 == 1 and np.isnan(rel) and np.isnan(rel0)
    assert torch.equal(torch.isnan(x), torch.isnan(x0)) and torch.equal(torch.nan_to_num(x), torch.nan_to_num(x0))


def test_solves_on_two_streams_and_beside_other_work():
    from lapis_b200 import workloads
    from lapis_b200.device import CsrMatrix
    import threading
    d = workloads.pcg_laplacian(200)
    n = 200 * 200
    A = CsrMatrix.from_host(d["pos"], d["crd"], d["val"], (n, n))
    b, dinv = torch.as_tensor(d["b"]).cuda(), torch.as_tensor(d["dinv"]).cuda()
    want = A.pcg(b, dinv, 1e-10, 2000)
    got, other = [], torch.rand((2048, 2048), device="cuda")

    def solve(stream):
        with torch.cuda.stream(stream):
            for _ in range(3):
                other @ other
                got.append(A.pcg(b, dinv, 1e-10, 2000))
    torch.cuda.synchronize()
    threads = [threading.Thread(target=solve, args=(torch.cuda.Stream(),)) for _ in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert len(got) == 9 and all(torch.equal(x, want[0]) and (it, rel) == want[1:] for x, it, rel in got)
