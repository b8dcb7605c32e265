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


@pytest.mark.parametrize("batch,m,n,k", [
    (1, 1, 1, 1), (1, 63, 65, 15), (1, 64, 64, 16), (1, 65, 63, 17), (1, 130, 1028, 100), (1, 33, 31, 900), (1, 1000, 1100, 49),  # one product
    (300, 33, 65, 31), (300, 30, 20, 52), (2000, 4, 5, 6), (150, 64, 40, 33), (65540, 2, 3, 4), (200, 20, 100, 7), (3, 40, 40, 0)])  # batches
def test_general_shape_matmul_tiles(batch, m, n, k):
    """Every tile the rule picks, at the edges of tiles and k-slabs, with and without 16-byte accesses: k ascending, the
    product and the sum rounded separately, C last, bit for bit."""
    from lapis_b200 import device
    dev = _dev()
    g = torch.Generator(device=dev).manual_seed(m * n + k)
    A, B, C = (torch.rand(s, generator=g, device=dev) * 2 - 1 for s in ((batch, m, k), (batch, k, n), (batch, m, n)))
    want = torch.zeros_like(C)
    for i in range(k):  # a product and a sum per k, as torch rounds them
        want = want + A[:, :, i, None] * B[:, i, None, :]
    want = want + C
    shifted = torch.empty(C.numel() + 1, device=dev)[1:].view_as(C)  # C off the 16-byte boundary
    shifted.copy_(C)
    assert torch.equal(device.bgemm(A, B, C), want)
    assert torch.equal(device.bgemm(A, B, shifted), want)


def test_general_shape_matmul_special_values():
    """Signed zeros, infinities and NaN as the sequential loop has them (padding of the last slab adds nothing)."""
    from lapis_b200 import device
    dev = _dev()
    A = torch.tensor([[0.0, -0.0, float("inf")], [-0.0, -1.0, 0.0], [1e-40, 3e38, float("nan")]], device=dev)
    B = torch.tensor([[-0.0, 1.0], [0.0, 3e38], [1.0, -0.0]], device=dev)
    C = torch.tensor([[-0.0, 1.0], [-0.0, -0.0], [0.0, -0.0]], device=dev)
    want = torch.zeros_like(C)
    for i in range(3):
        want = want + A[:, i, None] * B[i, None, :]
    want = want + C
    got = device.bgemm(A, B, C)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    ok = ~torch.isnan(want)
    assert torch.equal(got[ok].view(torch.int32), want[ok].view(torch.int32))


def _lens_with_long_rows(rng, rows):
    lens = rng.integers(0, 21, rows)
    for at, n in zip(rng.choice(rows, 7, replace=False), (255, 256, 257, 300, 1025, 2048, 2500)):
        lens[at] = n
    lens[-1], lens[rows // 2:rows // 2 + 4] = 400, 500  # the last row, neighbours
    return lens


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 13, 16, 17, 31, 32, 33, 37, 64, 65, 66, 97, 101, 130, 260])
def test_spmm_group_sizes_and_long_rows(k):
    """Every width the rule tells apart, rows on both sides of the limit for long rows, a block of rows that starts inside
    the arrays, CSR and DCSR (with repeated row numbers), operands on and off 16-byte boundaries: bit for bit."""
    from lapis_b200.device import CsrMatrix, spmm_dcsr
    dev = _dev()
    rng = np.random.default_rng(k)
    rows, ncols, first = 700, 3000, 5
    for idx in (np.int32, np.int64):
        pos, crd, val = _csr(rng, _lens_with_long_rows(rng, rows + first), ncols, idx)
        B, C = rng.uniform(-1, 1, (ncols, k)), rng.uniform(-1, 1, (rows, k))
        numbers = np.sort(rng.choice(2 * rows, rows)).astype(idx)  # ascending, some twice
        C2 = rng.uniform(-1, 1, (2 * rows, k))
        d = [torch.as_tensor(a).to(dev) for a in (pos, crd, val)]
        for shift in (0, 1):
            flat = torch.empty(B.size + shift, dtype=torch.float64, device=dev)
            Bd = flat[shift:].view(ncols, k)
            Bd.copy_(torch.as_tensor(B))
            for lo in (0, first):
                A = CsrMatrix(d[0][lo:lo + rows + 1], d[1], d[2], (rows, ncols))
                for acc in (True, False):
                    # the handle takes the entries that pos names; the oracle reads the same arrays
                    want = oracle.spmm(pos[lo:lo + rows + 1], crd, val, B, C if acc else np.zeros_like(C))
                    assert np.array_equal(A.spmm(Bd, torch.as_tensor(C).to(dev), accumulate=acc).cpu().numpy(), want)
            p2 = pos[first:rows + first + 1]
            want = oracle.spmm_dcsr(numbers, p2, crd, val, B, C2)
            got = spmm_dcsr(torch.as_tensor(numbers).to(dev), torch.as_tensor(p2).to(dev), d[1], d[2], Bd, torch.as_tensor(C2).to(dev), ncols)
            assert np.array_equal(got.cpu().numpy(), want)


def test_spmm_with_long_rows_in_a_chain():
    """The two kernels of a product with long rows overlap; the next product reads what both wrote."""
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    rng = np.random.default_rng(1)
    n, k = 3000, 20
    pos, crd, val = _csr(rng, _lens_with_long_rows(rng, n), n, np.int32)
    A = CsrMatrix.from_host(pos, crd, val / 50, (n, n), dev)
    start = torch.as_tensor(rng.uniform(-1, 1, (n, k))).to(dev)
    ends = []
    for sync in (True, False):
        a, b = start.clone(), torch.zeros_like(start)
        for _ in range(30):
            A.spmm(a, b, accumulate=False)
            if sync:
                torch.cuda.synchronize()
            a, b = b, a
        ends.append(a)
    assert torch.equal(ends[0], ends[1])


@pytest.mark.parametrize("n", [1, 2, 31, 1000, 1024, 1025, 4096, 4097, 8193, 16384])
def test_small_pcg_against_the_passes(n):
    """Systems solved in one launch: the iterations and the solution of the launch-per-pass form (taken when an SpMV kernel is
    forced), which the oracle tests cover; the same bits on a second run."""
    from lapis_b200._lib import check, load
    from lapis_b200.device import CsrMatrix
    dev, lib = _dev(), load()
    rng = np.random.default_rng(n)
    import scipy.sparse as sp
    half = sp.random(n, n, min(1.0, 2.0 / n), random_state=rng, format="csr") if n > 2 else sp.csr_matrix((n, n))
    sym = (half + half.T).tocsr()
    for idx in (np.int32, np.int64):
        a = (sym + sp.diags(np.asarray(abs(sym).sum(1)).ravel() + rng.uniform(0.5, 1, n))).tocsr()
        a.sort_indices()
        A = CsrMatrix.from_host(a.indptr.astype(idx), a.indices.astype(idx), a.data, (n, n), dev)
        b, dinv = torch.as_tensor(rng.uniform(0, 1, n)).to(dev), torch.as_tensor(1 / a.diagonal()).to(dev)
        for tol, maxiter in ((1e-8, 1000), (0.0, 1), (0.0, 5)):
            x, it, rel = A.pcg(b, dinv, tol, maxiter)
            again = A.pcg(b, dinv, tol, maxiter)
            check(lib.lapis_b200_spmv_select_kernel(1, 0, 1))
            try:
                x0, it0, rel0 = A.pcg(b, dinv, tol, maxiter)
            finally:
                check(lib.lapis_b200_spmv_select_kernel(0, 0, 0))
            assert torch.equal(x, again[0]) and again[1] == it and (again[2] == rel or rel != rel)
            if n <= 2:  # solved exactly after one step or two: what is left is rounding, then 0 / 0
                continue
            assert it == it0
            # a dominant diagonal amplifies the rounding of a dot product little
            assert float((x - x0).norm()) <= 1e-11 * float(x0.norm()) and abs(rel - rel0) <= 1e-6 * rel0 + 1e-15


def test_small_pcg_over_several_launches():
    """More iterations than one launch makes: the state carried from launch to launch gives the count asked for and the
    solution (tol 0 goes on past convergence; 4096 iterations a launch)."""
    from lapis_b200 import workloads
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    d = workloads.pcg_laplacian(128)
    A = CsrMatrix.from_host(d["pos"], d["crd"], d["val"], (128 * 128,) * 2, dev)
    b, dinv = torch.as_tensor(d["b"]).to(dev), torch.as_tensor(d["dinv"]).to(dev)
    x, it, rel = A.pcg(b, dinv, 0.0, 4200)
    assert it == 4200 and 0 <= rel < 1e-14
    y, _, _ = A.pcg(b, dinv, 1e-12, 4000)
    assert float((x - y).norm()) <= 1e-8 * float(y.norm())


@pytest.mark.parametrize("nh,dh", [(1, 1), (1, 5), (1, 8), (1, 64), (2, 9), (2, 10), (3, 20), (3, 43), (4, 1), (4, 4), (4, 5), (4, 17), (5, 13), (6, 64),
                                   (7, 33), (8, 30), (8, 64), (11, 40), (12, 47), (13, 41), (15, 128)])
def test_bspmm_widths(nh, dh):
    """Every width the rule tells apart, operands on and off 16-byte boundaries: bit for bit."""
    from lapis_b200.device import bspmm_csrv
    dev = _dev()
    rng = np.random.default_rng(nh * dh)
    n = 333
    for idx in (np.int32, np.int64):
        pos, crd, _ = _csr(rng, rng.integers(0, 23, n), n, idx)
        val, B = rng.uniform(-1, 1, crd.size * nh).astype(np.float32), rng.uniform(-1, 1, (n, dh, nh)).astype(np.float32)
        want = oracle.bspmm(pos, crd, val, B)
        for shift in (0, 1):
            v, b = (torch.empty(a.size + shift, dtype=torch.float32, device=dev)[shift:].view(a.shape) for a in (val, B))
            v.copy_(torch.as_tensor(val))
            b.copy_(torch.as_tensor(B))
            got = bspmm_csrv(torch.as_tensor(pos).to(dev), torch.as_tensor(crd).to(dev), v, b, n)
            assert np.array_equal(got.cpu().numpy(), want)


def test_calls_that_wait_for_the_queue_leave_python_running():
    """A launch waits where the stream's queue is full (about a thousand launches); other Python threads go on meanwhile."""
    import threading
    import time
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    rng = np.random.default_rng(0)
    n = 64
    A = CsrMatrix.from_host(*_csr(rng, np.full(n, 3), n, np.int32), (n, n), dev)
    x, y = (torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(2))
    A.spmv(x, y)
    torch.cuda.synchronize()
    gaps, stop = [], threading.Event()

    def other():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.0005)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    thread = threading.Thread(target=other)
    thread.start()
    torch.cuda._sleep(int(1e9))  # half a second of GPU time
    start = time.perf_counter()
    for _ in range(4000):
        A.spmv(x, y)
    waited = time.perf_counter() - start
    stop.set()
    thread.join()
    torch.cuda.synchronize()
    assert waited > 0.2, "the queue never filled up"
    assert max(gaps) < 0.5 * waited


def test_tuning_beside_calls_on_host_arrays():
    """A thread that tunes a matrix leaves the kernel choice of other threads' calls alone: a call on host arrays of short
    rows makes no plan for the kernels that need one."""
    import threading
    from lapis_b200 import KokkosBackend as KB
    from lapis_b200 import modules as mm
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    rng = np.random.default_rng(5)
    n = 5000
    pos, crd, val = _csr(rng, np.full(n, 9), n, np.int64)
    x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    A = CsrMatrix.from_host(pos, crd, val, (n, n), dev)
    want = A.spmv(torch.as_tensor(x).to(dev), torch.as_tensor(y).to(dev)).cpu().numpy()  # every kind of kernel has these bits
    module = KB.KokkosBackend(decompose_tensors=True).compile(mm.spmv(mm.CSR64))
    stop = threading.Event()

    def tune():
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            while not stop.is_set():
                A.tune()

    thread = threading.Thread(target=tune)
    thread.start()
    try:
        for _ in range(300):
            got = y.copy()
            module.spmv(pos, crd, val, ((n, n), (n + 1, len(crd), len(crd))), x, got)
            assert np.array_equal(got, want)
    finally:
        stop.set()
        thread.join()


@pytest.mark.parametrize("n,idx", [(30_000, np.int32), (60_000, np.int64)])
def test_solver_passes_have_their_own_kernel(n, idx):
    """Rows of 10 to 32 scattered entries on both sides of the limit for launch-bound systems: an untuned matrix above it
    runs the chunk kernel, which needs the direction pass; tuned or not, PCG makes the oracle's iterations."""
    import scipy.sparse as sp
    from lapis_b200._lib import load
    from lapis_b200.device import CsrMatrix
    dev, lib = _dev(), load()
    rng = np.random.default_rng(n)
    half = sp.coo_matrix((rng.uniform(-1, 0, 5 * n), (np.repeat(np.arange(n), 5), rng.integers(0, n, 5 * n))), shape=(n, n)).tocsr()
    sym = (half + half.T).tocsr()
    sym -= sp.diags(sym.diagonal())
    a = (sym + sp.diags(np.asarray(abs(sym).sum(1)).ravel() + 1.0)).tocsr()
    a.sort_indices()
    assert 10 <= np.diff(a.indptr).max() <= 32
    A = CsrMatrix.from_host(a.indptr.astype(idx), a.indices.astype(idx), a.data, (n, n), dev)
    assert bool(lib.lapis_b200_pcg_folds_direction(A.handle)) == (a.nnz < 1 << 19)
    b, dinv = rng.uniform(0, 1, n), 1 / a.diagonal()
    x0, it0, rel0 = oracle.pcg(a.indptr.astype(idx), a.indices.astype(idx), a.data, b, dinv, 1e-10, 500)
    for tune in (False, True):
        if tune:
            A.tune()
        for maxiter in (500, 8):  # a short solve does not tune
            x, it, rel = A.pcg(torch.as_tensor(b).to(dev), torch.as_tensor(dinv).to(dev), 1e-10, maxiter)
            assert it == min(it0, maxiter)
            if maxiter == 500:
                assert abs(rel - rel0) <= 1e-6 * rel0 and np.linalg.norm(x.cpu().numpy() - x0) <= 1e-11 * np.linalg.norm(x0)


def _passes(A, *args):
    """PCG in a launch per pass, whatever the size."""
    from lapis_b200._lib import check, load
    check(load().lapis_b200_spmv_select_kernel(1, 0, 1))
    try:
        return A.pcg(*args)
    finally:
        check(load().lapis_b200_spmv_select_kernel(0, 0, 0))


@pytest.mark.parametrize("idx", [np.int32, np.int64])
@pytest.mark.parametrize("n,half,scattered", [(8000, 7, True), (16000, 3, True), (8000, 7, False), (4096, 15, False)])
def test_small_pcg_leaves_scattered_systems_to_the_passes(n, half, scattered, idx):
    """More than 75,000 entries: solved in one launch where most columns are near the diagonal, by the passes (their bits)
    where they are not."""
    import scipy.sparse as sp
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    rng = np.random.default_rng(n + half)
    if scattered:
        a = sp.coo_matrix((rng.uniform(-1, 0, half * n), (np.repeat(np.arange(n), half), rng.integers(0, n, half * n))), shape=(n, n)).tocsr()
    else:
        a = sp.diags([rng.uniform(-1, 0, n - d) for d in range(1, half + 1)], list(range(1, half + 1))).tocsr()
    a = (a + a.T).tocsr()
    a -= sp.diags(a.diagonal())
    a = (a + sp.diags(np.asarray(abs(a).sum(1)).ravel() + 1.0)).tocsr()
    a.sort_indices()
    assert 75_000 < a.nnz <= 131_072 and np.diff(a.indptr).max() <= 32
    A = CsrMatrix.from_host(a.indptr.astype(idx), a.indices.astype(idx), a.data, (n, n), dev)
    b, dinv = torch.as_tensor(rng.uniform(0, 1, n)).to(dev), torch.as_tensor(1 / a.diagonal()).to(dev)
    for tol, maxiter in ((1e-9, 500), (0.0, 3)):
        (x, it, rel), (x0, it0, rel0) = A.pcg(b, dinv, tol, maxiter), _passes(A, b, dinv, tol, maxiter)
        assert it == it0 and abs(rel - rel0) <= 1e-6 * rel0
        assert float((x - x0).norm()) <= 1e-11 * float(x0.norm())
        assert bool(torch.equal(x, x0)) or not scattered


@pytest.mark.parametrize("n", [5, 1024, 5000, 16384])
def test_small_pcg_special_right_hand_sides(n):
    """A zero right-hand side, infinities and NaN stop after the iterations that the passes make, with the same values."""
    import scipy.sparse as sp
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    a = sp.diags([-np.ones(n - 1), np.full(n, 2.5), -np.ones(n - 1)], [-1, 0, 1]).tocsr()
    A = CsrMatrix.from_host(a.indptr.astype(np.int32), a.indices.astype(np.int32), a.data, (n, n), dev)
    dinv = torch.full((n,), 0.4, dtype=torch.float64, device=dev)
    for at, value in ((None, 0.0), (n - 1, float("nan")), (n // 2, float("inf")), (0, float("-inf"))):
        b = torch.full((n,), 0.0 if at is None else 1.0, dtype=torch.float64, device=dev)
        if at is not None:
            b[at] = value
        (x, it, rel), (x0, it0, rel0) = A.pcg(b, dinv, 1e-8, 50), _passes(A, b, dinv, 1e-8, 50)
        assert it == it0 == 1 and np.isnan(rel) and np.isnan(rel0)
        assert torch.equal(torch.isnan(x), torch.isnan(x0)) and torch.equal(torch.nan_to_num(x), torch.nan_to_num(x0))


@pytest.mark.parametrize("kernel", [(1, 0, 2), (1, 0, 3), (1, 0, 4), (256, 4, 1), (512, 3, 0), (-256, 3, 1), (2, 5, 1), (3, 4, 0), (4, 0, 0)], ids=str)
def test_products_read_the_values_that_the_one_before_wrote(kernel):
    """Overlapped launches of every kernel: the result of a product is the next one's vector and then its matrix values."""
    from lapis_b200._lib import check, load
    from lapis_b200.device import CsrMatrix
    dev, lib = _dev(), load()
    rng = np.random.default_rng(7)
    n, mean = 4000, 9
    pos, crd, val = (torch.as_tensor(a).to(dev) for a in _csr(rng, np.full(n, mean), n, np.int64))
    wide = CsrMatrix.from_host(*_csr(rng, np.full(n * mean, 3), n, np.int64), (n * mean, n), dev)  # y of this: the values of that
    ends = []
    check(lib.lapis_b200_spmv_select_kernel(*kernel))
    try:
        for sync in (True, False):
            v = val.clone()
            A = CsrMatrix(pos, crd, v, (n, n))
            a, b = torch.ones(n, dtype=torch.float64, device=dev), torch.zeros(n, dtype=torch.float64, device=dev)
            for _ in range(30):
                for call in (lambda: A.spmv(a, b, accumulate=False), lambda: wide.spmv(b, v, accumulate=False)):
                    call()
                    if sync:
                        torch.cuda.synchronize()
                v.clamp_(-1, 1)
                a, b = b, a
            ends.append((a, v))
    finally:
        check(lib.lapis_b200_spmv_select_kernel(0, 0, 0))
    assert torch.equal(ends[0][0], ends[1][0]) and torch.equal(ends[0][1], ends[1][1])
    assert bool(torch.isfinite(ends[0][0]).all())


@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("k,rows", [(16, 110_000), (65, 30_000)])
def test_spmm_at_the_limit_for_long_rows(k, rows, over):
    """The longest row at and just above what the kernel beside the main one takes: the host's rule and the kernels' agree."""
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    rng = np.random.default_rng(k)
    lens = np.full(rows, 16)
    rule = lambda nnz: max(256, (nnz * (k + 8) // ((k + 63) // 64)) >> 17)
    longest = 256
    while longest < rule(16 * (rows - 3) + 3 * longest) + over:
        longest += 1
    lens[[0, rows // 2, rows - 1]] = longest
    assert (longest > rule(int(lens.sum()))) == bool(over)
    pos, crd, val = _csr(rng, lens, rows, np.int32)
    B, C = rng.uniform(-1, 1, (rows, k)), rng.uniform(-1, 1, (rows, k))
    A = CsrMatrix.from_host(pos, crd, val, (rows, rows), dev)
    got = A.spmm(torch.as_tensor(B).to(dev), torch.as_tensor(C).to(dev))
    assert np.array_equal(got.cpu().numpy(), oracle.spmm(pos, crd, val, B, C))


@pytest.mark.parametrize("k", [1, 3, 8, 64, 101])
def test_spmm_special_values(k):
    """Infinities and NaN in values and operands, short and long rows, empty rows and an all-zero product: what the
    sequential loop makes of them, and nothing of them in the rows beside."""
    from lapis_b200.device import CsrMatrix, spmm_dcsr
    dev = _dev()
    rng = np.random.default_rng(k)
    rows, ncols = 300, 900
    lens = rng.integers(0, 12, rows)
    lens[[3, 150, 299]] = (700, 301, 513)
    for idx in (np.int32, np.int64):
        pos, crd, val = _csr(rng, lens, ncols, idx)
        for v in (np.inf, -np.inf, np.nan, -0.0):
            val[rng.integers(0, val.size, 6)] = v
        B, C = rng.uniform(-1, 1, (ncols, k)), rng.uniform(-1, 1, (rows, k))
        for v in (np.inf, np.nan, 0.0):
            B[rng.integers(0, ncols, 9), rng.integers(0, k, 9)] = v
        d = [torch.as_tensor(a).to(dev) for a in (pos, crd, val)]
        with np.errstate(all="ignore"):
            want = oracle.spmm(pos, crd, val, B, C)
        assert 0 < np.isnan(want).sum() < want.size
        got = [CsrMatrix(*d, (rows, ncols)).spmm(torch.as_tensor(B).to(dev), torch.as_tensor(C).to(dev)),
               spmm_dcsr(torch.arange(rows, device=dev, dtype=d[0].dtype), *d, torch.as_tensor(B).to(dev), torch.as_tensor(C).to(dev), ncols)]
        wants = [want, oracle.spmm_dcsr(np.arange(rows).astype(idx), pos, crd, val, B, C)]
        for g, w_ in zip(got, wants):
            assert np.array_equal(g.cpu().numpy(), w_, equal_nan=True)


def test_calls_on_host_arrays_from_two_threads():
    """Two threads in calls at once, operands of one piece and of more than the staging ring holds: each gets its own result."""
    import threading
    from lapis_b200 import KokkosBackend as KB
    from lapis_b200 import modules as mm
    from lapis_b200.device import CsrMatrix
    dev = _dev()
    module = KB.KokkosBackend(decompose_tensors=True).compile(mm.spmv(mm.CSR64))
    jobs, wrong = [], []
    for n in (900, 250_000):
        rng = np.random.default_rng(n)
        pos, crd, val = _csr(rng, np.full(n, 5), n, np.int64)
        x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
        A = CsrMatrix.from_host(pos, crd, val, (n, n), dev)
        want = A.spmv(torch.as_tensor(x).to(dev), torch.as_tensor(y).to(dev)).cpu().numpy()
        jobs.append((pos, crd, val, ((n, n), (n + 1, len(crd), len(crd))), x, y, want))

    def work(pos, crd, val, spec, x, y, want):
        for _ in range(40):
            got = y.copy()
            module.spmv(pos, crd, val, spec, x, got)
            if not np.array_equal(got, want):
                wrong.append(len(x))

    threads = [threading.Thread(target=work, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
