"""spmm_long_kernel at the edges of its tiles of 1280 products, of its list of 448 rows and of the 768 pieces that a team of four
blocks divides: bit for bit against the oracle's sequential loop."""
import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"
TILE, LONG = 1280, 256  # products of a tile; rows of up to 256 entries are not long


def _on(a):
    return torch.as_tensor(a).to(DEV)


@pytest.mark.parametrize("idx", [np.int32, np.int64])
@pytest.mark.parametrize("k", [1, 2, 5, 7, 16, 31, 33, 63, 64, 65, 128, 129, 200])
def test_rows_that_end_at_a_tile(k, idx):
    """One entry less and more than the first four whole numbers of tiles above 256 entries, each several times, in any order; in panels of
    up to 64 columns, or of up to 32 or 16 where a team has few rows."""
    from lapis_b200 import device
    panels = -(-k // 64)
    marks = [LONG - 1, LONG, LONG + 1]
    for entries in {TILE // -(-k // -(-k // most)) for most in (64, 32, 16)}:
        tiles = LONG // entries + 1
        ends = [e * entries + d for e in range(tiles, tiles + 4) for d in (-1, 0, 1)]
        marks += [n for n in ends if n > LONG] * (1 if k < 16 else 2)
    rng = np.random.default_rng(k)
    rows, cols = 600, 300
    lens = rng.integers(0, 9, rows)
    lens[rng.choice(rows, len(marks), replace=False)] = marks
    assert np.sum(lens) * (k + 8) // panels >> 18 < LONG  # the kernel's rule on the length beside the whole product
    pos = np.zeros(rows + 1, idx)
    pos[1:] = np.cumsum(lens)
    crd, val = rng.integers(0, cols, pos[-1]).astype(idx), rng.uniform(-1, 1, pos[-1])
    B, C = rng.uniform(-1, 1, (cols, k)), rng.uniform(-1, 1, (rows, k))
    A = device.CsrMatrix(_on(pos), _on(crd), _on(val), (rows, cols))
    for accumulate in (True, False):
        want = oracle.spmm(pos, crd, val, B, C if accumulate else np.zeros_like(C))
        assert np.array_equal(A.spmm(_on(B), _on(C), accumulate=accumulate).cpu().numpy(), want)
    number = np.arange(0, 2 * rows, 2).astype(idx)
    D = rng.uniform(-1, 1, (2 * rows, k))
    got = device.spmm_dcsr(_on(number), _on(pos), _on(crd), _on(val), _on(B), _on(D), cols).cpu().numpy()
    assert np.array_equal(got, oracle.spmm_dcsr(number, pos, crd, val, B, D))


@pytest.mark.parametrize("lengths", ["equal", "mixed"])
@pytest.mark.parametrize("k", [1, 33, 130])
@pytest.mark.parametrize("count", [1, 5, 64, 192, 256, 257, 447, 448, 449, 900])
@pytest.mark.parametrize("team", [4, 1])
def test_lists_of_long_rows(team, count, k, lengths):
    """Long rows that one team of four blocks, or one block alone, meets: fewer and more than its list of 448 holds and than the 768
    pieces (a row and up to 64 columns) that a team divides by length.  Up to 450,000 bytes of offsets blocks work in teams."""
    from lapis_b200 import device
    shares = torch.cuda.get_device_properties(0).multi_processor_count // team
    at = np.arange(count)
    where = (at // 8 * shares + shares // 2) * 8 + at % 8
    rows, cols = max(int(where[-1]) + 5, shares * team * 8, 1 if team == 4 else 120_000), 3000
    assert (rows * 4 <= 450_000) == (team == 4)
    rng = np.random.default_rng(k)
    long = np.full(count, 300) if lengths == "equal" else rng.integers(LONG + 1, 700, count)
    assert np.sum(long) * (k + 8) // -(-k // 64) >> 18 < LONG
    lens = np.zeros(rows, np.int64)
    lens[where] = long
    pos = np.zeros(rows + 1, np.int32)
    pos[1:] = np.cumsum(lens)
    few = np.concatenate([[0], np.cumsum(long)]).astype(np.int32)
    crd, val = rng.integers(0, cols, pos[-1]).astype(np.int32), rng.uniform(-1, 1, pos[-1])
    B = rng.uniform(-1, 1, (cols, k))
    C = torch.zeros((rows, k), dtype=torch.float64, device=DEV)
    got = device.CsrMatrix(_on(pos), _on(crd), _on(val), (rows, cols)).spmm(_on(B), C, accumulate=False)
    want = oracle.spmm(few, crd, val, B, np.zeros((count, k)))
    assert np.array_equal(got[_on(where)].cpu().numpy(), want)
    assert int((got != 0).any(1).sum()) == count


@pytest.mark.parametrize("idx", [np.int32, np.int64])
@pytest.mark.parametrize("rows", [333, 56_000, 150_001])
def test_runs_of_one_row_number(rows, idx):
    """DCSR: a number that is listed more than once is one row, long where its runs are together, also across the four rows that a thread
    looks at; short runs, single rows and empty ones between them."""
    from lapis_b200 import device
    rng = np.random.default_rng(rows)
    k, cols = 5, 900
    lens = rng.integers(0, 3, rows)
    runs = np.ones(rows, np.int64)  # length of the run that begins here; 0 inside one
    for start, n, each in ((0, 3, 100), (17, 2, 129), (30, 5, 52), (41, 9, 40), (60, 2, 128), (70, 4, 64), (rows - 6, 6, 50)):
        runs[start:start + n] = [n] + [0] * (n - 1)
        lens[start:start + n] = each
    lens[[100, 103, 211]] = 257, 300, 1281
    number = (np.cumsum(runs > 0) * 2 - 1).astype(idx)
    pos = np.zeros(rows + 1, idx)
    pos[1:] = np.cumsum(lens)
    crd, val = rng.integers(0, cols, pos[-1]).astype(idx), rng.uniform(-1, 1, pos[-1])
    B, C = rng.uniform(-1, 1, (cols, k)), rng.uniform(-1, 1, (2 * rows, k))
    got = device.spmm_dcsr(_on(number), _on(pos), _on(crd), _on(val), _on(B), _on(C), cols).cpu().numpy()
    assert np.array_equal(got, oracle.spmm_dcsr(number, pos, crd, val, B, C))
