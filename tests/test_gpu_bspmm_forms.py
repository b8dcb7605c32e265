"""Batched SpMM over the forms that its dispatch chooses among: lengths of a row around the groups of lanes, fibers that share their
values over a group and others, B in slices and whole, and rows of B too long for a slice each.  Every form returns the bits of the
sequential loop."""
import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _on(a):
    return torch.as_tensor(a).to(DEV)


@pytest.mark.parametrize("idx", [np.int32, np.int64])
@pytest.mark.parametrize("nh", [1, 3, 4, 6, 8, 12, 16, 20, 64])
@pytest.mark.parametrize("fours", [1, 2, 4, 5, 8, 9, 12, 13, 16, 17, 32, 33, 48, 64, 65, 95, 128, 130, 170, 257])
def test_row_lengths(fours, nh, idx):
    """Rows of B of about 4 * fours elements, short and long rows of A, against the oracle."""
    from lapis_b200 import device
    rng = np.random.default_rng(fours * 100 + nh)
    dh = -(-4 * fours // nh)
    n1, n2 = 60, 37
    lens = rng.integers(0, 11, n1)
    lens[[3, 17]] = 257, 64
    pos = np.zeros(n1 + 1, idx)
    pos[1:] = np.cumsum(lens)
    crd = rng.integers(0, n2, pos[-1]).astype(idx)
    val = rng.uniform(-1, 1, (pos[-1] * nh,)).astype(np.float32)
    B, C = (rng.uniform(-1, 1, (n, dh, nh)).astype(np.float32) for n in (n2, n1))
    args = [_on(a) for a in (pos, crd, val, B)]
    assert np.array_equal(device.bspmm_csrv(*args, n2).cpu().numpy(), oracle.bspmm(pos, crd, val, B))
    assert np.array_equal(device.bspmm_csrv(*args, n2, _on(C)).cpu().numpy(), oracle.bspmm(pos, crd, val, B, C))


def _sequential(pos, crd, val, B, C):
    out = C.clone()
    for r in range(len(pos) - 1):
        for j in range(pos[r], pos[r + 1]):
            out[r] = val[j] * B[crd[j]] + out[r]  # two roundings: no fused multiply-add between separate operations
    return out


@pytest.mark.parametrize("idx", [torch.int32, torch.int64])
@pytest.mark.parametrize("n2,dh,nh", [
    (27_000, 75, 12), (400_000, 24, 4), (600_000, 8, 8), (150_000, 4, 64), (262_144, 64, 4), (200_000, 40, 4), (131_072, 50, 8),  # fours
    (180_000, 32, 5), (400_000, 64, 1), (500_000, 26, 2), (130_000, 32, 7), (120_000, 256, 1),                                    # ones
    (2, 8_388_608, 4), (1, 25_000_000, 3)])  # more than 65,535 slices of 256 elements
def test_a_large_right_hand_side(n2, dh, nh, idx):
    """B of 100 to 300 MB, whole or in slices, rows of 0 to 9 entries."""
    from lapis_b200 import device
    g = torch.Generator(device=DEV).manual_seed(n2)
    n1 = 3 if n2 < 10 else 40
    lens = torch.arange(n1) * 7 % 10
    pos = torch.zeros(n1 + 1, dtype=torch.int64)
    torch.cumsum(lens, 0, out=pos[1:])
    nnz = int(pos[-1])
    crd = torch.randint(0, n2, (nnz,), device=DEV, generator=g)
    rand = lambda *s: torch.rand(s, device=DEV, generator=g) * 2 - 1
    val, B, C = rand(nnz, nh), rand(n2, dh, nh), rand(n1, dh, nh)
    want = _sequential(pos.tolist(), crd.tolist(), val[:, None, :], B, C)
    assert torch.equal(device.bspmm_csrv(pos.to(DEV, idx), crd.to(idx), val.reshape(-1), B, n2, C), want)
