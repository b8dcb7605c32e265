"""What a compiled module hands to its library for the operands it is given: no GPU is involved."""
import struct

import numpy as np
import pytest

from lapis_b200 import KokkosBackend as KB


class Library:
    """Stands for a module's library: keeps the bytes behind each argument (None stays None)."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, symbol):
        return lambda *args: self.calls.append(args)


@pytest.fixture(autouse=True)
def _no_status(monkeypatch):
    monkeypatch.setattr(KB, "check_last", lambda: None)  # the status of some earlier call into the real library


def _bound(kind, sfx=""):
    module = object.__new__(KB.LAPISModule)
    module.libHandle = Library()
    return module._bind(kind, kind, sfx, np.int32), module.libHandle.calls


def _vector(address, n):
    return struct.pack("PPqqq", address, address, 0, n, 1)


@pytest.mark.parametrize("column", [(), (1,), (1, 1)], ids=["vector", "column", "column3"])
def test_vectors_may_come_as_columns(column):
    spmv, calls = _bound("spmv")
    pos, crd, val = np.array([0, 1, 2], np.int32), np.array([0, 1], np.int32), np.ones(2)
    x, y = np.ones((2,) + column), np.zeros((2,) + column)
    assert spmv(pos, crd, val, ((2, 2), (3, 2, 2)), x, y) is y
    assert calls[0][-2:] == (_vector(x.ctypes.data, 2), _vector(y.ctypes.data, 2))
    with pytest.raises(ValueError):
        spmv(pos, crd, val, ((2, 2), (3, 2, 2)), np.ones((2, 2)), y)
    with pytest.raises(ValueError):
        spmv(pos, crd, val, ((2, 2), (3, 2, 2)), np.float64(1.0), y)


def test_matrices_of_one_column_may_come_with_more_extents():
    spmm, calls = _bound("spmm")
    pos, crd, val = np.array([0, 1, 2], np.int32), np.array([0, 1], np.int32), np.ones(2)
    B, C = np.ones((2, 1, 1)), np.zeros((2, 1))
    assert spmm(pos, crd, val, ((2, 2), (3, 2, 2)), B, C) is C
    assert calls[0][-2:] == tuple(struct.pack("PPqqqqq", m.ctypes.data, m.ctypes.data, 0, 2, 1, 1, 1) for m in (B, C))
    for bad in (np.ones(2), np.ones((2, 3, 1))):
        with pytest.raises(ValueError):
            spmm(pos, crd, val, ((2, 2), (3, 2, 2)), bad, C)


@pytest.mark.parametrize("spec", [((2, 2), (3, 2, 2)), ((2.0, 2.0), (3.0, 2, 2)), [np.array([2, 2]), np.array([3.0, 2.0, 2.0])],
                                  ((2, 2, 7), (3, 2, 2, 9))])
def test_specifiers_of_every_number_type(spec):
    spmv, calls = _bound("spmv")
    pos, crd, val = np.array([0, 1, 2], np.int32), np.array([0, 1], np.int32), np.ones(2)
    spmv(pos, crd, val, spec, np.ones(2), np.zeros(2))
    assert struct.unpack("5q", calls[0][4]) == (2, 2, 3, 2, 2)
