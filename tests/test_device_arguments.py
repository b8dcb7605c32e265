"""Operands and arguments that the device-resident calls cannot use: a Python exception, without a GPU."""
import pytest
import torch


def _unbacked(shape, dtype):
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode(allow_non_fake_inputs=True):
        return torch.empty(shape, dtype=dtype, device="cuda")  # a CUDA tensor without storage


def test_operands_that_torch_refuses_raise():
    """torch refuses the address of a tensor without storage by a C++ exception; it must not end the process."""
    from lapis_b200 import _calls, device
    f64, f32, i32 = (_unbacked(s, t) for s, t in (((4, 4), torch.float64), ((4, 4, 4), torch.float32), ((5,), torch.int32)))
    for call in (lambda: _calls.spmv(0, 16, 16, f64, f64, True), lambda: _calls.spmm(0, 4, 4, f64, f64, True),
                 lambda: device.bgemm(f32, f32, f32), lambda: device.spmm_dcsr(i32[1:], i32, i32, f64, f64, f64, 4),
                 lambda: device.bspmm_csrv(i32, i32[1:], f32[0], f32, 4, f32)):
        with pytest.raises(RuntimeError):
            call()


def test_arguments_of_another_type_raise():
    from lapis_b200 import _calls
    x = _unbacked((4, 4), torch.float64)
    for args in ((None, 4, 4, x, x, True), (0, "4", 4, x, x, True), (0, 4, 4, x, x, torch.ones(2)), (0, 4, 4, x)):
        with pytest.raises((TypeError, RuntimeError)):
            _calls.spmm(*args)


def test_a_released_matrix_refuses_products():
    """After its release a matrix must not pass the old handle on."""
    from lapis_b200.device import CsrMatrix

    class Library:
        released = 0

        def lapis_b200_csr_destroy(self, h):
            self.released += 1

    A = object.__new__(CsrMatrix)
    A._lib, A._h, A._addr, A.nrows, A.ncols = Library(), 4096, 4096, 0, 0
    A.__del__()
    assert (A._lib.released, A._h, A._addr) == (1, None, 0)
    A.__del__()
    assert A._lib.released == 1


def test_matrices_may_have_further_extents_of_one():
    """Row-major all the same: the call gets as far as the address, which a tensor without storage does not have."""
    from lapis_b200 import _calls
    for shape in ((4, 4), (4, 4, 1), (4, 4, 1, 1)):
        with pytest.raises(RuntimeError):
            _calls.spmm(0, 4, 4, _unbacked(shape, torch.float64), _unbacked((4, 4), torch.float64), True)
    for shape in ((4,), (16,), (4, 4, 2), (4, 1, 4)):
        assert _calls.spmm(0, 4, 4, _unbacked(shape, torch.float64), _unbacked((4, 4), torch.float64), True) == -1


@pytest.mark.parametrize("dims", [1, 4])
def test_matmul_of_other_ranks_is_a_value_error(dims):
    from lapis_b200 import device
    x = _unbacked((4,) * dims, torch.float32)
    with pytest.raises(ValueError):
        device.bgemm(x, x, x)
