"""The transient's sparse solve with a library that fails: a zero pivot in the kept pivot order is
answered by a host factorization, any other error reaches the caller."""
import ctypes
import types

import pytest

from xyce_b200 import _native
from xyce_b200.transient import GpuTransient

torch = pytest.importorskip("torch")


class Library:
    """xd_rf_solve_refined that returns the given codes in turn."""

    def __init__(self, *codes):
        self.codes, self.calls = list(codes), 0

    def xd_rf_solve_refined(self, h, vals, b, x, refactor, tol, refine, check):
        self.calls += 1
        return self.codes.pop(0)

    def xd_rf_destroy(self, h):
        pass


def transient(lib):
    tr = GpuTransient.__new__(GpuTransient)
    stream = types.SimpleNamespace(cuda_stream=0)
    tr.torch = types.SimpleNamespace(full_like=torch.full_like, empty_like=torch.empty_like,
                                     cuda=types.SimpleNamespace(current_stream=lambda dev: stream))
    tr.dev, tr._lib, tr._rf, tr._ptr = None, lib, ctypes.c_void_p(1), lambda t: None
    tr.jac, tr.rhs = torch.ones(3), torch.ones(3)
    tr.stats = types.SimpleNamespace(factorizations=0, solves=0, refinements=0, first_solve_berr=[])
    tr.setups = 0

    def setup():
        tr.setups += 1
        return True

    tr._rf_try_setup = setup
    return tr


def test_zero_pivot_is_factored_on_the_host():
    tr = transient(Library(-5, 0))
    assert tr._solve_rf() is not None
    assert (tr.setups, tr._lib.calls) == (1, 2)


@pytest.mark.parametrize("code", [-1, -3])
def test_other_errors_are_raised(code):
    tr = transient(Library(code, 0))
    with pytest.raises(_native.NativeError) as e:
        tr._solve_rf()
    assert e.value.code == code and (tr.setups, tr._lib.calls) == (0, 1)
