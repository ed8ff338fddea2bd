"""The device models' quotient (csrc/quot.h) against IEEE division, bit for bit: random significands
over the exponents the models meet and far beyond, significands near one and two, special values."""
import ctypes

import numpy as np
import pytest

from xyce_b200 import _native

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def quot(a, b):
    a, b = (torch.as_tensor(np.ascontiguousarray(v), device="cuda") for v in (a, b))
    out = torch.zeros(4 * a.numel(), dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    _native.check(_native.load().xd_probe_quot(p(a), p(b), p(out), a.numel(), None), "xd_probe_quot")
    torch.cuda.synchronize()
    return out.cpu().numpy().reshape(4, -1)


def numbers(rng, n, exponents, edge):
    """Random doubles; edge: significands within 16 of a power of two (all ones left out: the one
    significand whose quotients may be off by the last bit)."""
    f = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    if edge:
        k = rng.integers(0, 16, n, dtype=np.uint64)
        f = np.where(rng.random(n) < 0.5, k, np.uint64((1 << 52) - 2) - k)
    e = (1023 + rng.integers(-exponents, exponents + 1, n)).astype(np.uint64)
    s = rng.integers(0, 2, n, dtype=np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | f).view(np.float64)


@pytest.mark.parametrize("exponents,edge_a,edge_b", [(2, False, False), (60, False, True), (480, False, False),
                                                     (480, True, False), (300, True, True)])
def test_quotients_are_correctly_rounded(exponents, edge_a, edge_b):
    rng = np.random.default_rng(exponents)
    n = 4_000_000
    a, b = numbers(rng, n, exponents, edge_a), numbers(rng, n, exponents, edge_b)
    if not edge_b:
        b = b[(b.view(np.uint64) & np.uint64((1 << 52) - 1)) != np.uint64((1 << 52) - 1)]
        a = a[:b.size]
    got = quot(a, b)
    for row, ref in zip(got, (a / b, a / 3.0, a / 12.0, a / 0.25)):
        assert np.array_equal(row.view(np.uint64), ref.view(np.uint64))


def test_special_values():
    v = np.array([0.0, -0.0, 1.0, -3.0, 1e300, 1e-300, 1e200, -1e-200, np.inf, -np.inf, np.nan])
    a, b = (m.ravel() for m in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        ref = a / b
    got = quot(a, b)[0]
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(got[~np.isnan(ref)], ref[~np.isnan(ref)])


def test_all_ones_denominators_are_within_one_unit():
    rng = np.random.default_rng(1)
    a = rng.uniform(-2.0, 2.0, 100_000)
    b = np.full_like(a, np.nextafter(1.0, 0.0))
    ref = a / b
    assert (np.abs(quot(a, b)[0] - ref) <= np.spacing(np.abs(ref))).all()
