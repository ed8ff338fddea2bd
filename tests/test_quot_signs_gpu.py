"""The device models' quotients (csrc/quot.h) of zeros, infinities and ordinary values, signs included,
and of numerators down to 2^-968, against IEEE division bit for bit."""
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


def same_bits(got, ref):
    nan = np.isnan(ref)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(got[~nan].view(np.uint64), ref[~nan].view(np.uint64))


def test_signs_of_zeros_and_infinities():
    v = np.array([0.0, 1.0, 3.0, 1e300, 1e-300, 1e200, np.inf])
    v = np.concatenate([v, -v, [np.nan]])
    a, b = (m.ravel() for m in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        refs = [a / b, a / 3.0, a / 12.0, a / 0.25]
    # 1e-300 / 1e300 underflows to a zero of the right sign; no quotient here is subnormal.
    assert all(same_bits(g, r) for g, r in zip(quot(a, b), refs))


def test_small_numerators():
    rng = np.random.default_rng(2)
    a = rng.choice([-1.0, 1.0], 100_000) * np.ldexp(rng.uniform(1.0, 2.0, 100_000), -968)
    b = rng.choice([-1.0, 1.0], 100_000) * np.exp2(rng.uniform(-20.0, 20.0, 100_000))
    assert same_bits(quot(a, b)[0], a / b)
