"""The static-pivot solve by rounds of independent steps against the same solve step by step on one
warp: same order of every entry's updates, so the factors, the solution and the failing step agree
to the bit. Sizes from one unknown to the largest, sparse patterns (rings, trees, a supply column)
and a dense ones, whose lists do not fit and which stay on the one-warp kernel."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pattern(kind, n, rng):
    mask = np.eye(n, dtype=bool)
    i = np.arange(n)
    if kind == "ring":
        mask[i, (i + 1) % n] = mask[(i + 1) % n, i] = True
        mask[:, n - 1] = mask[n - 1, :] = True
    elif kind == "random":
        mask |= rng.random((n, n)) < 2.0 / n
    else:
        mask[:] = True
    return mask


@pytest.mark.parametrize("kind,n", [("ring", 1), ("ring", 2), ("ring", 3), ("ring", 33), ("ring", 103), ("ring", 160),
                                    ("random", 31), ("random", 64), ("random", 160), ("dense", 20), ("dense", 40), ("dense", 160)])
def test_rounds_give_the_bits_of_the_step_order(kind, n):
    from xyce_b200 import _native

    lib = _native.load()
    rng = np.random.default_rng(n)
    mask = _pattern(kind, n, rng)
    rows, cols = np.nonzero(mask)
    rowptr = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.int32)
    colind = cols.astype(np.int32)
    A = np.where(mask, rng.standard_normal((n, n)), 0.0)
    if kind == "ring" and n > 2:
        A[0, 0] = 0.0  # a zero on the diagonal: its rows are exchanged
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    T = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")
    slu = ctypes.c_void_p()
    v0 = np.ascontiguousarray(A[rows, cols])
    assert lib.xd_slu_create(n, rowptr.ctypes.data_as(_native._ip), colind.ctypes.data_as(_native._ip),
                             v0.ctypes.data_as(_native._dp), 1e-3, 0, ctypes.byref(slu)) == 0
    fits = {("ring", 160): None, ("dense", 40): 0, ("dense", 160): 0}.get((kind, n), 1)
    by_rounds = lib.xd_slu_rounds(slu, 1)
    assert by_rounds in (0, 1) and fits in (None, by_rounds)
    infos = []
    for trial in range(6):
        # The matrix itself, two nearby ones, then wide ones that fail some threshold test.
        near, spread = (0.0 if trial == 0 else 0.1), (0.0 if trial < 3 else 3.0)
        Ak = np.where(mask, A * 10.0 ** rng.uniform(-spread, spread, (n, n)) * (1 + near * rng.random((n, n))), 0.0)
        if trial == 5:
            Ak[n // 2, :] = np.where(mask[n // 2], np.nan, 0.0)
        vals, b = T(Ak[rows, cols]), T(rng.standard_normal(n))
        got = []
        for on in (1, 0):
            lib.xd_slu_rounds(slu, on)
            lu, x = T(np.full(n * n, 7.0)), T(np.full(n, 5.0))
            info = torch.full((1,), -9, dtype=torch.int32, device="cuda")
            assert lib.xd_slu_solve(slu, p(vals), p(b), p(lu), p(x), p(info), None) == 0
            torch.cuda.synchronize()
            got.append((lu.view(torch.int64).cpu(), x.view(torch.int64).cpu(), int(info)))
            if on == 1 and trial == 0 and got[0][2] == 0:  # without the factors: the same solution
                assert lib.xd_slu_solve(slu, p(vals), p(b), None, p(x), p(info), None) == 0
                assert torch.equal(x.view(torch.int64).cpu(), got[0][1])
        assert got[0][2] == got[1][2], trial
        assert torch.equal(got[0][1], got[1][1]) and torch.equal(got[0][0], got[1][0]), trial
        infos.append(got[0][2])
    assert infos[0] == 0 and (infos[5] > 0)
    lib.xd_slu_destroy(slu)
