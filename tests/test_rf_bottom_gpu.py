"""Refactorization of systems whose bottom groups hold more entries than shared memory (they work in the
factors' own array) and of the same structure with fewer: two million unknowns in chains of four,
and 20,000, against the known solution."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chains", [5_000, 500_000])
def test_chains_of_four(chains):
    from xyce_b200 import _native

    lib = _native.load()
    rng = np.random.default_rng(chains)
    n = 4 * chains
    # Tridiagonal 4 x 4 blocks, diagonally dominant: the factors have the matrix's own pattern.
    d = 4.0 + rng.random((chains, 4))
    lo, up = rng.uniform(-1, 1, (chains, 3)), rng.uniform(-1, 1, (chains, 3))
    piv, mul = d.copy(), np.zeros((chains, 3))
    for k in range(3):
        mul[:, k] = lo[:, k] / piv[:, k]
        piv[:, k + 1] = d[:, k + 1] - mul[:, k] * up[:, k]

    def csr(parts):  # parts: (column offset, [chains, 4] values, mask of rows), ascending offsets
        cols = np.concatenate([np.arange(n).reshape(chains, 4)[:, :, None] + o for o, _, _ in parts], axis=2)
        vals = np.stack([v for _, v, _ in parts], axis=2)
        keep = np.broadcast_to(np.stack([np.asarray(m, bool) for _, _, m in parts], axis=1)[None], vals.shape)
        ptr = np.concatenate([[0], np.cumsum(keep.sum(2).ravel())]).astype(np.int32)
        return ptr, np.ascontiguousarray(cols[keep], dtype=np.int32), np.ascontiguousarray(vals[keep])

    z = np.zeros((chains, 1))
    below, above = [0, 1, 1, 1], [1, 1, 1, 0]
    A = csr([(-1, np.hstack([z, lo]), below), (0, d, [1] * 4), (1, np.hstack([up, z]), above)])
    L = csr([(-1, np.hstack([z, mul]), below), (0, np.ones((chains, 4)), [1] * 4)])
    U = csr([(0, piv, [1] * 4), (1, np.hstack([up, z]), above)])
    order = np.arange(n, dtype=np.int32)
    ip = lambda a: a.ctypes.data_as(_native._ip)
    dp = lambda a: a.ctypes.data_as(_native._dp)
    h = ctypes.c_void_p()
    assert lib.xd_rf_create(n, len(A[1]), ip(A[0]), ip(A[1]), dp(A[2]), len(L[1]), ip(L[0]), ip(L[1]), dp(L[2]),
                            len(U[1]), ip(U[0]), ip(U[1]), dp(U[2]), ip(order), ip(order), 0, ctypes.byref(h)) == 0
    x = rng.standard_normal(n)
    X = x.reshape(chains, 4)
    b = d * X
    b[:, 1:] += lo * X[:, :3]
    b[:, :3] += up * X[:, 1:]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    vals, got = torch.as_tensor(A[2], device="cuda"), torch.as_tensor(b.ravel(), device="cuda")
    assert lib.xd_rf_refactor(h, p(vals)) == 0
    assert lib.xd_rf_solve(h, p(got)) == 0
    torch.cuda.synchronize()
    # Rows dominate by at least 2, so the inverse's norm is at most 1/2, the matrix's at most 7: a dozen
    # roundings a row, each 2^-53 of at most 7 max|x|, times 1/2.
    assert np.abs(got.cpu().numpy() - x).max() <= 12 * 2.0**-53 * 7 / 2 * np.abs(x).max()
    lib.xd_rf_destroy(h)
