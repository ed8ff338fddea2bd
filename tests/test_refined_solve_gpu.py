"""The checked solve (xd_rf_solve_refined) and the Newton norms on the device against numpy: rows of
every route of the residual (eight lanes, long rows in one segment and in several), corrections by
the factors of a nearby matrix, and the outcomes; norms by one block and by a cluster."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _system(n, long_rows, rng):
    """A diagonally dominant matrix, three entries a row, with rows of the given numbers of entries
    (and as many columns, so that the factors stay sparse)."""
    import scipy.sparse as sp

    i = np.arange(n)
    A = sp.lil_matrix((n, n))
    A[i, (i + 1) % n] = rng.uniform(-1, 1, n)
    A[i, (i + 7) % n] = rng.uniform(-1, 1, n)
    for q, count in enumerate(long_rows):
        at = rng.choice(n - 20, count - 3, replace=False)
        A[n - 1 - q, at] = rng.uniform(-1, 1, count - 3)
    A = A.tocsr()
    A = A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + 1.0)
    A.sort_indices()
    return A.tocsr()


def _create(lib, A):
    import scipy.sparse.linalg as spl
    from xyce_b200 import _native

    lu = spl.splu(A.tocsc(), permc_spec="MMD_AT_PLUS_A", diag_pivot_thresh=0.1, options=dict(SymmetricMode=True))
    P, Q = np.argsort(lu.perm_r).astype(np.int32), np.argsort(lu.perm_c).astype(np.int32)
    L, U = lu.L.tocsr(), lu.U.tocsr()
    L.sort_indices()
    U.sort_indices()
    i32 = lambda a: np.ascontiguousarray(a, dtype=np.int32)
    arrs = [i32(A.indptr), i32(A.indices), A.data, i32(L.indptr), i32(L.indices), L.data, i32(U.indptr),
            i32(U.indices), U.data, P, Q]
    ip = lambda a: a.ctypes.data_as(_native._ip)
    dp = lambda a: a.ctypes.data_as(_native._dp)
    h = ctypes.c_void_p()
    assert lib.xd_rf_create(A.shape[0], A.nnz, ip(arrs[0]), ip(arrs[1]), dp(arrs[2]), L.nnz, ip(arrs[3]),
                            ip(arrs[4]), dp(arrs[5]), U.nnz, ip(arrs[6]), ip(arrs[7]), dp(arrs[8]), ip(P), ip(Q), 0,
                            ctypes.byref(h)) == 0
    return h


@pytest.mark.parametrize("n,long_rows", [(1, []), (31, []), (33, []), (1500, [128, 129]), (3000, [1024, 1025, 2050])])
def test_checked_solve_reports_numpys_backward_error(n, long_rows):
    import scipy.sparse as sp
    from xyce_b200 import _native

    lib = _native.load()
    rng = np.random.default_rng(n)
    A = _system(n, long_rows, rng) if n > 1 else sp.csr_matrix([[2.0]])
    h = _create(lib, A)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    T = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")
    B = A.copy()
    B.data = A.data * (1 + 0.01 * rng.uniform(-1, 1, A.nnz))
    b = rng.standard_normal(n)
    vals, bd, x = T(B.data), T(b), torch.zeros(n, dtype=torch.float64, device="cuda")
    check = _native.XdRfCheck()

    def solve(v, rhs, refactor, tol, refine):
        rc = lib.xd_rf_solve_refined(h, p(v), p(rhs), p(x), refactor, tol, refine, ctypes.byref(check))
        return rc, check.outcome, check.solves, check.checks

    def berr():
        xs = x.cpu().numpy()
        return (np.abs(b - B @ xs) / (abs(B) @ np.abs(xs) + np.abs(b))).max()

    # A's factors on the nearby B: no refinement, then enough of it. Both sides sum a row's at most 2050
    # terms in their own order, an error of at most 2050 * 2^-53 = 2.3e-13 of the row's absolute sum.
    for refine, outcome in ((0, _native.XD_RF_ABOVE_TOL), (30, _native.XD_RF_WITHIN_TOL)):
        rc, got, solves, checks = solve(vals, bd, 0, 1e-11, refine)
        assert rc == 0 and got == outcome and checks == solves and 1 <= solves <= refine + 1
        assert abs(check.berr - berr()) <= 5e-13
        assert check.first_berr >= check.berr
    # B's own factors.
    assert solve(vals, bd, 1, 1e-10, 3) == (0, _native.XD_RF_WITHIN_TOL, 1, 1)
    assert berr() <= 1e-12
    # A right-hand side that is not finite, a zero pivot, and the factors usable afterwards.
    bad = bd.clone()
    bad[n // 2] = float("inf")
    rc, got, solves, checks = solve(vals, bad, 0, 1e-10, 3)
    assert rc == 0 and got == _native.XD_RF_NOT_FINITE and checks == 0
    zero = torch.zeros_like(vals)
    assert solve(zero, bd, 1, 1e-10, 3)[0] == -5
    assert solve(vals, bd, 1, 1e-10, 3) == (0, _native.XD_RF_WITHIN_TOL, 1, 1)
    assert lib.xd_rf_solve_refined(h, p(vals), p(bd), p(bd), 0, 1e-10, 3, ctypes.byref(check)) < 0
    lib.xd_rf_destroy(h)


@pytest.mark.parametrize("n", [1, 1025, 8192, 8193, 40_001])
@pytest.mark.parametrize("update", [0, 1])
def test_newton_norms(n, update):
    from xyce_b200 import _native

    lib = _native.load()
    rng = np.random.default_rng(n)
    rowptr, colind = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32)
    csr = _native.XdCsr(n, rowptr.ctypes.data_as(_native._ip), colind.ctypes.data_as(_native._ip))
    h = ctypes.c_void_p()
    assert lib.xd_tia_create(ctypes.byref(csr), 0, ctypes.byref(h)) == 0
    x, dx, xref, w, rhs = (rng.standard_normal(n) for _ in range(5))
    w = np.abs(w) + 0.1
    D = [torch.as_tensor(a, device="cuda") for a in (x, dx, xref, w, rhs)]
    norms = torch.zeros(3, dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.xd_tia_newton_update(h, p(D[0]), p(D[1]), p(D[2]), p(D[3]), 1e-3, 1e-6, update, p(norms), None) == 0
    assert lib.xd_tia_residual_norm(h, p(D[4]), None, p(norms), None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(D[0].cpu().numpy(), x + dx)
    wn = 1e-3 * np.maximum(np.abs(xref), np.abs(x + dx)) + 1e-6 if update else w
    assert np.array_equal(D[3].cpu().numpy(), wn)
    # A sum of n squares in any order: within n * 2^-53 of the sum, half of that in its root.
    assert abs(float(norms[0]) / np.sqrt(np.mean((dx / wn) ** 2)) - 1) <= (n + 4) * 2.0**-53
    assert float(norms[1]) == np.abs(rhs).max() and float(norms[2]) == 0.0
    for value in (np.inf, -np.nan):
        D[4][n - 1] = value
        assert lib.xd_tia_residual_norm(h, p(D[4]), None, p(norms), None) == 0
        assert np.isnan(float(norms[1]))
    lib.xd_tia_destroy(h)
