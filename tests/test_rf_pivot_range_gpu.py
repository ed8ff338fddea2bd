"""Pivots at the ends of the double range (csrc/lutree.cu divides by those whose reciprocal is not a
normal number): one row of a banded matrix scaled until its pivot is subnormal or above 2^1022, in
the bottom subtrees and at several places of the chains' blocks of eight. Refactorization and solve
accept them and solve the system."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from xyce_b200 import _native

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
N, W = 700, 40


def _banded(rng):
    A = sp.diags([rng.uniform(-1.0, 1.0, N - abs(k)) for k in range(-W, W + 1)], range(-W, W + 1)).tocsr()
    A.setdiag(0.0)
    A = sp.csr_matrix(A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + 1.0))
    A.sort_indices()
    return A


@pytest.mark.parametrize("row", [3, 640, 647, 650, 653, 699])
@pytest.mark.parametrize("target", [-1023, 1022])
def test_one_row_scaled(row, target):
    rng = np.random.default_rng(row)
    A = _banded(rng)
    lu = spl.splu(A.tocsc(), permc_spec="NATURAL", diag_pivot_thresh=0.0, options=dict(SymmetricMode=True))
    L, U = lu.L.tocsr(), lu.U.tocsr()
    L.sort_indices()
    U.sort_indices()
    lib, h = _native.load(), ctypes.c_void_p()
    i32 = lambda a: np.ascontiguousarray(a, np.int32)
    ip = lambda a: a.ctypes.data_as(_native._ip)
    dp = lambda a: a.ctypes.data_as(_native._dp)
    k = [i32(A.indptr), i32(A.indices), A.data, i32(L.indptr), i32(L.indices), L.data, i32(U.indptr), i32(U.indices),
         U.data, i32(np.arange(N))]
    assert lib.xd_rf_create(N, A.nnz, ip(k[0]), ip(k[1]), dp(k[2]), L.nnz, ip(k[3]), ip(k[4]), dp(k[5]), U.nnz, ip(k[6]),
                            ip(k[7]), dp(k[8]), ip(k[9]), ip(k[9]), 0, ctypes.byref(h)) == 0
    vals = A.data.copy()
    at = slice(A.indptr[row], A.indptr[row + 1])
    # Its diagonal entry to [2^target, 2^(target + 1)): the entries of L's column below it stay finite.
    exponent = target - int(np.floor(np.log2(vals[at].max())))
    vals[at] = np.ldexp(vals[at], exponent)
    # In units of the row's scale: the matrix as stored, a solution away from zero, its right-hand side.
    B = A.copy()
    B.data[at] = np.ldexp(vals[at], -exponent)
    x = rng.uniform(0.25, 0.5, N)
    unit = B @ x
    b = unit.copy()
    b[row] = np.ldexp(b[row], exponent)
    unit[row] = np.ldexp(b[row], -exponent)  # as stored
    v, got = torch.as_tensor(vals, device="cuda"), torch.as_tensor(b, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.xd_rf_refactor(h, p(v)) == 0, lib.xd_last_error()
    assert lib.xd_rf_solve(h, p(got)) == 0
    torch.cuda.synchronize()
    y = got.cpu().numpy()
    # As in the other refactorization tests at most 81 products a row, each with a few roundings, in
    # factors that the dominant diagonal keeps from growing: 81 x 2 x 4 x 2^-53 = 7.2e-14, and the
    # bound there. In a subnormal row there are as many roundings to 2^-1075 besides, at most 2^-47 of its
    # unit, over a diagonal of at least 16 times a solution of at least 1/4: 81 x 2 x 4 x 2^-49 = 1.2e-12.
    err = np.abs(unit - B @ y) / (abs(B) @ np.abs(y) + np.abs(unit))
    assert err.max() < (2.3e-13 + (1.2e-12 if target < 0 else 0.0)), err.max()
    # The checked solve, and an ordinary matrix again after it.
    check, v0, rhs = _native.XdRfCheck(), torch.as_tensor(A.data, device="cuda"), torch.as_tensor(A @ x, device="cuda")
    for vv, bb, want in ((v, torch.as_tensor(b, device="cuda"), y), (v0, rhs, None)):
        got.zero_()
        torch.cuda.synchronize()
        assert lib.xd_rf_solve_refined(h, p(vv), p(bb), p(got), 1, 1e-10, 3, ctypes.byref(check)) == 0
        torch.cuda.synchronize()
        assert (check.outcome, check.solves) == (_native.XD_RF_WITHIN_TOL, 1)
        assert want is None or np.array_equal(got.cpu().numpy(), want)
    lib.xd_rf_destroy(h)
