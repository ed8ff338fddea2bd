"""The refactorization's elimination-tree path (csrc/lutree.h) at the structures where its plan
changes shape: chain lengths around a block of pivots, frames around multiples of 16 slots and at
the largest size, joining chains, update-free pivots, and matrices it leaves to the level lists."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from xyce_b200 import _native

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


class Rf:
    """xd_rf on a matrix in its natural order (P = Q = identity), L and U from the host."""

    def __init__(self, A):
        self.A = A = sp.csr_matrix(A)
        A.sort_indices()
        lu = spl.splu(A.tocsc(), permc_spec="NATURAL", diag_pivot_thresh=0.0, options=dict(SymmetricMode=True))
        assert np.array_equal(lu.perm_r, np.arange(A.shape[0]))
        self.L, self.U = lu.L.tocsr(), lu.U.tocsr()
        for m in (self.L, self.U):
            m.sort_indices()
        i32 = lambda a: np.ascontiguousarray(a, np.int32)
        self.keep = k = [i32(A.indptr), i32(A.indices), A.data.copy(), i32(self.L.indptr), i32(self.L.indices),
                         self.L.data, i32(self.U.indptr), i32(self.U.indices), self.U.data, i32(lu.perm_r)]
        ip = lambda a: a.ctypes.data_as(_native._ip)
        dp = lambda a: a.ctypes.data_as(_native._dp)
        self.lib, self.h = _native.load(), ctypes.c_void_p()
        _native.check(self.lib.xd_rf_create(A.shape[0], A.nnz, ip(k[0]), ip(k[1]), dp(k[2]), self.L.nnz, ip(k[3]),
                                            ip(k[4]), dp(k[5]), self.U.nnz, ip(k[6]), ip(k[7]), dp(k[8]), ip(k[9]),
                                            ip(k[9]), 0, ctypes.byref(self.h)), "xd_rf_create")

    def refactor(self, vals):
        v = torch.as_tensor(vals, device="cuda")
        torch.cuda.synchronize()
        return self.lib.xd_rf_refactor(self.h, ctypes.c_void_p(v.data_ptr()))

    def solve(self, b):
        x = torch.as_tensor(b, device="cuda").clone()
        torch.cuda.synchronize()
        _native.check(self.lib.xd_rf_solve(self.h, ctypes.c_void_p(x.data_ptr())), "xd_rf_solve")
        torch.cuda.synchronize()
        return x.cpu().numpy()

    def factors(self):
        n = ctypes.c_int()
        _native.check(self.lib.xd_rf_stats(self.h, ctypes.byref(n), ctypes.byref(ctypes.c_int()),
                                           ctypes.byref(ctypes.c_longlong())), "xd_rf_stats")
        out = np.zeros(n.value)
        _native.check(self.lib.xd_rf_copy_factors(self.h, out.ctypes.data_as(_native._dp)), "xd_rf_copy_factors")
        return out

    def close(self):
        self.lib.xd_rf_destroy(self.h)


def dominant(pattern, rng):
    """Random values on the pattern, rows dominated by their diagonals."""
    A = sp.csr_matrix(pattern)
    A.data[:] = rng.uniform(-1.0, 1.0, A.nnz)
    A.setdiag(0.0)
    d = np.asarray(abs(A).sum(1)).ravel() + rng.uniform(1.0, 2.0, A.shape[0])
    A = sp.csr_matrix(A + sp.diags(d))
    A.sort_indices()
    return A


def band(n, w):
    return sp.diags([np.ones(n - abs(k)) for k in range(-w, w + 1)], range(-w, w + 1)).tocsr()


def comb(teeth, n, w):
    """Bands that join one another: tooth t's last w variables also touch the spine."""
    A = sp.lil_matrix(((teeth + 1) * n, (teeth + 1) * n))
    for t in range(teeth + 1):
        A[t * n:(t + 1) * n, t * n:(t + 1) * n] = band(n, w)
    for t in range(teeth):
        at = teeth * n + (t * (n - w)) // teeth
        A[(t + 1) * n - w:(t + 1) * n, at:at + w] = 1.0
        A[at:at + w, (t + 1) * n - w:(t + 1) * n] = 1.0
    return A.tocsr()


def rails(n, w):
    """A band whose variables all touch a supply: first a current whose equation is the rail's long
    row, last the rail's voltage, set by a one-entry row."""
    A = sp.lil_matrix((n + 2, n + 2))
    A[1:n + 1, 1:n + 1] = band(n, w)
    A[0, :] = 1.0            # the rail's current balance, pivot: the source current's column
    A[1:n + 1, n + 1] = 1.0  # every variable's row reads the rail's voltage
    A[n + 1, n + 1] = 1.0    # the source's equation
    return A.tocsr()


CASES = {f"band{n}x{w}": (lambda n=n, w=w: band(n, w)) for n, w in
         ((129, 1), (700, 8), (701, 9), (703, 24), (705, 40), (711, 41), (704, 56), (709, 57), (400, 72),
          (400, 105), (397, 120), (300, 121))}
CASES |= {"comb3": lambda: comb(3, 220, 20), "comb6": lambda: comb(6, 181, 33), "rails": lambda: rails(900, 23),
          "dense130": lambda: band(130, 129), "diagonal": lambda: sp.identity(37).tocsr(),
          "random": lambda: sp.random(260, 260, 0.02, random_state=3, format="csr") + sp.identity(260)}


@pytest.mark.parametrize("name", CASES)
def test_factors_and_solutions(name):
    """The componentwise backward error of L U against A and of the solution. Each entry of L U sums
    at most min(n, 2 w + 1) <= 260 products of factors that a dominant diagonal keeps from growing
    (by at most 2), each with a few roundings: 260 x 2 x 4 x 1.1e-16 = 2.3e-13."""
    rng = np.random.default_rng(len(name))
    A = dominant(CASES[name](), rng)
    rf = Rf(A)
    vals = dominant(A, rng).data
    assert rf.refactor(vals) == 0, rf.lib.xd_last_error()
    B = sp.csr_matrix((vals, A.indices, A.indptr), shape=A.shape)
    # The bundled pattern is the closure of L's and U's: read the factors through their union.
    pat = sp.csr_matrix(abs(sp.tril(rf.L, -1)) + abs(rf.U))
    pat.sort_indices()
    f1 = rf.factors()
    if f1.shape[0] == pat.nnz:
        M = sp.csr_matrix((f1, pat.indices, pat.indptr), shape=A.shape)
        L, U = sp.tril(M, -1) + sp.identity(A.shape[0]), sp.triu(M)
        bound = (abs(L) @ abs(U)).toarray() + 1e-300
        assert (abs((L @ U - B).toarray()) / bound).max() < 2.3e-13
    b = rng.standard_normal(A.shape[0])
    x = rf.solve(b)
    assert (np.abs(b - B @ x) / (abs(B) @ np.abs(x) + np.abs(b))).max() < 2.3e-13
    # The same values again: the same bits.
    assert rf.refactor(vals) == 0 and np.array_equal(rf.factors(), f1) and np.array_equal(rf.solve(b), x)
    rf.close()


@pytest.mark.parametrize("row", [3, 650])
def test_zero_pivot_is_reported(row):
    """A pivot that becomes zero, in a bottom subtree and in a chain, is an error and not a solution."""
    rng = np.random.default_rng(5)
    A = dominant(band(700, 40), rng)
    rf = Rf(A)
    B = A.copy()
    for k in range(A.indptr[row], A.indptr[row + 1]):
        B.data[k] = 0.0
    assert rf.refactor(B.data) < 0
    assert rf.refactor(A.data) == 0
    b = rng.standard_normal(700)
    x = rf.solve(b)
    assert (np.abs(b - A @ x) / (abs(A) @ np.abs(x) + np.abs(b))).max() < 2.3e-13
    rf.close()
