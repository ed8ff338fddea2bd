"""Which route of the elimination-tree plan (csrc/lutree_plan.cpp) a matrix takes, asked of the plan
itself on the host, and the factorization and solve of those that take the long lists: destinations
and rows with so many entries that a warp or a block takes them, rows solved last in several chunks,
and columns outside the panels."""
import json
import os
import shutil
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from tests import test_rf_tree_gpu as tree
from xyce_b200 import build

FIGURES = r"""
#include <algorithm>
#include <cstdio>
#include "lutree.h"
int main(int, char **argv) {
  FILE *f = fopen(argv[1], "rb");
  int n = 0, nnz = 0;
  auto get = [&](int *p, size_t k) { if (fread(p, 4, k, f) != k) throw 1; };
  get(&n, 1);
  get(&nnz, 1);
  std::vector<int> mp(n + 1), mi(nnz), diag(n);
  get(mp.data(), n + 1);
  get(mi.data(), nnz);
  for (int i = 0; i < n; ++i) diag[i] = (int)(std::lower_bound(&mi[mp[i]], &mi[0] + mp[i + 1], i) - &mi[0]);
  XdTreePlan p;
  const bool on = xd_tree_plan(n, mp, mi, diag, &p);
  int pairs = 0, schur = 0, row = 0, tail = 0, lanes = 0;
  for (const XdPos4 &q : p.fwd.pass) lanes = std::max(lanes, 1 << (q.y >> 16 & 0xff));
  for (const XdPos4 &d : p.dst) pairs = std::max(pairs, d.w < 0 ? d.z : 1);
  for (size_t k = 0; k + 1 < p.sptr.size(); ++k) schur = std::max(schur, p.sptr[k + 1] - p.sptr[k]);
  for (size_t k = 0; k + 1 < p.lptr.size(); ++k) row = std::max(row, p.lptr[k + 1] - p.lptr[k]);
  for (size_t k = 0; k + 1 < p.tptr.size(); ++k) tail = std::max(tail, p.tptr[k + 1] - p.tptr[k]);
  // Long destinations stand behind the others of their level.
  bool order = p.llong.size() + 1 == p.ldst.size();
  for (size_t l = 0; order && l < p.llong.size(); ++l)
    for (int d = p.ldst[l]; d < p.ldst[l + 1]; ++d)
      order = order && (p.dst[d].w < 0 && p.dst[d].z > kLongPairs) == (d >= p.llong[l]);
  printf("{\"plan\": %d, \"frame\": %d, \"groups\": %d, \"chains\": %d, \"joins\": %zu, \"top\": %d, \"pairs\": %d, "
         "\"long\": %d, \"order\": %d, \"schur\": %d, \"lanes\": %d, \"row\": %d, \"tail\": %d, \"tdiv\": %zu}\n",
         on, p.F, p.ngroups, p.nchains, p.jchild.size(), p.ntop, pairs, p.any_long, order, schur, lanes, row, tail, p.tdiv.size());
}
"""


@pytest.fixture(scope="module")
def figures(tmp_path_factory):
    nvcc = os.path.realpath(build._which(build._nvcc()))
    include = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    if shutil.which("g++") is None or not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no host C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("plan")
    (d / "figures.cpp").write_text(FIGURES)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", build.CSRC, "-I", include, str(d / "figures.cpp"),
                    os.path.join(build.CSRC, "lutree_plan.cpp"), "-o", str(d / "figures")], check=True)

    def ask(A):
        lu = spl.splu(A.tocsc(), permc_spec="NATURAL", diag_pivot_thresh=0.0, options=dict(SymmetricMode=True))
        assert np.array_equal(lu.perm_r, np.arange(A.shape[0]))
        M = sp.csr_matrix(abs(sp.tril(lu.L, -1)) + abs(lu.U))
        M.sort_indices()
        with open(d / "m.bin", "wb") as f:
            for a in ([A.shape[0], M.nnz], M.indptr, M.indices):
                np.asarray(a, np.int32).tofile(f)
        return json.loads(subprocess.run([str(d / "figures"), str(d / "m.bin")], check=True, capture_output=True).stdout)

    return ask


def arrows(sizes, linked=False):
    """Hubs with the given numbers of leaves, the leaves of each before it; linked: each hub to the next."""
    n = sum(sizes) + len(sizes)
    hub = np.cumsum(np.asarray(sizes) + 1) - 1
    leaf = np.setdiff1d(np.arange(n), hub)
    a = sp.coo_matrix((np.ones(len(leaf)), (leaf, np.repeat(hub, sizes))), shape=(n, n))
    if linked:
        a = a + sp.coo_matrix((np.ones(len(hub) - 1), (hub[:-1], hub[1:])), shape=(n, n))
    return sp.csr_matrix(a + a.T + sp.identity(n))


def rail(n, w, at_row=None):
    """test_rf_tree_gpu's rails for many unknowns; the rail's voltage last, or at a row in between."""
    band = sp.block_diag([sp.csr_matrix((1, 1)), tree.band(n, w), sp.csr_matrix((1, 1))])
    at = np.arange(1, n + 1)
    full = np.concatenate([np.zeros(n + 2), at, [n + 1]]), np.concatenate([np.arange(n + 2), np.full(n, n + 1), [n + 1]])
    A = sp.csr_matrix(band + sp.coo_matrix((np.ones(len(full[0])), full), shape=(n + 2, n + 2)))
    order = np.arange(n + 2) if at_row is None else np.insert(np.arange(n + 1), at_row, n + 1)
    return sp.csr_matrix(A[order][:, order])


# Hubs of 31 to 34 leaves, at the border between a thread and a warp, and of 255 to 1,025, whose rows take
# a warp and up to eight; a subtree with more entries than
# shared memory holds; hubs above the subtree limit, whose updates (from 513) and rows (from 1025) a
# block takes; a rail in three chunks; a rail's voltage whose column reaches rows on both sides and
# whose own row is empty.
LONG = {"arrows31to34": lambda: arrows([31, 32, 33, 34] * 45),
        "arrows256up": lambda: arrows([255, 256, 257, 300, 512, 513, 600, 1024, 1025] * 2, linked=True),
        "arrow6000": lambda: arrows([6000]),
        "path_of_hubs": lambda: arrows([11000, 512, 513, 1024, 1025, 1], linked=True),
        "rail5000": lambda: rail(5000, 23),
        "rail_between": lambda: rail(3000, 23, 700)}


def matrix(name):
    make = LONG.get(name) or tree.CASES[name]
    return tree.dominant(make(), np.random.default_rng(len(name)))


def test_long_lists_take_their_routes(figures):
    f = {k: figures(matrix(k)) for k in LONG}
    assert all(v["plan"] and v["order"] for v in f.values()), f
    assert (f["arrows31to34"]["pairs"], f["arrows31to34"]["long"], f["arrows31to34"]["chains"]) == (34, 1, 0)
    assert (f["arrow6000"]["pairs"], f["arrow6000"]["groups"], f["arrow6000"]["chains"]) == (6000, 1, 0)
    assert (f["arrow6000"]["lanes"], f["arrows31to34"]["lanes"]) == (512, 32)
    assert f["arrows256up"]["lanes"] == 256
    assert (f["path_of_hubs"]["schur"], f["path_of_hubs"]["row"], f["path_of_hubs"]["top"]) == (11000, 11000, 6)
    assert f["rail5000"]["chains"] > 0 and f["rail5000"]["tail"] > 2 * 2048
    assert f["rail_between"]["chains"] > 0 and f["rail_between"]["tdiv"] > 2000


def test_the_other_tests_matrices_take_their_routes(figures):
    f = {k: figures(matrix(k)) for k in tree.CASES}
    lists = {"band129x1", "band300x121", "dense130", "diagonal", "random"}  # the level lists
    assert {k for k, v in f.items() if not v["plan"]} == lists
    for k in set(f) - lists:
        n, w = (int(q) for q in k[4:].split("x")) if k.startswith("band") else (0, 0)
        assert f[k]["chains"] >= 1 and f[k]["order"] and not f[k]["long"], k
        assert not n or (f[k]["frame"] == -(-(w + 8) // 16) * 16 and f[k]["top"] > n - 70), (k, f[k])
    assert (f["comb3"]["joins"], f["comb6"]["joins"], f["rails"]["tail"]) == (2, 5, 901)


@pytest.mark.gpu
@pytest.mark.parametrize("name", LONG)
def test_long_lists(name):
    """Backward error of the solution. A row sums at most 11,001 products, each with a few roundings, in
    an order of depth at most 1,000 (6,000 over 32 lanes is 188 deep, then a tree; a chunk of a rail 8,
    a chain's row at most 100), in factors that a dominant diagonal keeps from growing (by at most 2):
    1,000 x 2 x 4 x 1.1e-16 = 8.9e-13. The check's own products run in sequence: 11,001 x 1.1e-16 = 1.3e-12."""
    rng = np.random.default_rng(len(name))
    A = matrix(name)
    rf = tree.Rf(A)
    B = tree.dominant(A, rng)
    assert rf.refactor(B.data) == 0, rf.lib.xd_last_error()
    b = rng.standard_normal(A.shape[0])
    x, f1 = rf.solve(b), rf.factors()
    assert (np.abs(b - B @ x) / (abs(B) @ np.abs(x) + np.abs(b))).max() < 2.2e-12
    assert rf.refactor(B.data) == 0 and np.array_equal(rf.factors(), f1) and np.array_equal(rf.solve(b), x)
    rf.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", tree.CASES)
def test_factors_of_the_other_tests_are_compared(name):
    """The factor check of test_rf_tree_gpu reads the library's factors through the pattern of L's and U's
    entries, where both have as many: they have."""
    rf = tree.Rf(matrix(name))
    pat = sp.csr_matrix(abs(sp.tril(rf.L, -1)) + abs(rf.U))
    assert rf.factors().shape[0] == pat.nnz
    rf.close()
