"""Gathers of the same stamps that overlap on two streams: rows of one chunk and of several, each into
outputs of its own, against the same gathers one after the other, bit for bit; a load after them; and
a captured load."""
import ctypes

import numpy as np
import pytest

from xyce_b200 import MosfetDevice, SolverFlags, _native, netlist

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_overlapping_gathers():
    c = netlist.random_logic(30_000, seed=4, n_inputs=8)
    pat = netlist.jacobian_pattern(c)
    dev = MosfetDevice(*netlist.mosfet_family(c), pat, c.n_unknowns, level=14)
    lib, nu, nnz = _native.load(), c.n_unknowns, int(pat[0][-1])
    z = lambda k: torch.zeros(k, dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    state = lambda: [z(dev.n_state), z(dev.n_state), z(dev.n_store), z(dev.n_store)]
    x = torch.as_tensor(np.random.default_rng(1).uniform(0.0, c.vdd, nu), device="cuda")
    want = [z(k) for k in (nu, nu, nu, nu, nnz, nnz)]
    flags = SolverFlags(newton_iter=1, transient=1)
    for _ in range(2):  # (a context's first load differs from the later ones by its devices' own history)
        for w in want:
            w.zero_()
        dev.load(flags, x, *state(), *want)
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(50):
        outs = [[z(len(w)) for w in want] for _ in streams]
        torch.cuda.synchronize()
        for s, o in zip(streams, outs):
            st = ctypes.c_void_p(s.cuda_stream)
            _native.check(lib.xd_load_vectors(dev._h, *[p(t) for t in o[:4]], st), "xd_load_vectors")
            _native.check(lib.xd_load_matrices(dev._h, p(o[4]), p(o[5]), st), "xd_load_matrices")
        torch.cuda.synchronize()
        for o in outs:
            assert all(torch.equal(a, b) for a, b in zip(o, want))
    again = [z(len(w)) for w in want]
    dev.load(flags, x, *state(), *again)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(again, want))
    # The same load as a graph: its launches' dependence is captured with them.
    held, side = state(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        for a in again:
            a.zero_()
        dev.load(flags, x, *held, *again)
    for _ in range(5):
        for s in held:
            s.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(again, want))
