"""The gather's two routes at their edges: a node shared by m MOSFETs, so that its row, column and
diagonal have m contributions (short up to 32, then chunks of 1024, combined by the last of up to
more than 256 chunks), against numpy's sums of the staged stamps; adding and assigning, and absolute
values."""
import numpy as np
import pytest

from xyce_b200 import MosfetDevice, SolverFlags, netlist

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m", [1, 32, 33, 1024, 1025, 257 * 1024 + 1])
def test_shared_node(m):
    cards, im, _, params = netlist.mosfet_family(netlist.random_logic(40, seed=1, n_inputs=4))
    # Drains of their own (2 ..), one gate (0), one source (1), bulk on ground.
    i = np.arange(m)
    nd = np.stack([i + 2, np.zeros(m), np.ones(m), -np.ones(m)], axis=1).astype(np.int32)
    nu = m + 2
    rows = [np.repeat(i + 2, 3), np.zeros(nu), np.ones(nu)]
    cols = [np.stack([np.zeros(m), np.ones(m), i + 2], axis=1).ravel(), np.arange(nu), np.arange(nu)]
    rows, cols = np.concatenate(rows).astype(np.int64), np.concatenate(cols).astype(np.int64)
    order = np.lexsort((cols, rows))
    rows, cols = rows[order], cols[order]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=nu))]).astype(np.int32)
    colind = cols.astype(np.int32)
    take = lambda a: np.ascontiguousarray(np.resize(np.asarray(a), m))
    dev = MosfetDevice(cards, take(im), nd, {k: take(v) for k, v in params.items()}, (rowptr, colind), nu)
    rng = np.random.default_rng(m)
    T = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")
    z = lambda k: torch.zeros(k, dtype=torch.float64, device="cuda")
    x = T(rng.uniform(0.0, 1.2, nu))
    sta, sto = [z(dev.n_state) for _ in range(2)], [z(dev.n_store) for _ in range(2)]
    start = [rng.standard_normal(k) for k in (nu, nu, nu, nu, len(cols), len(cols))]
    out = [T(a) for a in start]
    dev.load(SolverFlags(newton_iter=1, transient=1), x, sta[0], sta[1], sto[0], sto[1], *out)
    torch.cuda.synchronize()
    st = dev.copy_stamps()
    key = rows * nu + cols
    unit = 2.0**-53
    for absolute in (False, True):
        if absolute:
            out = [z(len(a)) for a in start]
            dev.load_abs(*out)
            torch.cuda.synchronize()
        for o in range(6):
            want, size = (np.zeros(len(start[o])) if absolute else start[o].copy()), np.abs(start[o])
            parts = []
            if o < 4:
                parts = [(nd[:, r], st[4 * o + r]) for r in range(4)]
            else:
                for r in range(4):
                    for c in range(4):
                        live = (nd[:, r] >= 0) & (nd[:, c] >= 0)
                        at = np.searchsorted(key, nd[:, r].astype(np.int64) * nu + nd[:, c])
                        parts.append((np.where(live, np.minimum(at, len(key) - 1), -1), st[16 * (o - 3) + 4 * r + c]))
            for at, v in parts:
                v = np.abs(v) if absolute else v
                np.add.at(want, at[at >= 0], v[at >= 0])
                np.add.at(size, at[at >= 0], np.abs(v[at >= 0]))
            # Sums of at most 2 m + 1 terms in two orders: each within (2 m + 1) * 2^-53 of the terms' size.
            err = np.abs(out[o].cpu().numpy() - want)
            assert (err <= 2 * (2 * m + 1) * unit * size).all(), (o, absolute, err.max())
