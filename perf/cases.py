"""The work users of this package have it do, as callable cases.

A case names a path (``kind``), a size and the options in use. ``prepare`` makes what a user's
program holds before the call (circuit, device family, solver state, handles), ``run`` makes one
pass through the public entry points (the classes of ``xyce_b200`` and the C ABI of ``include/``),
``work`` gives the bytes and operations a pass cannot do without, and ``exact`` the 64-bit result
where plain numpy gives one: the sparse solve and the surrogate. A compact model's load, and a
transient built on it, have no restatement in plain numpy.

The circuits are the package's own seeded generators at a fixed netlist seed (a program simulates
one circuit at many iterates); the iterates, matrix values, right-hand sides and samples come from
the case's seed.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from xyce_b200 import ModelCard, MosfetDevice, SolverFlags, _native, netlist
from xyce_b200.device import internal_nodes
from xyce_b200.surrogate import N_HID, N_IN, N_LAYERS, N_OUT, PAD_IN, PAD_OUT, AdamConfig, SurrogateMLP
from xyce_b200.transient import GpuTransient, NewtonParams, tia_coef

NETLIST_SEED = 2026
DEV = "cuda:0"
H = 10e-12  # time step of the transients (s)


def listed():
    return [
        # Smallest load: the 101-stage ring oscillator's 202 BSIM3 devices, once per Newton iteration.
        {"name": "ring_load", "kind": "load", "family": "bsim3", "circuit": "ring", "n": 101, "flags": "tran"},
        # Monte-Carlo sweep: many circuits with their own cards merged into one family, operating point.
        {"name": "sweep_load", "kind": "load", "family": "bsim4", "circuit": "sweep", "n": 32, "flags": "dcop"},
        # The scale benchmark: ~1M BSIM4 devices with RC ladders at a transient iterate.
        {"name": "scale_load", "kind": "load", "family": "bsim4", "circuit": "logic", "n": 1_000_000, "flags": "tran"},
        # Gate/body resistance networks, rdsMod and NQS: the general 15-node topology.
        {"name": "general_load", "kind": "load", "family": "bsim4gen", "circuit": "logic", "n": 60_000, "flags": "tran"},
        # Level-1 devices, the cheap model, bound by memory and assembly.
        {"name": "mos1_load", "kind": "load", "family": "mos1", "circuit": "logic", "n": 300_000, "flags": "tran"},
        # One Newton iterate's load and combine as the transient of the placed netlist makes it.
        {"name": "load_combine", "kind": "combine", "n": 100_000, "limiter": True, "order": 2},
        # Refactor and solve of a small circuit's Newton matrix (any-net wiring, dense fill).
        {"name": "newton_small", "kind": "newton", "n": 1_200},
        # Refactor and solve at the placed-netlist benchmark's size (200k unknowns).
        {"name": "newton_placed", "kind": "newton", "n": 100_000},
        # Whole call: the BSIM3 ring through 40 time steps (dense solves, graph-replayed iterations).
        {"name": "ring_transient", "kind": "ring", "n": 101, "steps": 40},
        # Whole call: a placed BSIM4 netlist through 4 time steps on the sparse refactorization.
        {"name": "placed_transient", "kind": "placed", "n": 20_000, "steps": 4},
        # One training step of the surrogate at its training batch.
        {"name": "surrogate_train", "kind": "train", "n": 16_384},
        # Surrogate inference over a large circuit's devices.
        {"name": "surrogate_forward", "kind": "forward", "n": 250_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case over the same paths: each size from the smallest to the largest in use."""
    kind = rng.choice(["load", "load", "load", "combine", "newton", "newton", "ring", "placed", "train", "forward"])
    if kind == "load":
        family = rng.choice(["bsim3", "bsim4", "bsim4", "bsim4gen", "mos1"])
        flags = rng.choice(["tran", "dcop"])
        circuit = rng.choice(["logic", "ring"] if family in ("bsim3", "mos1") else
                             ["logic", "sweep"] if family == "bsim4" else ["logic"])
        n = {"ring": lambda: 2 * rng.randint(5, 250) + 1, "sweep": lambda: rng.randint(2, 40),
             "logic": lambda: _log_int(rng, 200, 100_000 if family == "bsim4gen" else 500_000)}[circuit]()
        return {"kind": kind, "family": family, "circuit": circuit, "n": n, "flags": flags}
    if kind == "combine":
        return {"kind": kind, "n": _log_int(rng, 300, 200_000), "limiter": rng.random() < 0.7,
                "order": rng.choice([1, 2])}
    if kind == "newton":
        return {"kind": kind, "n": _log_int(rng, 300, 60_000)}
    if kind == "ring":
        return {"kind": kind, "n": 2 * rng.randint(5, 77) + 1, "steps": rng.randint(10, 60)}
    if kind == "placed":
        return {"kind": kind, "n": _log_int(rng, 500, 30_000), "steps": rng.randint(2, 6)}
    if kind == "train":
        return {"kind": kind, "n": _log_int(rng, 500, 50_000)}
    return {"kind": kind, "n": _log_int(rng, 300, 1_000_000)}


# ---- circuits ------------------------------------------------------------------------------------

def _locality(n):
    """Small netlists are wired any-to-any; larger ones are placed (a pin takes a nearby net)."""
    return 0 if n < 2_000 else 64


@functools.lru_cache(maxsize=4)
def _circuit(circuit, n, locality=0):
    """(circuit, CSR pattern, sweep batch or None) of a case: the netlist a user's program has read."""
    batch = None
    if circuit == "ring":
        c = netlist.inverter_ring(n, vdd=1.8)
    elif circuit == "sweep":
        batch = netlist.batched_sweep(n, 1000, 20000, seed=NETLIST_SEED)
        c = batch.circuit
    else:
        c = netlist.random_logic(n, seed=NETLIST_SEED, wire_segments=4 if n > 400_000 else 2, locality=locality)
    return c, netlist.jacobian_pattern(c), batch


@functools.lru_cache(maxsize=2)
def _general(n):
    """The general-topology cards and circuit: NMOS with gate-mid, body and charge nodes and
    bias-dependent S/D resistance, PMOS with the gate node and the geometry-scaled body network."""
    c = _circuit("logic", n)[0]
    cards = [ModelCard(False, {"RGATEMOD": 3, "RBODYMOD": 1, "RDSMOD": 1, "TRNQSMOD": 1, "RSH": 20.0}),
             ModelCard(True, {"RGATEMOD": 2, "RBODYMOD": 2, "RBPS0": 60.0, "RBPD0": 70.0})]
    family = netlist.mosfet_family(c, cards, {"NRD": np.full(c.n_mos, 2.0), "NRS": np.full(c.n_mos, 1.5)})
    flags, _ = internal_nodes(*family, general=True)
    c = netlist.with_internal_nodes(c, flags)
    return c, netlist.jacobian_pattern(c), family


def _f64(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=DEV)


def _p(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _family(case):
    """The case's device family: (circuit, pattern, MosfetDevice)."""
    if case["family"] == "bsim4gen":
        c, pat, fam = _general(case["n"])
        return c, pat, MosfetDevice(*fam, pat, c.n_unknowns, level=14, inst_internal=c.mos_internal)
    c, pat, batch = _circuit(case["circuit"], case["n"])
    if batch is not None:
        return c, pat, MosfetDevice(batch.cards, batch.inst_model, c.mos_nodes, batch.inst_params, pat, c.n_unknowns,
                                    level=14)
    cards = netlist.ring_bsim3_cards() if case["family"] == "bsim3" else None
    level = {"bsim3": 9, "bsim4": 14, "mos1": 1}[case["family"]]
    return c, pat, MosfetDevice(*netlist.mosfet_family(c, cards), pat, c.n_unknowns, level=level)


class _LoadState:
    """Buffers of one family: device history, the iterate, and the outputs as the loader holds them."""

    def __init__(self, c, pat, fam, rng):
        self.c, self.fam = c, fam
        z = lambda k: torch.zeros(k, dtype=torch.float64, device=DEV)
        self.sta, self.csta, self.sto, self.csto = z(fam.n_state), z(fam.n_state), z(fam.n_store), z(fam.n_store)
        nu, nnz = c.n_unknowns, int(pat[0][-1])
        self.flat = z(4 * nu + 2 * nnz)  # F, Q, both limiter vectors, dF/dx, dQ/dx: zeroed as one buffer
        self.out = list(torch.split(self.flat, [nu] * 4 + [nnz] * 2))
        # The previous iterate (its limited junction voltages become the store) and the one to load.
        x0 = rng.uniform(0.0, c.vdd, nu)
        self.x = _f64(x0 + rng.normal(0.0, 0.02, nu))
        fam.load(SolverFlags(newton_iter=1, voltlim=0), _f64(x0), self.sta, self.csta, self.sto, self.csto, *self.out)
        self.csto.copy_(self.sto)
        self.csta.copy_(self.sta)


def _linear(c, pat):
    """The linear devices' constant dF/dx and dQ/dx, as the transient driver assembles them."""
    from xyce_b200.transient import LinearDevices

    lin = LinearDevices(c, np.asarray(pat[0]), np.asarray(pat[1]))
    return lin.lin_f, lin.lin_q


# ---- Newton matrices of the sparse solve ---------------------------------------------------------

@functools.lru_cache(maxsize=2)
def _stamps(n):
    """Where each device's conductances go in the CSR values: (circuit, pattern, matrix positions)."""
    c, pat, _ = _circuit("logic", n, _locality(n))
    nu = c.n_unknowns
    key = np.repeat(np.arange(nu, dtype=np.int64), np.diff(pat[0])) * nu + pat[1]

    def two(a, b):  # a conductance between a and b: positions of (aa, ab, ba, bb), -1 with ground
        r, cc = np.stack([a, a, b, b]).astype(np.int64), np.stack([a, b, a, b]).astype(np.int64)
        return np.where((r >= 0) & (cc >= 0), np.searchsorted(key, np.maximum(r, 0) * nu + np.maximum(cc, 0)), -1)

    def trans(d, s, a, b):  # a current d -> s controlled by V(a) - V(b)
        r, cc = np.stack([d, d, s, s]).astype(np.int64), np.stack([a, b, a, b]).astype(np.int64)
        return np.where((r >= 0) & (cc >= 0), np.searchsorted(key, np.maximum(r, 0) * nu + np.maximum(cc, 0)), -1)

    D, G, S, B = (c.mos_nodes[:, k] for k in range(4))
    br = np.arange(c.n_nodes, c.n_nodes + c.n_vsrc, dtype=np.int64)
    p = c.vsrc_nodes[:, 0].astype(np.int64)
    src = np.concatenate([np.searchsorted(key, p * nu + br), np.searchsorted(key, br * nu + p)])
    return c, pat, {"res": two(*c.res_nodes.T), "cap": two(*c.cap_nodes.T), "gds": two(D, S), "gm": trans(D, S, G, S),
                    "gmb": trans(D, S, B, S), "cgs": two(G, S), "cgd": two(G, D), "cdb": two(D, B), "csb": two(S, B),
                    "src": src}


def _newton_system(case, seed):
    """(circuit, pattern, first matrix, later matrix, right-hand side): J = G + C / h of the netlist
    with the wires' R and C and small-signal conductances and capacitances of switching and idle
    transistors; the later matrix has the transistors moved on, as in the next Newton iteration."""
    c, pat, at = _stamps(case["n"])
    rng = np.random.default_rng([seed, case["n"]])
    m, nnz = c.n_mos, int(pat[0][-1])
    lin = {"res": 1.0 / c.res_value, "cap": c.cap_value / H}
    lo = lambda a, b: np.exp(rng.uniform(math.log(a), math.log(b), m))
    dev = {"gds": lo(1e-9, 1e-3), "gm": lo(1e-9, 1e-3), "gmb": lo(1e-10, 2e-4), "cgs": lo(2e-16, 2e-15) / H,
           "cgd": lo(2e-16, 2e-15) / H, "cdb": lo(5e-16, 2e-15) / H, "csb": lo(5e-16, 2e-15) / H}

    def values(moved):
        v = np.zeros(nnz)
        for name, g in {**lin, **dev}.items():
            if moved and name in dev:
                g = g * np.exp(rng.normal(0.0, 0.3, m))
            pos = at[name]
            w = np.stack([g, -g, -g, g])
            ok = pos >= 0
            v += np.bincount(pos[ok], weights=w[ok], minlength=nnz)
        v[at["src"]] = 1.0
        return v

    return c, pat, values(False), values(True), rng.normal(0.0, 1e-5, c.n_unknowns)


# ---- the cases -----------------------------------------------------------------------------------

def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng([seed, case["n"]])
    if kind == "load":
        s = _LoadState(*_family(case), rng)
        s.kind = kind
        s.flags = (SolverFlags(newton_iter=2, pdt=1.0 / H) if case["flags"] == "tran" else
                   SolverFlags(newton_iter=2, dcop=1, transient=0, tranop=1))
        return s
    if kind == "combine":
        c, pat, _ = _circuit("logic", case["n"], _locality(case["n"]))
        fam = MosfetDevice(*netlist.mosfet_family(c), pat, c.n_unknowns, level=14)
        s = _LoadState(c, pat, fam, rng)
        s.kind, s.flags = kind, SolverFlags(newton_iter=2, pdt=1.0 / H)
        s.lib = _native.load()
        csr = _native.XdCsr(c.n_unknowns, pat[0].ctypes.data_as(_native._ip), pat[1].ctypes.data_as(_native._ip))
        s.tia, s.fused = ctypes.c_void_p(), ctypes.c_void_p()
        _native.check(s.lib.xd_tia_create(ctypes.byref(csr), 0, ctypes.byref(s.tia)), "xd_tia_create")
        _native.check(s.lib.xd_tia_fused_create(s.tia, fam._h, ctypes.byref(s.fused)), "xd_tia_fused_create")
        s.lin = [_f64(a) for a in _linear(c, pat)]
        nu = c.n_unknowns
        s.b, s.qn0, s.fh = (_f64(rng.normal(0.0, k, nu)) for k in (0.1, 1e-15, 1e-5))
        s.limiter, s.coef = int(case["limiter"]), tia_coef(1, H, case["order"])
        s.jac = torch.zeros(int(pat[0][-1]), dtype=torch.float64, device=DEV)
        s.vec = [torch.zeros(nu, dtype=torch.float64, device=DEV) for _ in range(3)]
        s.flat.zero_()
        return s
    if kind == "newton":
        c, pat, first, later, b = _newton_system(case, seed)
        s = _State(kind=kind, lib=_native.load())
        s.fam = MosfetDevice(*netlist.mosfet_family(c), pat, c.n_unknowns, level=14)
        s.tr = GpuTransient(c, s.fam, *pat, solver="rf")
        s.tr.jac.copy_(_f64(first))
        s.tr._rf_setup()  # one host factorization: pivot order and fill of every later matrix
        s.vals, s.b = _f64(later), _f64(b)
        s.x = torch.empty_like(s.b)
        return s
    if kind in ("ring", "placed"):
        s = _State(kind=kind, steps=case["steps"])
        if kind == "ring":
            c, pat, _ = _circuit("ring", case["n"])
            s.fam = MosfetDevice(*netlist.mosfet_family(c, netlist.ring_bsim3_cards()), pat, c.n_unknowns, level=9)
            s.tr = GpuTransient(c, s.fam, *pat)
            # Alternating rails with one travelling edge, the outputs slightly off the rails.
            x = np.zeros(c.n_unknowns)
            x[0] = c.vdd
            x[1:c.n_nodes] = np.where(np.arange(c.n_nodes - 1) % 2 == 0, 0.0, c.vdd) * rng.uniform(0.97, 1.0)
            x[1:c.n_nodes] += rng.uniform(0.0, 0.02, c.n_nodes - 1)
            s.x0 = _f64(x)
        else:
            c, pat, _ = _circuit("logic", case["n"], _locality(case["n"]))
            s.fam = MosfetDevice(*netlist.mosfet_family(c), pat, c.n_unknowns, level=14)
            s.tr = GpuTransient(c, s.fam, *pat, solver="rf")
            # Operating point from the inputs' logic levels; the run starts a little off it.
            s.tr.dcop(x0=netlist.logic_initial_guess(c))
            x = s.tr.x.clone()
            x[1:c.n_nodes] += _f64(rng.normal(0.0, 0.01, c.n_nodes - 1))
            s.x0 = x
            s.tr.set_initial_state(s.x0)
            s.tr.run(H, H, params=NewtonParams.transient())  # the time steps' pivot order is in hand
        return s
    s = _State(kind=kind, n=case["n"])
    s.net = SurrogateMLP(seed=seed, max_batch=case["n"])
    x, t = _samples(case, seed)
    if kind == "train":
        s.x, s.t, s.cfg = torch.as_tensor(x, device=DEV), torch.as_tensor(t, device=DEV), AdamConfig()
    else:
        s.net.X32[:case["n"], :N_IN] = torch.as_tensor(x, device=DEV)
    return s


class _State:
    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        if getattr(self, "tr", None) is not None:
            self.tr.close()


def _combine_del(self):
    if getattr(self, "fused", None) is not None:
        self.lib.xd_tia_fused_destroy(self.fused)
        self.lib.xd_tia_destroy(self.tia)


_LoadState.__del__ = _combine_del


def _samples(case, seed):
    """Surrogate inputs uniform over the training box, targets of the encoded outputs' size."""
    rng = np.random.default_rng([seed, case["n"]])
    x = rng.uniform(-1.0, 1.0, (case["n"], N_IN)).astype(np.float32)
    t = np.stack([np.sin((k + 1) * x[:, 0] + x[:, k % N_IN]) * 3.0 + x[:, 3] * k for k in range(N_OUT)], 1)
    return x, t.astype(np.float32)


def run(s):
    if s.kind == "load":
        s.flat.zero_()  # the loader's zeroing: devices only add
        s.fam.load(s.flags, s.x, s.sta, s.csta, s.sto, s.csto, *s.out)
        return {"f": s.out[0], "q": s.out[1], "fx": s.out[2], "qx": s.out[3], "jf": s.out[4], "jq": s.out[5],
                "sta": s.sta, "sto": s.sto}
    if s.kind == "combine":
        f = s.flags.to_c()
        _native.check(s.lib.xd_tia_load_combine(
            s.fused, ctypes.byref(f), ctypes.byref(s.coef), _p(s.x), _p(s.sta), _p(s.csta), _p(s.sto), _p(s.csto),
            *[_p(t) for t in s.out], _p(s.lin[0]), _p(s.lin[1]), s.limiter, _p(s.b), _p(s.qn0), _p(s.fh), _p(s.jac),
            *[_p(t) for t in s.vec], _stream()), "xd_tia_load_combine")
        return {"jac": s.jac, "rhs": s.vec[0], "qtot": s.vec[1], "ftot": s.vec[2], "sta": s.sta, "sto": s.sto}
    if s.kind == "newton":
        s.x.copy_(s.b)
        _native.check(s.lib.xd_rf_refactor(s.tr._rf, _p(s.vals)), "xd_rf_refactor")
        _native.check(s.lib.xd_rf_solve(s.tr._rf, _p(s.x)), "xd_rf_solve")
        return {"x": s.x}
    if s.kind in ("ring", "placed"):
        s.tr.set_initial_state(s.x0)
        times, waves = s.tr.run(s.steps * H, H, params=NewtonParams.transient())
        return {"times": times, "waves": waves, "q": s.tr.qtot, "f": s.tr.ftot, "sta": s.tr.curr_sta, "sto": s.tr.curr_sto}
    if s.kind == "train":
        loss = s.net.train_step(s.x, s.t, s.cfg)
        return {"loss": loss, "gW": s.net.gW, "gb": s.net.gb, "W": s.net.W, "b": s.net.b}
    return {"y": s.net.forward_fused(s.n)}


# FP64 operations and unknowns / nonzeros per device of the paths, for ``work``: the compact models'
# executed counts, and the placed netlists' factor sizes.
_FLOPS = {"bsim4": 6600.0, "bsim4gen": 8000.0, "bsim3": 5000.0, "mos1": 600.0}


def _load_bytes(c, nnz, n_state, n_store):
    m = c.n_mos
    return m * (16 + 4 + 40 + 8 * n_state + 8 * n_store) + 8.0 * (c.n_unknowns * 5 + 2 * nnz)


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "load":
        if case["family"] == "bsim4gen":
            c, pat, _ = _general(n)
        else:
            c, pat, _ = _circuit(case["circuit"], n)
        ns = {"bsim4": (3, 14), "bsim4gen": (8, 14), "bsim3": (5, 5), "mos1": (8, 5)}[case["family"]]
        return {"bytes": _load_bytes(c, int(pat[0][-1]), *ns), "flops": _FLOPS[case["family"]] * c.n_mos}
    if kind in ("combine", "newton", "placed"):
        c, pat, _ = _circuit("logic", n, _locality(n))
        nnz, nu = int(pat[0][-1]), c.n_unknowns
        load = {"bytes": _load_bytes(c, 0, 3, 14) + 8.0 * (3 * nnz + 8 * nu), "flops": _FLOPS["bsim4"] * c.n_mos}
        solve = {"bytes": 8.0 * (nnz + 2 * nu), "flops": 2.0 * 60 * nu + 4.0 * 9 * nu}
        if kind == "combine":
            return load
        if kind == "newton":
            return solve
        return {k: 2.0 * case["steps"] * (load[k] + solve[k]) for k in load}
    if kind == "ring":
        iters = 3.0 * case["steps"]
        return {"bytes": iters * 2 * n * 400.0, "flops": iters * 2 * n * _FLOPS["bsim3"]}
    macs = N_IN * N_HID + (N_LAYERS - 1) * N_HID * N_HID + N_HID * N_OUT
    if kind == "train":
        return {"bytes": 4.0 * n * (N_IN + N_OUT) + 28.0 * macs, "flops": 6.0 * n * macs}
    return {"bytes": 4.0 * n * (N_IN + N_OUT), "flops": 2.0 * n * macs}


def _weights(seed):
    """The network's initial weights in the precision it computes with, as float64 (host)."""
    g = torch.Generator().manual_seed(seed)
    dims = [(N_HID, N_IN)] + [(N_HID, N_HID)] * (N_LAYERS - 1) + [(N_OUT, N_HID)]
    w = [(torch.rand(o, i, generator=g) * 2 - 1) * math.sqrt(6.0 / (i + o)) for o, i in dims]
    return [w[0].double()] + [a.to(torch.bfloat16).double() for a in w[1:]]


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "newton" and n <= 1_500:
        c, pat, _, v, b = _newton_system(case, seed)
        a = np.zeros((c.n_unknowns, c.n_unknowns))
        a[np.repeat(np.arange(c.n_unknowns), np.diff(pat[0])), pat[1]] = v
        x = np.linalg.solve(a, b)
        return {"x": x + np.linalg.solve(a, b - a @ x)}
    if kind not in ("train", "forward"):
        return None
    x, t = (torch.as_tensor(a).double() for a in _samples(case, seed))
    w = _weights(seed)
    h, zs, hs = x, [], [x]
    for a in w[:-1]:
        zs.append(h @ a.T)
        h = zs[-1] * torch.sigmoid(zs[-1])
        hs.append(h)
    y = h @ w[-1].T
    if kind == "forward":
        return {"y": y}
    d = 2.0 * (y - t) / (n * N_OUT)
    gw, gb = [None] * len(w), [None] * len(w)
    for k in range(len(w) - 1, -1, -1):
        po, pi = (PAD_OUT if k == N_LAYERS else N_HID), (PAD_IN if k == 0 else N_HID)
        gw[k], gb[k] = torch.zeros(po, pi, dtype=torch.float64), torch.zeros(po, dtype=torch.float64)
        gw[k][:w[k].shape[0], :w[k].shape[1]] = d.T @ hs[k]
        gb[k][:w[k].shape[0]] = d.sum(0)
        if k:
            sg = torch.sigmoid(zs[k - 1])
            d = (d @ w[k]) * (sg * (1.0 + zs[k - 1] * (1.0 - sg)))
    return {"loss": ((y - t) ** 2).mean(), "gW": gw, "gb": gb, "W": None, "b": None}
