"""Measured workloads of gbrkc, through its public Python entry points.

Three kinds of case, each a dict of plain values:

* ``cells``: one engine of ``n`` systems of one cell type (``nx`` x ``ny`` cells
  each), advanced by ``iv`` output intervals of 0.125 ms a pass; the pass
  reads the output voltages, the elem voltages, calcium and the soma record
  back, as a stepping program does.
* ``batch``: the four cell types together in one engine (the benchmark's
  mixed batch, scaled), same pass.
* ``network``: the synaptic network workload, scaled; one launch and one
  synapse update per interval.
* ``serve``: a request server; a pass submits ``n`` requests, advances the
  server until all are done and reads them back.

Sizes, currents and shapes come from the repository's workloads
(configs.py), its tests and its benchmark.  A ``trial`` pass refills every
system with its own initial cell (Engine.reset_systems, as a repeated-trial
program does) and advances [0, iv] intervals, so every pass is the same work.
The other passes continue: prepare has advanced the engine by ``warm`` ms,
into the firing regime, and each pass covers the intervals after the last.

``exact`` integrates the first pass of the ``cells`` cases that start at t = 0
in numpy, in 64 bits, with platform exp/log and none of this repository's
numerics.
"""
from __future__ import annotations

import functools
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cerebellum-neuron-model-simulation-using-rkc_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import configs  # noqa: E402
import gbrkc as G  # noqa: E402
import morph as M  # noqa: E402

TYPES = {"gr": G.GR, "go": G.GO, "pkj": G.PKJ, "io": G.IO}
STIM_COMP = {"gr": 1, "go": 30, "pkj": 1599, "io": 0}
NCOND = {"gr": 10, "go": 13, "pkj": 11, "io": 8}


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the drop-in's loop: the olive network the reference ships as its example
        # size, one output interval per call -- the smallest call, all latency
        {"name": "olive 4x4 one interval", "kind": "cells", "type": "io", "n": 1, "nx": 4, "ny": 4, "prec": "fp64",
         "iv": 1, "sweep": False, "trial": False, "warm": 0},
        # the reference's full granule cell (578 compartments), stepped one
        # interval at a time: a few hundred short step attempts in a row
        {"name": "full granule one interval", "kind": "cells", "type": "grfull", "n": 1, "nx": 1, "ny": 1,
         "prec": "fp64", "iv": 1, "sweep": False, "trial": True, "warm": 0},
        # a granule population in mixed precision, one server quantum (8 intervals)
        {"name": "granules 512 mixed", "kind": "cells", "type": "gr", "n": 512, "nx": 1, "ny": 1, "prec": "mixed",
         "iv": 8, "sweep": False, "trial": True, "warm": 0},
        # the parameter sweep's granule half in plain FP64 (per-channel factors),
        # an odd number of instances
        {"name": "granule sweep 999 fp64", "kind": "cells", "type": "gr", "n": 999, "nx": 1, "ny": 1, "prec": "fp64",
         "iv": 4, "sweep": True, "trial": True, "warm": 0},
        # the parameter sweep's Golgi half in mixed precision
        {"name": "golgi sweep 2048 mixed", "kind": "cells", "type": "go", "n": 2048, "nx": 1, "ny": 1,
         "prec": "mixed", "iv": 8, "sweep": True, "trial": False, "warm": 20},
        # a small Golgi population in plain FP64: fewer systems than the GPU has warps
        {"name": "golgi 77 fp64", "kind": "cells", "type": "go", "n": 77, "nx": 1, "ny": 1, "prec": "fp64", "iv": 5,
         "sweep": False, "trial": True, "warm": 0},
        # the reference-style plain run: nine Purkinje cells with gap junctions, one system
        {"name": "purkinje 3x3 fp64", "kind": "cells", "type": "pkj", "n": 1, "nx": 3, "ny": 3, "prec": "fp64",
         "iv": 8, "sweep": False, "trial": False, "warm": 5},
        # separate Purkinje cells in mixed precision, more than fit the SMs one each
        {"name": "purkinje 200 mixed", "kind": "cells", "type": "pkj", "n": 200, "nx": 1, "ny": 1, "prec": "mixed",
         "iv": 8, "sweep": False, "trial": False, "warm": 10},
        # the mixed batch's olive network
        {"name": "olive 16x16 mixed", "kind": "cells", "type": "io", "n": 1, "nx": 16, "ny": 16, "prec": "mixed",
         "iv": 16, "sweep": False, "trial": True, "warm": 0},
        # the benchmark's mixed batch at half its populations: every role of the
        # persistent launch at once (the largest case)
        {"name": "mixed batch half", "kind": "batch", "gr": 2048, "go": 512, "pkj": 128, "io_side": 16,
         "prec": "mixed", "iv": 8, "warm": 10},
        # the synaptic network, scaled: one launch per interval
        {"name": "network mixed", "kind": "network", "gr": 512, "go": 64, "pkj": 48, "syn": 60000, "prec": "mixed",
         "iv": 4, "warm": 5},
        # a served burst of requests of all cell types, submitted to completion
        {"name": "serve burst", "kind": "serve", "n": 12, "iv": 24, "prec": "mixed"},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["cells"] * 6 + ["batch", "network", "serve"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        return {"kind": kind, "gr": _log(rng, 64, 2048), "go": _log(rng, 16, 512), "pkj": _log(rng, 4, 128),
                "io_side": rng.choice([4, 8, 16]), "prec": "mixed", "iv": rng.randint(1, 8), "warm": 10}
    if kind == "network":
        return {"kind": kind, "gr": _log(rng, 64, 512), "go": _log(rng, 8, 64), "pkj": _log(rng, 4, 48),
                "syn": _log(rng, 12000, 60000), "prec": prec, "iv": rng.randint(1, 4), "warm": 5}
    if kind == "serve":
        return {"kind": kind, "n": rng.randint(3, 12), "iv": rng.randint(5, 24), "prec": prec}
    t = rng.choice(["gr", "gr", "go", "go", "pkj", "io", "grfull"])
    c = {"kind": kind, "type": t, "n": 1, "nx": 1, "ny": 1, "prec": prec, "iv": rng.randint(1, 8), "sweep": False}
    if t == "gr":
        c.update(n=_log(rng, 1, 4096 if prec == "mixed" else 999), sweep=rng.random() < 0.5)
        c["iv"] = rng.randint(1, 4)
    elif t == "go":
        c.update(n=_log(rng, 1, 2048 if prec == "mixed" else 512), sweep=rng.random() < 0.5)
        c["iv"] = rng.randint(1, 8 if prec == "mixed" else 4)
        if rng.random() < 0.2:
            c.update(n=_log(rng, 1, 200), nx=2, ny=2)
    elif t == "pkj":
        if rng.random() < 0.5:
            c.update(nx=rng.randint(1, 3), ny=rng.randint(1, 3))
        else:
            c.update(n=_log(rng, 1, 200))
    elif t == "io":
        s = rng.randint(1, 16)
        c.update(nx=s, ny=s, n=_log(rng, 1, 16))
    else:
        c.update(n=_log(rng, 1, 32), iv=1)
    # refilling on the host costs a trial pass little up to this size
    c["trial"] = c["n"] * c["nx"] * c["ny"] * NC[t] <= 12000
    c["warm"] = 0 if c["trial"] else {"gr": 1, "go": 10, "pkj": 5}.get(t, 0)
    return c


@functools.lru_cache(maxsize=None)
def _rows(shape, k):
    if shape == "gr":
        return M.gr_reduced4()
    if shape == "grfull":
        return M.gr_synthetic(11 + k)
    if shape == "go":
        return M.go_synthetic(2000 + configs.GO_STABLE_VARIANTS[k % len(configs.GO_STABLE_VARIANTS)])
    if shape == "pkj":
        return M.pkj_synthetic(configs.PKJ_STABLE_SEEDS[k % len(configs.PKJ_STABLE_SEEDS)])
    return M.io_rows()


def _systems(case, seed):
    """The systems of a ``cells`` case: (rows, jitter, amplitudes, factors) each."""
    t = case["type"]
    ct = "gr" if t == "grfull" else t
    rng = np.random.default_rng(seed)
    amp = {"gr": 0.05e-3, "grfull": 0.01e-3, "go": 0.4e-3, "pkj": 0.4e-3, "io": 6.0}[t]
    cells = case["nx"] * case["ny"]
    out = []
    for i in range(case["n"]):
        rows = _rows(t, 0 if (case["sweep"] or t == "grfull") else i)
        jit = rng.uniform(-0.5, 0.5, cells)
        cur = rng.uniform(0.0, amp, cells)
        fac = rng.uniform(0.8, 1.2, NCOND[ct]) if case["sweep"] else None
        out.append((rows, jit, cur, fac))
    return out


def _stim_comp(case, rows):
    return 16 if case["type"] == "grfull" else min(STIM_COMP[case["type"]], rows.shape[0] - 1)


def _cell_type(case):
    return G.GR if case["type"] == "grfull" else TYPES[case["type"]]


class _Stepper:
    """An engine that a program advances window by window, from t = 0 each
    time where ``refill`` (Engine.reset_systems' arguments) is given."""

    def __init__(self, eng, runs, iv, warm=0, refill=None):
        self.eng, self.runs, self.iv, self.t, self.refill = eng, runs, iv, float(warm), refill
        if warm:
            eng.advance(0.0, int(warm / G.H_MAX), tolerate_retire=True)
        self.types = sorted({r[0] for r in runs})
        eng.record_soma(iv)
        self.soma = {t: np.empty((iv, eng.type_cells(t))) for t in self.types}

    def __call__(self):
        e = self.eng
        if self.refill is not None:
            e.reset_systems(**self.refill)
            self.t = 0.0
        e.rewind_soma()
        e.advance(self.t, self.iv, tolerate_retire=True)
        self.t += self.iv * G.H_MAX
        out = {}
        for k, (t, first, n, nc) in enumerate(self.runs):
            name = M.TYPE_NAMES[t]
            out[name] = {"v_new": e.read_run(first, n, G.F_VNEW, nc), "v": e.read_run(first, n, G.F_V, nc),
                         "ca": e.read_run(first, n, G.F_CA, nc),
                         "soma": e.read_soma_type(t, self.iv, self.soma[t]).copy()}
        return out


class _Server:
    def __init__(self, srv, reqs):
        self.srv, self.reqs = srv, reqs

    def __call__(self):
        s = self.srv
        ids = [s.submit(cid, n_sys, iv, jit, stim=stim, io_gap_g=gg) for cid, n_sys, iv, jit, stim, gg, _ in self.reqs]
        while any(s.state(r)[0] in (G.REQ_QUEUED, G.REQ_RESIDENT) for r in ids):
            s.advance()
        out = []
        for r, q in zip(ids, self.reqs):
            cells = np.bincount(s.spikes(r)[1], minlength=q[3].size)      # spikes of each cell
            out.append({"v": s.read(r, q[6]), "spikes": cells})
            s.destroy(r)
        return out


def prepare(case, seed):
    prec = G.FP64 if case["prec"] == "fp64" else G.MIXED
    if case["kind"] == "cells":
        eng = G.Engine(prec)
        ct, cells = _cell_type(case), case["nx"] * case["ny"]
        rng = np.random.default_rng(seed + 1)
        first = total = 0
        gaps, comps = [], []
        systems = _systems(case, seed)
        for i, (rows, jit, cur, fac) in enumerate(systems):
            gg = None
            if ct == G.IO and cells > 1:
                gg = configs.G_C_IO * rng.uniform(0.5, 1.5, 4 * cells)
                gaps.append(gg)
            comps += [_stim_comp(case, rows)] * cells
            gj = M.PKJ_GJ_PAIRS if ct == G.PKJ and cells > 1 else None
            sid = eng.add_system(ct, case["nx"], case["ny"], rows, jit, gap=cells > 1, gj_pairs=gj, io_gap_g=gg,
                                 stim=(_stim_comp(case, rows), cur, 0.0, 1e9), cond_scale_ch=fac)
            first = sid if i == 0 else first
            total += cells * rows.shape[0]
        eng.build()
        refill = None
        if case["trial"]:
            n = len(comps)
            refill = {"first": first, "n": case["n"], "jitter": np.concatenate([x[1] for x in systems]),
                      "stim": (np.array(comps, np.int32), np.concatenate([x[2] for x in systems]), np.zeros(n),
                               np.full(n, 1e9)),
                      "io_gap_g": np.concatenate(gaps) if gaps else None,
                      "cond_scale_ch": np.concatenate([x[3] for x in systems]) if case["sweep"] else None}
        return _Stepper(eng, [(ct, first, case["n"], total)], case["iv"], case["warm"], refill)
    if case["kind"] == "batch":
        eng = G.Engine(prec)
        specs = configs.mixed_batch(seed=seed, n_gr=case["gr"], n_go=case["go"], n_pkj=case["pkj"],
                                    io_side=case["io_side"], go_variants=(0,), pkj_seeds=(7,))
        for i, s in enumerate(specs):    # tree shapes by the shared tables, not by the seed
            if s.cell_type in (G.GO, G.PKJ):
                s.rows = _rows(M.TYPE_NAMES[s.cell_type], i)
        return _Stepper(eng, _add_runs(eng, specs), case["iv"], case["warm"])
    if case["kind"] == "network":
        eng = G.Engine(prec)
        specs, groups = configs.network_batch(seed=seed, n_gr=case["gr"], n_go=case["go"], n_pkj=case["pkj"],
                                              n_syn=case["syn"], distinct_trees=False)
        return _Stepper(eng, _add_runs(eng, specs, groups), case["iv"], case["warm"])
    classes, reqs = _serve_requests(case, seed)
    srv = G.Server(prec)
    for t, nx, ny, rows, slots, gap in classes:
        srv.add_class(t, nx, ny, rows, slots=slots, gap=gap)
    srv.start()
    return _Server(srv, reqs)


def _add_runs(eng, specs, groups=None):
    ids = configs.add_network(eng, specs, groups) if groups is not None else configs.add_to(eng, specs)
    eng.build()
    runs = []
    for t in (G.GR, G.GO, G.PKJ, G.IO):
        mine = [k for k, s in enumerate(specs) if s.cell_type == t]
        if mine:
            runs.append((t, int(ids[mine[0]]), len(mine), sum(specs[k].nc for k in mine)))
    return runs


def _serve_requests(case, seed):
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(case["n"] * 1000 + case["iv"])
    classes = [(G.GR, 1, 1, _rows("gr", 0), 1024, False), (G.GO, 1, 1, _rows("go", 0), 128, False),
               (G.PKJ, 1, 1, _rows("pkj", 0), 24, False), (G.IO, 4, 4, _rows("io", 0), 16, True)]
    reqs = []
    for i in range(case["n"]):
        cid = i % 4
        t, nx, ny, rows, slots, gap = classes[cid]
        n_sys = int(sizes.integers(slots // 16, slots // 4 + 1))
        cells = n_sys * nx * ny
        iv = max(1, int(case["iv"] * sizes.uniform(0.5, 1.0)))
        comp = min(STIM_COMP[M.TYPE_NAMES[t]], rows.shape[0] - 1)
        stim = (np.full(cells, comp, np.int32), rng.uniform(0, configs.AMP_MAX[t], cells), np.zeros(cells),
                np.full(cells, 1e9))
        gg = configs.G_C_IO * rng.uniform(0.5, 1.5, 4 * cells) if gap else None
        reqs.append((cid, n_sys, iv, rng.uniform(-0.5, 0.5, cells), stim, gg, cells * rows.shape[0]))
    return classes, reqs


def run(state):
    return state()


# -------------------------------------------------------------------- work
# compartment-updates (right-hand-side evaluations of one compartment) per
# compartment and simulated ms that the method's own step sequence takes, the
# state bytes of a compartment, and the floating-point operations of one
# update with its share of the ion updates
UPDATES_PER_MS = {"gr": 12000.0, "grfull": 40000.0, "go": 1600.0, "pkj": 1200.0, "io": 5000.0}
STATE = {"gr": 20 + 10, "grfull": 20 + 10, "go": 24 + 13, "pkj": 18 + 11, "io": 10 + 8}
FLOPS_PER_UPDATE = 20.0


def _work_cells(t, nc, iv, prec):
    real = 8 if prec == "fp64" else 4
    b = nc * (2 * 14 * 8 + 2 * STATE[t] * real)
    return b, nc * UPDATES_PER_MS[t] * iv * G.H_MAX * FLOPS_PER_UPDATE


NC = {"gr": 4, "grfull": 578, "go": 131, "pkj": 1600, "io": 3}


def work(case):
    if case["kind"] == "cells":
        parts = [(case["type"], case["n"] * case["nx"] * case["ny"], case["iv"])]
    elif case["kind"] == "serve":
        parts = []
        classes, reqs = _serve_requests(case, 0)
        for q in reqs:
            t = M.TYPE_NAMES[classes[q[0]][0]]
            parts.append((t, q[6] // NC[t], q[2]))
    else:
        parts = [(t, case[t], case["iv"]) for t in ("gr", "go", "pkj")]
        if case["kind"] == "batch":
            parts.append(("io", case["io_side"] ** 2, case["iv"]))
    b = f = 0.0
    for t, cells, iv in parts:
        x, y = _work_cells(t, cells * NC[t], iv, case["prec"])
        b, f = b + x, f + y
    if case["kind"] == "network":
        b += case["syn"] * case["iv"] * 8 * 6
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- exact
# The method in numpy, 64 bits: every system of a case side by side, (S, N)
# arrays, each with its own controller; a system waits (masked) while others
# take more stages or iterations.
H_MAX, UROUND = 0.125, 2.22e-16
TOL = {"gr": 1e-9, "go": 1e-6, "pkj": 1e-6, "io": 1e-6}
HMIN = {"gr": 2.0 ** -12, "go": 2.0 ** -10, "pkj": 2.0 ** -10, "io": 2.0 ** -10}
EXACT_LIMIT = {"gr": 20000, "grfull": 8 * 578, "go": 300000, "pkj": 120000, "io": 20000}   # compartments x intervals


def _trap(dt, inf, tau, x):
    return (2.0 * dt * inf + (2.0 * tau - dt) * x) / (2.0 * tau + dt)


def _xr(c, x, k):
    return c * x / (1.0 - np.exp(-x / k))


class _Gr:
    """Granule cell: gates, the 12-state Na channel (Crank-Nicolson) and currents."""
    v0, dv = -80.0, 2.0

    def __init__(self, rows):
        d1, d2, d3, d4 = rows[:, 2], rows[:, 3], rows[:, 4], rows[:, 5]
        rad, ln, ra = 0.5e-4 * d1, 1e-4 * d2, 1e-3 * d3
        area = 2 * np.pi * rad * ln
        self.ctype = rows[:, 6].astype(int)
        self.cm = d4 * area
        self.g = rows[:, 7:].T * area
        self.parent = rows[:, 1].astype(int)
        self.r = ra * ln / (np.pi * rad ** 2)

    def couplings(self):
        i = np.nonzero(self.parent >= 0)[0]
        p = self.parent[i]
        g = 2.0 / (self.r[i] + self.r[p])
        return i, p, g, g

    def init(self, v, ctype, cond):
        e = np.exp
        self.ca = np.full_like(v, 1e-4)
        a, b = self._nkv(v)
        x = {"n": a / (a + b), "a": 1 / (1 + e(-(v + 38) / 17)), "b": 1 / (1 + e((v + 78.8) / 8.4))}
        a, b = self._kir(v)
        x["ir"] = a / (a + b)
        x["s"] = 1 / (1 + e(-(v + 35) / 6))
        a, b = self._kca(v, self.ca)
        x["c"] = a / (a + b)
        a, b = 0.0856 * e((v + 29.6) / 15.873), 0.1437 * e(-(v + 18.66) / 25.641)
        x["ch"] = a / (a + b)
        a, b = 0.0023 * e(-(v + 48) / 18.183), 0.0025 * e((v + 48) / 83.33)
        x["ci"] = a / (a + b)
        x["na"] = np.zeros(v.shape + (12,))
        x["na"][..., 0] = 1.0
        self.x, self.ct = x, ctype

    @staticmethod
    def _nkv(v):
        y = v + 25.0
        return -0.017 * y / (np.exp(-y / 10) - 1), 0.2223 * np.exp(-(v + 35) / 80)

    @staticmethod
    def _kir(v):
        return 0.2302 * np.exp(-(v + 83.94) / 24.3902), 0.2943 * np.exp((v + 83.94) / 35.714)

    @staticmethod
    def _kca(v, c):
        q = np.exp(-v / 11.765)
        return 1.4433 / (1 + 1.5e-3 * q / c), 0.8660 / (1 + c / (1.5e-4 * q))

    def _q(self, v, ct):
        """Rate generator of the Na channel, states c1..c5, i1..i6, o: dx/dt = Q x."""
        late = ct >= 7
        n1, n2, n3, n4 = 5.422, 3.279, 1.83, 0.738
        vs = np.where(late, -25.0, -22.0)
        con, coff = np.where(late, 0.09353, 0.003464), np.where(late, 0.04676, 0.4157)
        oon, ooff = np.where(late, 2.5981, 1.8186), np.where(late, 0.000173, 0.006928)
        a, b = (oon / con) ** 0.25, (ooff / coff) ** 0.25
        al, be = 8.85 * np.exp((v - vs) / 10), 0.0318 * np.exp(-(v - vs) / 10)
        q = np.zeros(v.shape + (12, 12))

        def edge(i, j, r):      # from state i to state j
            q[..., j, i] += r
            q[..., i, i] -= r
        for k, n in enumerate((n1, n2, n3, n4)):
            edge(k, k + 1, n * al)
            edge(k + 1, k, (n4, n3, n2, n1)[k] * be)
            edge(5 + k, 6 + k, n * al * a)
            edge(6 + k, 5 + k, (n4, n3, n2, n1)[k] * be * b)
        for k in range(5):
            edge(k, 5 + k, con * a ** k)
            edge(5 + k, k, coff * b ** k)
        edge(4, 11, 259.8)
        edge(11, 4, 69.3)
        edge(9, 10, 259.8)
        edge(10, 9, 69.3)
        edge(10, 11, ooff)
        edge(11, 10, oon)
        return q

    def ion(self, s, v_old, v_new, dt):
        x, e = self.x, np.exp
        dt = dt[:, None]
        v = 0.5 * (v_old + v_new)
        ct = self.ct[s]
        w = ct >= 5
        if w.any():
            d = np.broadcast_to(dt, v.shape)[w][:, None, None]
            q0, q1 = self._q(v_old[w], ct[w]), self._q(v_new[w], ct[w])
            na = x["na"][s]
            eye = np.eye(12)
            rhs = (eye * (2 / d) + q0) @ na[w][..., None]
            na[w] = np.linalg.solve(eye * (2 / d) - q1, rhs)[..., 0]
            x["na"][s] = na

        def ab(key, a, b):
            x[key][s] = _trap(dt, a / (a + b), 1 / (a + b), x[key][s])
        ab("n", *self._nkv(v))
        a, b = 0.771 / (1 + e(-(v + 9.17203) / 23.32708)), 0.1567 / e((v + 18.27914) / 19.47175)
        x["a"][s] = _trap(dt, 1 / (1 + e(-(v + 38) / 17)), 1 / (a + b), x["a"][s])
        a, b = 0.0348 / (1 + e((v + 111.33208) / 12.8433)), 0.0327 / (1 + e(-(v + 49.9537) / 8.90123))
        x["b"][s] = _trap(dt, 1 / (1 + e((v + 78.8) / 8.4)), 1 / (a + b), x["b"][s])
        ab("ir", *self._kir(v))
        a, b = 0.0046 * e((v + 30) / 40), 0.0046 * e(-(v + 30) / 20)
        x["s"][s] = _trap(dt, 1 / (1 + e(-(v + 35) / 6)), 1 / (a + b), x["s"][s])
        ab("c", *self._kca(v, self.ca[s]))

    def current(self, s, v, g, iext):
        x = {k: (u[s] if k != "na" else u[s][..., 11]) for k, u in self.x.items()}
        ek = v + 84.69
        return (g[0] * (v + 16.5) + g[1] * (v + 65) + g[2] * (v + 74.5) - iext + g[3] * (v - 87.39) * x["na"]
                + g[9] * (v - 129.33) * x["ch"] ** 2 * x["ci"] + ek * (g[4] * x["n"] ** 4 + g[8] * x["ir"]
                + g[5] * x["a"] ** 3 * x["b"] + g[6] * x["c"] + g[7] * x["s"]))


class _Go:
    """Golgi cell, with the 6-state KAHP channel."""
    v0, dv = -60.0, 2.0
    F, D, CA0 = 9.6485e4, 0.2e-4, 5e-5

    def __init__(self, rows):
        _Gr.__init__(self, rows)
        self.area = 2 * np.pi * 0.5e-4 * rows[:, 2] * 1e-4 * rows[:, 3]

    couplings = _Gr.couplings

    def _rates(self, v, c):
        e = np.exp
        i = lambda z: 1 / (1 + e(z))  # noqa: E731

        def ab(a, b):
            return a / (a + b), 1 / (a + b)
        x = np.minimum((v + 44) / 0.11, 200.0)
        r1, s1, s2 = 0.0021 * v + 0.97, i((v + 72.5) * 0.11), i((v + 81.9) * 0.16)
        r2 = np.where(v >= -64.70, 0.0, np.where(v <= -108.70, 1.0, -0.0227 * v - 1.47))
        z = e(-v / 11.7)
        return {
            "m": ab(_xr(0.417, v + 25, 10.0), 16.68 * e(-0.055 * (v + 50))),
            "h": ab(0.292 * e(-0.3 * (v + 50)), 4.17 * i(-(v + 17) / 5)),
            "r": ab((1.11 + _xr(68.5, v - 4.48, 6.8)) * 1e-4, (66.0 + 21.7 * (v + 44) / (e(x) - 1)) * 1e-3),
            "s": ab(0.443 * e(-(v + 80) / 62.5), 0.014 * e((v + 83.3) / 16.1)),
            "p": (i(-(v + 43) / 5), 5.0 / (_xr(0.421, v + 40, 5.0) + _xr(-0.287, v + 40, -5.0))),
            "n": ab(_xr(0.062, v + 26, 10.0), 0.78 * e(-(v + 36) / 80)),
            "a": (i(-(v + 38) / 17), 1 / (0.62 * i(-(v + 9.17) / 23.32) + 0.126 / e((v + 18.28) / 19.47))),
            "b": (i((v + 78.8) / 8.4), 1 / (0.028 * i((v + 111) / 12.84) + 0.026 * i(-(v + 49.95) / 8.9))),
            "sl": (i(-(v + 35) / 6), 1 / (0.0037 * e((v + 30) / 40) + 0.0037 * e(-(v + 30) / 20))),
            "c": ab(3.2 / (1 + 0.0015 * z / c), 0.46 / (1 + c / (1.5e-4 * z))),
            "ch": ab(0.0687 * e(0.063 * (v + 29)), 0.115 * e(-0.039 * (v + 18.66))),
            "ci": ab(1.8e-3 * e(-(v + 48) / 18), 1.8e-3 * e((v + 48) / 83)),
            "cl": (i(-(v + 52) / 7.4), (3 + 1 / (e((v + 27) / 10) + e(-(v + 102) / 15))) / 0.85),
            "cm": (i((v + 80) / 5), (85 + 1 / (e((v + 48) / 4) + e(-(v + 407) / 50))) / 0.9),
            "hf1": (r1 * s1, e((0.0137 * v + 3.37) * 2.3)), "hf2": (r2 * s2, e((0.027 * v + 5.6) * 2.3)),
            "hs1": ((1 - r1) * s1, e((0.0145 * v + 4.06) * 2.3)), "hs2": ((1 - r2) * s2, e((0.015 * v + 5.3) * 2.3)),
        }

    def init(self, v, ctype, cond):
        self.ca, self.ca2, self.ca_old = (np.full_like(v, self.CA0) for _ in range(3))
        self.rev = np.full_like(v, 120.0)
        self.x = {k: inf for k, (inf, _) in self._rates(v, self.ca).items()}
        self.k = np.zeros(v.shape + (6,))
        self.k[..., 0] = 1.0
        self.cond = cond

    def ion(self, s, v_old, v_new, dt):
        x, dt = self.x, dt[:, None]
        g = self.cond[:, s]
        v = 0.5 * (v_old + v_new)

        def ca_step(c, cur):
            f = lambda z: dt * (-cur / (2 * self.F * self.D) - 1.3 * (z - self.CA0))  # noqa: E731
            k1 = f(c)
            k2 = f(c + k1 / 2)
            k3 = f(c + k2 / 2)
            return c + (k1 + 2 * k2 + 2 * k3 + f(c + k3)) / 6
        old = self.ca[s]
        i1 = 1e-3 * g[8] / self.area * x["ch"][s] ** 2 * x["ci"][s] * (v_old - 120.0)
        i2 = 1e-3 * g[9] / self.area * x["cl"][s] ** 2 * x["cm"][s] * (v_old - self.rev[s])
        self.ca[s] = ca_step(old, i1)
        self.ca2[s] = ca_step(self.ca2[s], i2)
        self.rev[s] = 1e3 * 8.313424 * (23.0 + 273.15) / (2 * self.F) * np.log(2.0 / self.ca2[s])
        for key, (inf, tau) in self._rates(v, 0.5 * (old + self.ca[s])).items():
            x[key][s] = _trap(dt, inf, tau, x[key][s])

        def q(c):
            m = np.zeros(c.shape + (6, 6))
            d = (200 * c / 3, 160 * c / 3, 80 * c / 3)
            back, opn = (80e-3, 80e-3, 200e-3), ((2, 4, 160e-3, 1.0), (3, 5, 1.2, 100e-3))
            edges = [(k, k + 1, d[k], back[k]) for k in range(3)] + list(opn)
            for i, j, f, r in edges:
                m[..., j, i] += f
                m[..., i, i] -= f
                m[..., i, j] += r
                m[..., j, j] -= r
            return m
        w = 2 / dt[..., None, None] * np.eye(6)
        self.k[s] = np.linalg.solve(w - q(self.ca[s]), (w + q(self.ca_old[s])) @ self.k[s][..., None])[..., 0]
        self.ca_old[s] = self.ca[s]

    def current(self, s, v, g, iext):
        x = {k: u[s] for k, u in self.x.items()}
        ek, ena, eh = v + 84.69, v - 87.39, v + 20.0
        return (-iext + g[0] * (v + 55) + ena * (g[1] * x["m"] ** 3 * x["h"] + g[2] * x["r"] * x["s"] + g[3] * x["p"])
                + g[8] * (v - 120) * x["ch"] ** 2 * x["ci"] + g[9] * (v - self.rev[s]) * x["cl"] ** 2 * x["cm"]
                + ek * (g[12] * self.k[s][..., 4:].sum(-1) + g[4] * x["n"] ** 4 + g[5] * x["a"] ** 3 * x["b"]
                        + g[6] * x["c"] + g[7] * x["sl"])
                + eh * (g[10] * (x["hf1"] + x["hs1"]) + g[11] * (x["hf2"] + x["hs2"])))


class _Pkj:
    """Purkinje cell."""
    v0, dv = -68.0, 2.0
    SHELL, CA0, OUT, F = 0.2e-4, 4.0e-5, 2.4, 9.6485e4
    DENS = np.array([[7500.0, 1.0, 0.0, 0.5, 0.3, 600.0, 0.040, 15.0, 0.0, 0.0],
                     [0.0, 0.0, 4.5, 0.5, 0.0, 60.0, 0.01, 2.0, 80.0, 0.39],
                     [0.0, 0.0, 4.5, 0.5, 0.0, 0.0, 0.013, 0.0, 80.0, 0.39],
                     [0.0, 0.0, 4.5, 0.5, 0.0, 0.0, 0.013, 0.0, 80.0, 0.39]])

    def __init__(self, rows):
        d = rows[:, 5] * 1e-4
        self.ctype = t = rows[:, 6].astype(int)
        rad = 0.5 * d
        ln = np.where(t == 0, d, 1e-4 * np.sqrt((rows[:, 2:5] ** 2).sum(1)))
        area = np.where(t == 0, 4 * np.pi * rad ** 2, 2 * np.pi * rad * ln)
        wide = np.where(t == 3, area + ln * 1.33e-8 * 13.0e4, area)
        D = self.SHELL
        self.shell = np.where(t == 0, D - 2 * D ** 2 / d + 4 * D ** 3 / (3 * d ** 2), D - D ** 2 / d) * area
        self.cm = 1.64 * wide
        self.g = np.concatenate([(np.where(t == 0, area / 10.0, wide / 30.0))[None], self.DENS[t].T * area])
        self.parent = rows[:, 1].astype(int)
        self.r = 0.25 * ln / (np.pi * rad ** 2)

    couplings = _Gr.couplings

    @staticmethod
    def _rates(v, cq):
        e = np.exp
        l = lambda A, B, C, D: A / (B + e((v + C) / D))  # noqa: E731,E741

        def ab(a, b):
            return a / (a + b), 1 / (a + b)

        def kdr(y):
            return -0.0235 * y / (e(-y / 12) - 1)
        k1 = 1 / (1 + e((v + 82) / 7))
        a1, b1, a2, b2 = kdr(v + 12), 5 * e(-(v + 147) / 30), kdr(v - 8), 5 * e(-(v + 127) / 30)
        kc, k2 = l(0.110, 0.0, -35.0, 14.9), l(0.075, 0.0, 25.0, 6.0)
        return {
            "mNaF": ab(l(35.0, 0.0, 5.0, -10.0), l(7.0, 0.0, 65.0, 20.0)),
            "hNaF": ab(l(0.225, 1.0, 80.0, 10.0), l(7.5, 0.0, -3.0, -18.0)),
            "mNaP": ab(l(200.0, 1.0, -18.0, -16.0), l(25.0, 1.0, 58.0, 8.0)),
            "mCaP": ab(l(8.5, 1.0, -8.0, -12.5), l(35.0, 1.0, 74.0, 14.5)),
            "hCaP": ab(l(0.0015, 1.0, 29.0, 8.0), l(0.0055, 1.0, 23.0, -8.0)),
            "mCaT": ab(l(2.60, 1.0, 21.0, -8.0), l(0.180, 1.0, 40.0, 4.0)),
            "hCaT": ab(l(0.0025, 1.0, 40.0, 8.0), l(0.190, 1.0, 50.0, -10.0)),
            "Kh1": (0.8 * k1, 7.6), "Kh2": (0.2 * k1, 36.8),
            "mKdr": (a2 / (a2 + b2), 1 / (a1 + b1)),
            "hKdr": (1 / (1 + e((v + 25) / 4)), np.where(v < -25.0, 1200.0, 10.0)),
            "KM": (1 / (1 + e(-(v + 35) / 10)), 200 / (3.3 * e((v + 35) / 20) + e(-(v + 35) / 20))),
            "mKA": ab(l(1.40, 1.0, 27.0, -12.0), l(0.490, 1.0, 30.0, 4.0)),
            "hKA": ab(l(0.0175, 1.0, 50.0, 8.0), l(1.30, 1.0, 13.0, -10.0)),
            "mKC": ab(7.5, kc), "zKC": (1 / (1 + 4.0 / cq), 10.0),
            "mK2": ab(25.0, k2), "zK2": (1 / (1 + 0.20 / cq), 10.0),
        }

    def init(self, v, ctype, cond):
        self.ca = np.full_like(v, self.CA0)
        self.rev = np.full_like(v, 135.0)
        self.x = {k: inf + np.zeros_like(v) for k, (inf, _) in self._rates(v, self.ca).items()}
        self.cond = cond
        self.fixed = np.arange(v.shape[1]) % 1599 == 0

    def ion(self, s, v_old, v_new, dt):
        x, dt = self.x, dt[:, None]
        g, old = self.cond[:, s], self.ca[s]
        v = 0.5 * (v_old + v_new)
        cur = 1e-3 * (v_old - self.rev[s]) * (g[3] * x["mCaP"][s] * x["hCaP"][s] + g[4] * x["mCaT"][s] * x["hCaT"][s])
        cur = np.where(cur > 0, 0.0, -cur / (2 * self.F * self.shell))
        f = lambda z: dt * (cur - 10.0 * (z - self.CA0))  # noqa: E731
        k1 = f(old)
        k2 = f(old + k1 / 2)
        k3 = f(old + k2 / 2)
        new = old + (k1 + 2 * k2 + 2 * k3 + f(old + k3)) / 6
        self.ca[s] = new
        c = 0.5 * (old + new)
        self.rev[s] = np.where(self.fixed, 12.5 * np.log(self.OUT / self.CA0), 13.361624877 * np.log(self.OUT / c))
        cq = np.floor((c * 1000 - 0.04) / 0.099986667) * 0.099986667 + 0.04
        for key, (inf, tau) in self._rates(v, cq).items():
            x[key][s] = _trap(dt, inf, tau, x[key][s])

    def current(self, s, v, g, iext):
        x = {k: u[s] for k, u in self.x.items()}
        ek, ena, eca, eh = v + 85.0, v - 45.0, v - self.rev[s], v + 30.0
        return (-iext + g[0] * (v + 80) + ena * (g[1] * x["mNaF"] ** 3 * x["hNaF"] + g[2] * x["mNaP"] ** 3)
                + eca * (g[3] * x["mCaP"] * x["hCaP"] + g[4] * x["mCaT"] * x["hCaT"])
                + eh * g[5] * (x["Kh1"] + x["Kh2"])
                + ek * (g[6] * x["mKdr"] ** 2 * x["hKdr"] + g[7] * x["KM"] + g[8] * x["mKA"] ** 4 * x["hKA"]
                        + g[9] * x["mKC"] * x["zKC"] ** 2 + g[10] * x["mK2"] * x["zK2"] ** 2))


class _Io:
    """Inferior olive cell (three compartments)."""
    v0, dv = -60.0, 10.0
    DENS = np.array([[0.016, 0.0, 0.0, 0.0, 0.0, 4.5, 35.0, 0.15], [0.016, 0.83, 120.0, 9.0, 5.0, 0.0, 0.0, 0.0],
                     [0.016, 0.0, 240.0, 0.0, 20.0, 0.0, 0.0, 0.0]])

    def __init__(self, rows):
        self.ctype = rows[:, 5].astype(int)
        self.cm = rows[:, 4].copy()
        self.g = self.DENS[self.ctype].T
        self.parent = rows[:, 1].astype(int)

    def couplings(self):
        i = np.nonzero(self.parent >= 0)[0]
        p = self.parent[i]
        t = self.ctype[i]
        up = np.where((t == 0) & (p == 1), 0.13 / 0.8, np.where((t == 1) & (p == 2), 0.13 / 0.869, 0.0))
        dn = np.where((t == 0) & (p == 1), 0.13 / 0.2, np.where((t == 1) & (p == 2), 0.13 / 0.131, 0.0))
        return i, p, up, dn

    def init(self, v, ctype, cond):
        self.ct, self.cond = ctype, cond
        x = {k: inf + np.zeros_like(v) for k, (inf, _) in self._rates(v, np.ones_like(v), ctype).items()}
        self.ca = -cond[5] * x["r"] ** 2 * (v - 120.0) * 3.0 / 0.075
        a = np.minimum(0.00002 * self.ca, 0.01)
        x["s"] = a / (a + 0.015)
        self.x = x

    @staticmethod
    def _rates(v, c, ct):
        e = np.exp
        ar, br = 1.7 / (1 + e(-(v - 5) / 13.9)), 0.02 * (v + 8.5) / (e((v + 8.5) / 5) - 1)
        ax, bx = 0.13 * (v + 25) / (1 - e(-(v + 25) / 10)), 1.69 * e(-0.0125 * (v + 35))
        a = np.minimum(0.00002 * c, 0.01)
        nt = 47 * e((v + 50) / 900) + 5
        hi = np.where(ct == 1, 1 / (1 + e((v + 70) / 5.8)), np.where(ct == 2, 1 / (1 + e((v + 60) / 5.8)), 1.0))
        ht = np.where(ct == 1, 3 * e((-v - 40) / 33), np.where(ct == 2, 1.5 * e((-v - 40) / 33), 1.0))
        return {"k": (1 / (1 + e((-v - 61) / 4.2)), 1.0),
                "l": (1 / (1 + e((v + 85.5) / 8.5)), 20 * e((v + 160) / 30) / (1 + e((v + 84) / 7.3)) + 35),
                "n": (1 / (1 + e((-v - 3) / 10)), nt), "p": (1 / (1 + e((v + 51) / 12)), nt),
                "x": (ax / (ax + bx), 1 / (ax + bx)), "r": (ar / (ar + br), 5 / (ar + br)),
                "q": (1 / (1 + e((v + 80) / 4)), 1 / (e(-0.086 * v - 14.6) + e(0.07 * v - 1.87))),
                "s": (a / (a + 0.015), 1 / (a + 0.015)), "m": (1 / (1 + e((-v - 30) / 5.5)), None), "h": (hi, ht)}

    def ion(self, s, v_old, v_new, dt):
        x, dt = self.x, dt[:, None]
        cur = self.cond[5][s] * x["r"][s] ** 2 * (v_old - 120.0)
        old = self.ca[s]
        f = lambda z: dt * (-cur * 3.0 - 0.075 * z)  # noqa: E731
        k1 = f(old)
        k2 = f(old + k1 / 2)
        k3 = f(old + k2 / 2)
        self.ca[s] = old + (k1 + 2 * k2 + 2 * k3 + f(old + k3)) / 6
        for key, (inf, tau) in self._rates(0.5 * (v_old + v_new), 0.5 * (old + self.ca[s]), self.ct[s]).items():
            x[key][s] = inf if tau is None else _trap(dt, inf, tau, x[key][s])

    def current(self, s, v, g, iext):
        x = {k: u[s] for k, u in self.x.items()}
        ek = v + 75.0
        return (-iext + g[0] * (v - 10) + g[1] * (v - 120) * x["k"] ** 3 * x["l"] + g[2] * (v - 55) * x["m"] ** 3 * x["h"]
                + ek * (g[3] * x["n"] * x["p"] + g[4] * x["x"] ** 4 + g[6] * x["s"]) + g[5] * (v - 120) * x["r"] ** 2
                + g[7] * (v + 43) * x["q"])


MODELS = {"gr": _Gr, "grfull": _Gr, "go": _Go, "pkj": _Pkj, "io": _Io}


@functools.lru_cache(maxsize=None)
def _stages(m):
    """The second-order RKC coefficients of m stages (Sommeijer, Shampine & Verwer 1998), eps = 2/13."""
    w0 = 1 + 2 / (13.0 * m * m)
    t, d, d2 = [1.0, w0], [0.0, 1.0], [0.0, 0.0]
    for _ in range(2, m + 1):
        d2.append(2 * w0 * d2[-1] - d2[-2] + 4 * d[-1])
        d.append(2 * w0 * d[-1] - d[-2] + 2 * t[-1])
        t.append(2 * w0 * t[-1] - t[-2])
    w1 = d[m] / d2[m]
    b = [0.0, 0.0] + [d2[j] / d[j] ** 2 for j in range(2, m + 1)]
    b[0] = b[1] = 1 / (4 * w0 * w0)      # b_0 = b_1, as the reference takes them
    out = [w1 * b[1]]
    for j in range(2, m + 1):
        mu, nu = 2 * w0 * b[j] / b[j - 1], -b[j] / b[j - 2]
        out.append((mu, nu, 1 - mu - nu, mu * w1 / w0, 1 - t[j - 1] * b[j - 1]))
    return out


class _Exact:
    """All systems of a ``cells`` case, integrated by the method in numpy."""

    def __init__(self, case, seed):
        t = case["type"]
        self.t = "gr" if t == "grfull" else t
        self.cells, self.nx, self.ny = case["nx"] * case["ny"], case["nx"], case["ny"]
        syss = _systems(case, seed)
        rng = np.random.default_rng(seed + 1)
        model = {id(r): MODELS[t](r) for r, *_ in syss}
        ms = [model[id(r)] for r, *_ in syss]
        nc1, S, C = syss[0][0].shape[0], len(syss), self.cells
        N = nc1 * C
        self.S, self.N, self.nc1 = S, N, nc1
        tile = lambda key: np.array([np.tile(getattr(m, key), C) for m in ms])  # noqa: E731
        self.invcm = 1 / tile("cm")
        ctype = tile("ctype")
        fac = [np.ones(len(m.g)) if f is None else f for m, (_, _, _, f) in zip(ms, syss)]
        self.cond = np.array([np.tile(m.g * np.resize(f, len(m.g))[:, None], C) for m, f in zip(ms, fac)]).transpose(1, 0, 2)
        self.P = ms[0]
        self.per = {k: tile(k) for k in ("area", "shell") if hasattr(ms[0], k)}
        self.idx, self.g = self._operator(ms)
        v = np.array([np.repeat(self.P.v0 + self.P.dv * jit, nc1) for _, jit, _, _ in syss])
        self.iext = np.zeros((S, N))
        comp = _stim_comp(case, syss[0][0])
        self.amp = np.zeros((S, N))
        for k, (_, _, cur, _) in enumerate(syss):
            self.amp[k, comp::nc1][:C] = cur
        self.gap = None
        if self.t == "io" and C > 1:
            self.gap = [configs.G_C_IO * rng.uniform(0.5, 1.5, 4 * C) for _ in range(S)]
            self.gap = np.array(self.gap).reshape(S, C, 4)
        self.P.init(v, ctype, self.cond)
        self.v = v.copy()
        self.y = v.copy()
        self.tol, self.hmin = TOL[self.t], HMIN[self.t]
        self.integ = 2.0 ** np.log10(self.tol)

    def _operator(self, ms):
        nc1, C, rows = self.nc1, self.cells, []
        gj = []
        if C > 1 and self.t == "pkj":
            for y in range(self.ny):
                for x in range(self.nx - 1):
                    for a, b in M.PKJ_GJ_PAIRS:
                        gj.append((int(a) + (x + y * self.nx) * nc1, int(b) + (x + 1 + y * self.nx) * nc1))
        if C > 1 and self.t == "go":
            for y in range(self.ny):
                for x in range(self.nx):
                    i = (x + y * self.nx) * nc1
                    if x + 1 < self.nx:
                        gj.append((i, i + nc1))
                    if y + 1 < self.ny:
                        gj.append((i, i + self.nx * nc1))
        done = {}
        for m in ms:
            if id(m) not in done:
                adj = [[] for _ in range(self.N)]
                i, p, gi, gp = m.couplings()
                for c in range(C):
                    for a, b, u, w in zip(i + c * nc1, p + c * nc1, gi, gp):
                        adj[a].append((b, u))
                        adj[b].append((a, w))
                for a, b in gj:
                    adj[a].append((b, 2.5e-6))
                    adj[b].append((a, 2.5e-6))
                done[id(m)] = adj
            rows.append(done[id(m)])
        deg = max(len(r) for adj in rows for r in adj)
        idx = np.zeros((self.S, self.N, deg), np.int64)
        g = np.zeros((self.S, self.N, deg))
        made = {}
        for k, adj in enumerate(rows):
            if id(adj) not in made:
                one, two = np.zeros((self.N, deg), np.int64), np.zeros((self.N, deg))
                one[:] = np.arange(self.N)[:, None]
                for i, r in enumerate(adj):
                    for q, (j, w) in enumerate(sorted(r)):
                        one[i, q], two[i, q] = j, w
                made[id(adj)] = (one, two)
            idx[k] = made[id(adj)][0] + k * self.N
            g[k] = made[id(adj)][1]
        return idx, g

    def f(self, s, y):
        full = np.zeros((self.S, self.N))
        full[s] = y
        flat = full.ravel()
        d = -self.b[s]
        for q in range(self.idx.shape[2]):
            d = d + self.g[s, :, q] * (flat[self.idx[s, :, q]] - y)
        return d * self.invcm[s]

    def currents(self, s, update, dt=None):
        y = self.y[s]
        if update:
            P = self.P
            keep = {}
            for k, a in self.per.items():      # per-compartment statics of these systems
                keep[k] = getattr(P, k)
                setattr(P, k, a[s])
            P.ion(s, self.v[s], y, dt)
            for k, a in keep.items():
                setattr(P, k, a)
            self.v[s] = y
        b = self.P.current(s, y, self.cond[:, s], self.iext[s])
        if update and self.gap is not None:
            n, side = self.cells, self.nx
            post = np.arange(n) * self.nc1
            v = self.v[s][:, post]
            r, c = np.divmod(np.arange(n), side)
            for k, (dr, dc) in enumerate(((0, -1), (-1, 0), (0, 1), (1, 0))):
                ok = (r + dr >= 0) & (r + dr < side) & (c + dc >= 0) & (c + dc < side)
                pre = np.where(ok, np.arange(n) + dr * side + dc, np.arange(n))
                d = v - v[:, pre]
                b[:, post] += self.gap[s][:, :, k] * (0.8 * np.exp(-0.01 * d * d) + 0.2) * d
        self.b[s] = b

    def rho(self, s):
        """The nonlinear power method from the last eigenvector estimate."""
        yn, fn = self.yn[s], self.fn[s]
        nrm = lambda a: np.sqrt((a * a).sum(1))  # noqa: E731
        ynrm, vnrm = nrm(yn), nrm(self.ede[s])
        dyn = ynrm * np.sqrt(UROUND)
        v1 = yn + (dyn / vnrm)[:, None] * self.ede[s]
        sigma, live = np.zeros(len(s)), np.ones(len(s), bool)
        for it in range(1000):
            w = np.nonzero(live)[0]
            if not len(w):
                break
            v2 = self.f(s[w], v1[w])
            dfn = nrm(v2 - fn[w])
            new = dfn / dyn[w]
            self.sprad[s[w]] = 1.2 * new
            ok = (it >= 1) & (np.abs(new - sigma[w]) <= np.maximum(new, 8.0) * 0.001)
            sigma[w] = new
            self.ede[s[w[ok]]] = v1[w[ok]] - yn[w[ok]]
            live[w[ok]] = False
            w, v2, dfn = w[~ok], v2[~ok], dfn[~ok]
            v1[w] = yn[w] + (dyn[w] / dfn)[:, None] * (fn[w] - v2)

    def start(self):
        S = self.S
        s = np.arange(S)
        self.b = np.zeros((S, self.N))
        self.currents(s, False)
        self.yn = self.y.copy()
        self.fn = self.f(s, self.yn)
        self.ede = self.fn.copy()
        self.sprad = np.zeros(S)
        self.rho(s)
        h = np.maximum(np.minimum(H_MAX, 1 / self.sprad), self.hmin)
        wt = self.tol * np.abs(self.yn) + self.tol
        d = (self.f(s, self.yn + h[:, None] * self.fn) - self.fn) / wt
        est = h * np.sqrt((d * d).sum(1) / self.N)
        self.h = np.where(0.1 * h < H_MAX * np.sqrt(est), np.maximum(0.1 * h / np.sqrt(est), self.hmin), H_MAX)
        self.t_now, self.t_old = np.zeros(S), np.zeros(S)
        self.sum_dt, self.newspc, self.fresh = np.zeros(S), np.ones(S, bool), np.zeros(S, bool)
        self.first, self.hold, self.cold = np.ones(S, bool), np.zeros(S), np.zeros(S)
        x = np.sqrt(self.tol / (10 * UROUND))
        self.mmax = int(x) if x - int(x) < 0.5 else int(x + 0.9)
        self.iext = self.amp.copy()

    def step(self, s, h, m):
        yn, fn = self.yn[s], self.fn[s]
        hc = h[:, None]
        first = np.array([_stages(k)[0] for k in m])[:, None]
        a, b, c = self.y[s], yn.copy(), yn + hc * first * fn      # Y_{j-2}, Y_{j-1}, Y_j
        for j in range(1, int(m.max())):
            w = np.nonzero(m > j)[0]
            co = np.array([_stages(m[k])[j] for k in w]).T[:, :, None]
            f = self.f(s[w], c[w])
            out = co[0] * c[w] + co[1] * b[w] + co[2] * yn[w] + hc[w] * co[3] * (f - co[4] * fn[w])
            a[w], b[w], c[w] = b[w], c[w], out
        return a, c

    def interval(self, tend):
        """Every system to the end of one output interval."""
        s = np.nonzero(self.sum_dt != 0)[0]
        if len(s):
            self.currents(s, True, self.sum_dt[s])
            self.sum_dt[s] = 0
        live = np.ones(self.S, bool)
        while live.any():
            s = np.nonzero(live)[0]
            r = s[self.newspc[s]]
            if len(r):
                self.rho(r)
                self.fresh[r] = True
            left = np.abs(tend - self.t_now[s])
            last = 1.1 * self.h[s] >= left
            self.h[s] = np.where(last, left, self.h[s])
            m = 1 + np.sqrt(1.54 * self.h[s] * self.sprad[s] + 1).astype(int)
            over = m > self.mmax
            m = np.where(over, self.mmax, m)
            self.h[s] = np.where(over, (m * m - 1.0) / (1.54 * self.sprad[s]), self.h[s])
            last &= ~over
            h = np.maximum(self.h[s], self.hmin)
            a, y = self.step(s, h, m)
            yn, fn = self.yn[s], self.fn[s]
            f = self.f(s, y)
            wt = self.tol * np.maximum(np.abs(y), np.abs(yn)) + self.tol
            d = (0.8 * (yn - y) + 0.4 * h[:, None] * (fn + f)) / wt
            err = np.sqrt((d * d).sum(1) / self.N)
            cr = np.cbrt(err)
            self.y[s] = y
            bad = err > 1
            self.h[s] = np.where(bad, 0.8 * self.h[s] / cr, self.h[s])
            small = bad & (self.h[s] < self.hmin)
            rej = bad & ~small
            self.newspc[s[rej]] = ~self.fresh[s[rej]]
            k = np.nonzero(~rej)[0]
            if not len(k):
                continue
            q = s[k]
            self.t_now[q] += h[k]
            self.fresh[q] = False
            self.newspc[q] = False
            self.yn[q], self.fn[q], self.y[q] = y[k], f[k], a[k]
            ratio = np.where(self.first[q], 0.8 / np.maximum(cr[k], 1e-300),
                             0.8 * self.h[q] * self.cold[q] / np.maximum(np.abs(self.hold[q]) * cr[k] ** 2, 1e-300))
            self.h[q] = np.maximum(0.1, np.minimum(10.0, ratio)) * self.h[q]
            self.h[q] = np.maximum(self.hmin, np.minimum(H_MAX, self.h[q]))
            self.first[q], self.hold[q], self.cold[q] = False, h[k], cr[k]
            self.sum_dt[q] += self.t_now[q] - self.t_old[q]
            self.t_old[q] = self.t_now[q]
            due = (self.sum_dt[q] >= self.integ) if self.t in ("go", "pkj") else (self.sum_dt[q] > self.integ)
            end = last[k]
            u = q[due & ~end]
            if len(u):
                self.currents(u, True, self.sum_dt[u])
                self.sum_dt[u] = 0
            live[q[end]] = False
        return self.yn.copy()


def exact(case, seed):
    if case["kind"] != "cells" or case["warm"]:
        return None      # all types together, or a start within a spiking run: minutes in numpy
    nc = NC[case["type"]] * case["n"] * case["nx"] * case["ny"]
    if nc * case["iv"] > EXACT_LIMIT[case["type"]]:
        return None
    t = "gr" if case["type"] == "grfull" else case["type"]
    with np.errstate(all="ignore"):
        X = _Exact(case, seed)
        X.start()
        soma = []
        for k in range(case["iv"]):
            out = X.interval((k + 1) * H_MAX)
            comp = 16 if case["type"] == "grfull" else {"pkj": 1599, "go": 30}.get(t, 1)
            soma.append(out[:, comp::X.nc1].ravel())
    return {t: {"v_new": out.ravel(), "v": X.v.ravel(), "ca": X.P.ca.ravel(), "soma": np.array(soma)}}
