"""What this library is timed on: calls that a Pauli-propagation program makes.

A case is a dict of plain values.  `prepare` makes what the program has in hand
before the call (an observable on the host, a circuit, a resident vector),
`run` makes one pass through the public API and returns the term arrays and
numbers it computed, `exact` restates the same pass in numpy where that is
quick.  Term arrays are read into GPU tensors (pp_download takes device
pointers): a program that goes on with a propagated operator keeps it there.

Kinds, and what each stands for:
  circuit   a Trotterised circuit in one evolve! call from the observable: the
            method's main use.  Open lattices of rows x cols qubits (RZZ on the
            edges, RX on the sites), or the degree-3 random graph on 127 qubits.
  layers    the same circuit one evolve! call per layer, a channel and <O> after
            each, as a program that records a time series runs it.
  step      evolve (the non-mutating form) of a resident operator by a few
            rotations: one Trotter step of an operator that is large already, or
            a single gate on a small one; with or without EnergyCorrection.
  window    evolve! that merges every `window` rotations only, with a local
            truncation of the appended terms: a Heisenberg chain.
  adaptive  evolve! under AdaptiveTruncation (a fixed term budget): the same chain.
  batch     many independent instances of one circuit in a single pass.
  product   the anticommutator of two operators.
  measure   numbers read off a resident operator: <O>, variance, norm.
  learned   the network-ranked budget cut of a resident operator.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paulioperators.jl_b200"))
import pauliprop as pp  # noqa: E402
from pauliprop import circuits  # noqa: E402

M64 = (1 << 64) - 1


def listed():
    return [
        # the smallest circuit anyone runs: 20-qubit chain, a few hundred terms; latency
        {"name": "chain20", "kind": "circuit", "rows": 1, "cols": 20, "layers": 8, "theta_j": 0.3, "theta_h": 0.2,
         "thresh": 1e-5, "wmax": 20, "noise": 0.0},
        # 127 qubits (two-word keys), noisy, tens of thousands of terms
        {"name": "graph127", "kind": "circuit", "graph_seed": 130, "layers": 24, "thresh": 1e-4, "wmax": 10,
         "noise": 5e-4},
        # the headline circuit: 8 x 8 lattice, 3,520 rotations, millions of terms
        {"name": "lattice64", "kind": "circuit", "rows": 8, "cols": 8, "layers": 20, "theta_j": 0.3, "theta_h": 0.25,
         "thresh": 1e-5, "wmax": 12, "noise": 1e-3},
        # a time series, layer by layer, on a lattice that is no power of two
        {"name": "layers_7x9", "kind": "layers", "rows": 7, "cols": 9, "layers": 9, "theta_j": 0.25, "theta_h": 0.2,
         "thresh": 2e-5, "wmax": 10, "noise": 1e-3},
        # one gate on a small operator: the smallest call
        {"name": "gate_small", "kind": "step", "qubits": 20, "terms": 511, "rotations": 1, "thresh": 1e-6, "wmax": 20,
         "energy": False},
        # part of a Trotter step on a large operator
        {"name": "step_large", "kind": "step", "qubits": 64, "terms": 1500001, "rotations": 9, "thresh": 1e-5,
         "wmax": 12, "energy": False},
        # the same with the truncation's energy change recorded, two-word keys
        {"name": "step_energy", "kind": "step", "qubits": 100, "terms": 200003, "rotations": 24, "thresh": 1e-5,
         "wmax": 12, "energy": True},
        # rare merges with a local truncation
        {"name": "window8", "kind": "window", "qubits": 24, "steps": 4, "dt": 0.05, "window": 8, "thresh": 1e-6,
         "local": 1e-7},
        # a fixed term budget after every rotation
        {"name": "adaptive", "kind": "adaptive", "qubits": 30, "steps": 3, "dt": 0.08, "budget": 20000},
        # independent instances in one pass
        {"name": "batch", "kind": "batch", "rows": 6, "cols": 6, "instances": 48, "layers": 8, "thresh": 1e-4},
        # {H, O}: operator algebra
        {"name": "anticommutator", "kind": "product", "qubits": 40, "left": 157, "right": 9001},
        # numbers off a resident operator
        {"name": "measure", "kind": "measure", "qubits": 64, "terms": 1200007},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _int(rng, lo, hi):
    return int(round(_log(rng, lo, hi)))


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "graph", "layers", "step", "step", "window", "adaptive", "batch",
                       "product", "measure", "learned"])
    if kind in ("circuit", "layers"):
        return {"kind": kind, "rows": rng.randint(1, 8), "cols": rng.randint(3, 10),
                "layers": _int(rng, 2, 20 if kind == "circuit" else 10), "theta_j": rng.uniform(0.1, 0.28),
                "theta_h": rng.uniform(0.1, 0.22), "thresh": _log(rng, 1.5e-5, 3e-4), "wmax": rng.randint(5, 11),
                "noise": rng.choice([0.0, 1e-3, 5e-3])}
    if kind == "graph":
        return {"kind": "circuit", "graph_seed": circuits.default_graph_seed(start=rng.randint(127, 999)),
                "layers": _int(rng, 3, 20), "thresh": _log(rng, 2e-4, 3e-3), "wmax": rng.randint(6, 10),
                "noise": rng.choice([0.0, 5e-4])}
    if kind == "step":
        qubits = rng.randint(16, 127)
        return {"kind": "step", "qubits": qubits, "terms": _int(rng, 100, 1500000 if qubits <= 64 else 700000),
                "rotations": _int(rng, 1, 28), "thresh": _log(rng, 1e-6, 1e-4), "wmax": rng.randint(8, 16),
                "energy": rng.random() < 0.4}
    if kind == "window":
        return {"kind": "window", "qubits": rng.randint(8, 80), "steps": rng.randint(1, 4),
                "dt": rng.uniform(0.02, 0.06), "window": rng.randint(2, 12), "thresh": _log(rng, 1e-6, 1e-4),
                "local": _log(rng, 1e-8, 1e-6)}
    if kind == "adaptive":
        return {"kind": "adaptive", "qubits": rng.randint(8, 70), "steps": rng.randint(1, 4),
                "dt": rng.uniform(0.03, 0.1), "budget": _int(rng, 300, 60000)}
    if kind == "batch":
        return {"kind": "batch", "rows": rng.randint(2, 6), "cols": rng.randint(2, 7),
                "instances": _int(rng, 3, 80), "layers": rng.randint(3, 8), "thresh": _log(rng, 1e-4, 1e-3)}
    if kind == "product":
        return {"kind": "product", "qubits": rng.randint(10, 120), "left": _int(rng, 5, 300),
                "right": _int(rng, 50, 12000)}
    if kind == "measure":
        return {"kind": "measure", "qubits": rng.randint(20, 127), "terms": _int(rng, 200, 1200000)}
    return {"kind": "learned", "rows": rng.randint(4, 8), "cols": rng.randint(4, 8), "terms": _int(rng, 2000, 1500000),
            "keep": rng.uniform(0.2, 0.8)}


# ------------------------------------------------------------------ circuits
def _lattice(rows, cols):
    """Edges of an open lattice, row by row and then column by column (1-based qubits)."""
    q = lambda r, c: cols * r + c + 1  # noqa: E731
    edges = [(q(r, c), q(r, c + 1)) for r in range(rows) for c in range(cols - 1)]
    return edges + [(q(r, c), q(r + 1, c)) for r in range(rows - 1) for c in range(cols)]


class Frame:
    """What a seed changes: the labels of the qubits (rotated by `shift`) and the signs a
    conjugation by a Pauli string R gives (of coefficients and of angles).  Seeds are
    different inputs with different results, and cost exactly the same."""

    def __init__(self, N, seed):
        rng = np.random.default_rng([7, seed])
        self.N = N
        self.shift = int(rng.integers(0, N))
        bits = rng.integers(0, 2, (2, N))
        self.rz, self.rx = (sum(1 << q for q in range(N) if row[q]) for row in bits.tolist())

    def label(self, m):
        return ((m << self.shift) | (m >> (self.N - self.shift))) & ((1 << self.N) - 1)

    def sign(self, z, x):
        return -1.0 if ((z & self.rx).bit_count() + (x & self.rz).bit_count()) & 1 else 1.0

    def circuit(self, gens, angles):
        out = [pp.PauliBasis(self.N, self.label(g.z), self.label(g.x)) for g in gens]
        return out, [a * self.sign(g.z, g.x) for g, a in zip(out, angles)]

    def terms(self, obs):
        out = [(self.label(z), self.label(x), c) for z, x, c in obs]
        return [(z, x, c * self.sign(z, x)) for z, x, c in out]

    def arrays(self, z, x, c):
        """The same of term arrays, which come back sorted by (z, x)."""
        z, x = _rotl(z, self.shift, self.N), _rotl(x, self.shift, self.N)
        rz, rx = pp.pack_keys(self.N, [(self.rz, self.rx)])
        c = np.where(_parity(z & rx) ^ _parity(x & rz), -c, c)
        o = _order(z, x)
        return z[o], x[o], c[o]


def _shl(v, s):
    if v.shape[1] == 1:
        return v << np.uint64(s) if s < 64 else np.zeros_like(v)
    lo, hi = v[:, 0], v[:, 1]
    if s == 0:
        return v
    if s >= 64:
        return np.stack([np.zeros_like(lo), lo << np.uint64(s - 64)], 1)
    return np.stack([lo << np.uint64(s), (hi << np.uint64(s)) | (lo >> np.uint64(64 - s))], 1)


def _shr(v, s):
    if v.shape[1] == 1:
        return v >> np.uint64(s) if s < 64 else np.zeros_like(v)
    lo, hi = v[:, 0], v[:, 1]
    if s == 0:
        return v
    if s >= 128:
        return np.zeros_like(v)
    if s >= 64:
        return np.stack([hi >> np.uint64(s - 64), np.zeros_like(hi)], 1)
    return np.stack([(lo >> np.uint64(s)) | (hi << np.uint64(64 - s)), hi >> np.uint64(s)], 1)


def _rotl(v, s, N):
    mask = pp.pack_word(N, (1 << N) - 1)[None, :]
    return (_shl(v, s) | _shr(v, N - s)) & mask


def _circuit(case, seed):
    """(N, one layer's generators, its angles, the observable's (z, x, c))."""
    if "graph_seed" in case:
        w = circuits.random_graph127(seed=case["graph_seed"], layers=1)
        N, layer, ang, obs = w.N, w.layer, w.angles, w.observable
    else:
        rows, cols = case["rows"], case["cols"]
        N = rows * cols
        edges = _lattice(rows, cols)
        layer = [circuits.zz(N, i, j) for i, j in edges] + [circuits.xq(N, q) for q in range(1, N + 1)]
        ang = [case["theta_j"]] * len(edges) + [case["theta_h"]] * N
        obs = [(1 << (N // 2 - 1), 0, 1.0)] if rows == 1 else [(1 << q, 0, 1.0 / N) for q in range(N)]
    f = Frame(N, seed)
    return (N, *f.circuit(layer, ang), f.terms(obs))


def _chain(case, seed):
    """Trotter steps of a Heisenberg chain, evolving Z of the middle site."""
    N = case["qubits"]
    terms = circuits.heisenberg_chain_terms(N)
    gens, ang = circuits.trotterize(terms, case["dt"] * case["steps"], case["steps"], order=1)
    f = Frame(N, seed)
    return (N, *f.circuit(gens, ang), f.terms([(1 << (N // 2), 0, 1.0)]))


def _strategy(case):
    return pp.CompositeTruncation(pp.CoeffTruncation(case["thresh"]), pp.WeightTruncation(case["wmax"]))


def _words(N, obs):
    z, x = pp.pack_keys(N, [(o[0], o[1]) for o in obs])
    return z, x, np.array([o[2] for o in obs], dtype=np.float64)


# ------------------------------------------------------------------ resident operators
def _operator(N, n, seed, wmax=8, gens=(), tag=0):
    """About n terms of a propagated operator: strings of weight up to wmax, some of
    them partners of others under `gens`, |c| spread over four decades; sorted by
    (z, x), unique keys.  The strings are those of (N, n), in the seed's frame."""
    rng = np.random.default_rng([3, N, n, tag])
    nw = (N + 63) // 64
    z = np.zeros((n, nw), dtype=np.uint64)
    x = np.zeros((n, nw), dtype=np.uint64)
    wt = rng.integers(1, wmax + 1, n)
    one = np.uint64(1)
    for j in range(wmax):
        on = wt > j
        site = rng.integers(0, N, n)
        kind = rng.integers(0, 3, n)
        bit = one << (site & 63).astype(np.uint64)
        for w in range(nw):
            here = on & (site >> 6 == w)
            x[:, w] ^= np.where(here & (kind < 2), bit, np.uint64(0))
            z[:, w] ^= np.where(here & (kind > 0), bit, np.uint64(0))
    if len(gens):
        # the second half: partners of terms of the first half that anticommute
        half = n // 2
        at = np.linspace(half, n, len(gens) + 1).astype(int)
        for g, a, b in zip(gens, at[:-1], at[1:]):
            gz, gx = pp.pack_keys(N, [(g.z, g.x)])
            src = rng.integers(0, half, b - a)
            zz, xx = z[src], x[src]
            anti = (_parity(zz & gx) ^ _parity(xx & gz))[:, None]
            z[a:b] = np.where(anti, zz ^ gz, z[a:b])
            x[a:b] = np.where(anti, xx ^ gx, x[a:b])
    c = 10.0 ** rng.uniform(-5, -1, n) * rng.choice([-1.0, 1.0], n)
    first = np.unique(_mix(z, x), return_index=True)[1]
    return Frame(N, seed).arrays(z[first], x[first], c[first])


def _order(z, x):
    cols = [x[:, w] for w in range(x.shape[1])] + [z[:, w] for w in range(z.shape[1])]
    return np.lexsort(cols)


def _popcount(a):
    return np.bitwise_count(a).sum(axis=-1).astype(np.int64)


def _parity(a):
    return (_popcount(a) & 1).astype(bool)


def _step(case, seed):
    """The operator, and some consecutive generators of a chain's Trotter layer."""
    N, k = case["qubits"], case["rotations"]
    rng = np.random.default_rng([5, N, k])
    at = int(rng.integers(0, N - 1))
    pool = [circuits.zz(N, i, i + 1) for i in range(1, N)] + [circuits.xq(N, q) for q in range(1, N + 1)]
    gens = [pool[(at + 3 * i) % len(pool)] for i in range(k)]
    obs = _operator(N, case["terms"], seed, gens=gens)
    return (N, obs, *Frame(N, seed).circuit(gens, rng.uniform(0.1, 0.4, k).tolist()))


def _product(case, seed):
    N = case["qubits"]
    return N, _operator(N, case["left"], seed, wmax=3, tag=1), _operator(N, case["right"], seed, wmax=6, tag=2)


def _measure(case, seed):
    N = case["qubits"]
    return N, _operator(N, case["terms"], seed), Frame(N, seed + 1).rx


def _vector(N, z, x, c):
    v = pp.SparsePauliVector(N, 2 * len(c), 2 * len(c))
    v.upload(z, x, c, sorted=True)
    return v


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("circuit", "layers"):
        N, layer, ang, obs = _circuit(case, seed)
        s.update(N=N, obs=_words(N, obs), trunc=_strategy(case), noise=case["noise"], per=len(layer),
                 channel="dephasing" if "graph_seed" in case else "depolarizing",
                 v=pp.SparsePauliVector(N, 1 << 16, 1 << 24))
        if kind == "circuit":
            s.update(gens=layer * case["layers"], ang=ang * case["layers"])
        else:
            s.update(gens=layer, ang=ang)
    elif kind == "step":
        N, obs, gens, ang = _step(case, seed)
        s.update(gens=gens, ang=ang, trunc=_strategy(case), v=_vector(N, *obs))
    elif kind in ("window", "adaptive"):
        N, gens, ang, obs = _chain(case, seed)
        s.update(N=N, obs=_words(N, obs), gens=gens, ang=ang, v=pp.SparsePauliVector(N, 1 << 16, 1 << 20))
    elif kind == "batch":
        rows, cols, count = case["rows"], case["cols"], case["instances"]
        edges = _lattice(rows, cols)
        N = rows * cols
        f = Frame(N, seed)
        rng = np.random.default_rng([13, N, count])
        layer = [circuits.zz(N, i, j) for i, j in edges] + [circuits.xq(N, q) for q in range(1, N + 1)]
        layer, sign = f.circuit(layer, [1.0] * len(layer))
        obs = []
        for _ in range(count):
            z = x = 0
            for site in rng.choice(N, min(N, int(rng.integers(1, 4))), replace=False):
                t = int(rng.integers(0, 3))
                x |= int(t < 2) << int(site)
                z |= int(t > 0) << int(site)
            obs.append(f.terms([(z, x, 1.0)]))
        # four angle columns: RZZ and RX with each sign; depths spread over [layers / 2, layers]
        ang = rng.uniform(0.08, 0.25, (count, 2))
        col = [2 * (i >= len(edges)) + (sg < 0) for i, sg in enumerate(sign)]
        depth = [case["layers"] - (i * 5) % max(1, case["layers"] // 2) for i in range(count)]
        s.update(N=N, obs=obs, gens=layer * case["layers"], acol=col * case["layers"],
                 ang=np.stack([ang[:, 0], -ang[:, 0], ang[:, 1], -ang[:, 1]], 1), ends=[d * len(layer) for d in depth],
                 trunc=pp.CoeffTruncation(case["thresh"]), v=pp.SparsePauliVector(128, 1 << 16, 16))
    elif kind == "product":
        N, a, b = _product(case, seed)
        s.update(a=_vector(N, *a), b=_vector(N, *b))
    elif kind == "measure":
        N, obs, ket = _measure(case, seed)
        s.update(v=_vector(N, *obs), ket=ket)
    elif kind == "learned":
        rows, cols = case["rows"], case["cols"]
        s.update(v=_vector(rows * cols, *_operator(rows * cols, case["terms"], seed)),
                 mlp=pp.MLP(pp.learned.init_params(seed)),
                 ctx=pp.lattice_feature_ctx(rows, cols, 5, 10, 0.27, 0.23))
        s["budget"] = int(case["keep"] * len(s["v"]))
    return s


# ------------------------------------------------------------------ run
def _terms(v):
    """The term arrays of v in GPU tensors."""
    n = len(v)
    z = torch.empty((n, v.nw), dtype=torch.int64, device="cuda")
    x = torch.empty((n, v.nw), dtype=torch.int64, device="cuda")
    c = torch.empty(n, dtype=torch.float64, device="cuda")
    pp.spv.check(pp.spv.lib.pp_download(v._h, z.data_ptr(), x.data_ptr(), c.data_ptr(), n, None))
    return {"z": z, "x": x, "c": c}


def run(s):
    kind = s["case"]["kind"]
    if kind == "circuit":
        v = s["v"]
        v.upload(*s["obs"])
        noise = {"channel": (s["channel"], s["noise"], None), "channel_every": s["per"]} if s["noise"] else {}
        _, e = pp.evolve_(v, s["gens"], s["ang"], truncation=s["trunc"], return_expectation=True, **noise)
        return {"expect": e, **_terms(v)}
    if kind == "layers":
        v = s["v"]
        v.upload(*s["obs"])
        series = []
        for _ in range(s["case"]["layers"]):
            pp.evolve_(v, s["gens"], s["ang"], truncation=s["trunc"])
            if s["noise"]:
                pp.depolarizing_channel_(v, s["noise"])
            series.append(pp.expectation_value(v, 0))
        return {"expect": np.array(series), **_terms(v)}
    if kind == "step":
        corr = pp.EnergyCorrection(0) if s["case"]["energy"] else None
        w = pp.evolve(s["v"], s["gens"], s["ang"], truncation=s["trunc"], correction=corr)
        out = _terms(w)
        if corr is not None:
            out["energy"] = corr.accumulated_energy
        return out
    if kind in ("window", "adaptive"):
        v = s["v"]
        v.upload(*s["obs"])
        if kind == "window":
            kw = {"window": s["case"]["window"], "truncation": pp.CoeffTruncation(s["case"]["thresh"]),
                  "local_truncation": pp.CoeffTruncation(s["case"]["local"])}
        else:
            kw = {"truncation": pp.AdaptiveTruncation(s["case"]["budget"], 1e-12)}
        _, e = pp.evolve_(v, s["gens"], s["ang"], return_expectation=True, **kw)
        return {"expect": e, **_terms(v)}
    if kind == "batch":
        r = pp.evolve_batch(s["obs"], s["gens"], s["acol"], s["ang"], s["ends"], nq=s["N"], truncation=s["trunc"],
                            vector=s["v"])
        return {"expect": r.expect, "terms": r.n_final}
    if kind == "product":
        return _terms(pp.anticommutator(s["a"], s["b"]))
    if kind == "measure":
        v = s["v"]
        return {"expect": pp.expectation_value(v, s["ket"]), "variance": pp.variance(v, s["ket"]), "norm": pp.norm(v)}
    w = s["v"].copy()
    cut = pp.learned_truncate_(w, s["mlp"], s["ctx"], s["budget"])
    return {"cut": torch.tensor(cut, dtype=torch.float32), **_terms(w)}


# ------------------------------------------------------------------ work
def _mean_terms(case):
    """Rough mean live terms of a circuit-like pass (fitted to a few runs; the order of
    magnitude is what it is for)."""
    kind = case["kind"]
    if kind == "adaptive":
        return 0.5 * case["budget"]
    if kind == "window":
        return 4e3 * min(1.0, 1e-6 / case["thresh"]) ** 0.5
    if "graph_seed" in case:
        return 4e4 * (1e-4 / case["thresh"]) ** 0.9
    N = case["rows"] * case["cols"]
    if case["rows"] == 1:
        return 200.0
    full = 1.75e6 * (1e-5 / case["thresh"]) * (N / 64.0)
    return max(N, full * min(1.0, case["layers"] / 20.0) ** 2 * (case.get("theta_j", 0.2) / 0.3) ** 2)


def work(case):
    kind = case["kind"]
    if kind in ("circuit", "layers", "window", "adaptive"):
        if "graph_seed" in case:
            nw, rot = 2, 271 * case["layers"]
        elif kind in ("window", "adaptive"):
            nw, rot = (1 if case["qubits"] <= 64 else 2), (4 * case["qubits"] - 3) * case["steps"]
        else:
            n = case["rows"] * case["cols"]
            nw, rot = (1 if n <= 64 else 2), case["layers"] * (len(_lattice(case["rows"], case["cols"])) + n)
        t = _mean_terms(case)
        return {"bytes": 2.0 * rot * t * (16 * nw + 8), "flops": 4.0 * rot * t}
    if kind == "step":
        b = 16 * (1 if case["qubits"] <= 64 else 2) + 8
        return {"bytes": 2.0 * case["rotations"] * case["terms"] * b, "flops": 4.0 * case["rotations"] * case["terms"]}
    if kind == "batch":
        n = case["rows"] * case["cols"]
        rot = case["layers"] * 0.75 * (len(_lattice(case["rows"], case["cols"])) + n)
        t = case["instances"] * 2e3 * (1e-4 / case["thresh"])
        return {"bytes": 2.0 * rot * t * 40, "flops": 4.0 * rot * t}
    if kind == "product":
        b = 16 * (1 if case["qubits"] <= 64 else 2) + 8
        return {"bytes": float((case["left"] + case["right"] + 0.5 * case["left"] * case["right"]) * b),
                "flops": 2.0 * case["left"] * case["right"]}
    if kind == "measure":
        return {"bytes": float(case["terms"] * (16 * (1 if case["qubits"] <= 64 else 2) + 8)),
                "flops": 8.0 * case["terms"]}
    return {"bytes": 24.0 * case["terms"] * (1 + 2 * case["keep"]), "flops": 2.0 * 5200 * case["terms"]}


# ------------------------------------------------------------------ exact
def _mix(z, x):
    """A 64-bit hash of each key (equal keys equal, distinct ones distinct in practice)."""
    h = np.zeros(len(z), dtype=np.uint64)
    for w in range(z.shape[1]):
        for a in (z[:, w], x[:, w]):
            h = (h ^ a) * np.uint64(0x9E3779B97F4A7C15)
            h ^= h >> np.uint64(29)
            h *= np.uint64(0xBF58476D1CE4E5B9)
            h ^= h >> np.uint64(32)
    return h


def _combine(z, x, c):
    """Equal keys summed."""
    o = np.argsort(_mix(z, x), kind="stable")
    z, x, c = z[o], x[o], c[o]
    head = np.ones(len(c), dtype=bool)
    head[1:] = (z[1:] != z[:-1]).any(1) | (x[1:] != x[:-1]).any(1)
    at = np.flatnonzero(head)
    return z[at], x[at], np.add.reduceat(c, at) if len(at) else c[:0]


def _rotated(z, x, c, gz, gx, th):
    """The cos branch (in place in c) and the appended sin branches of one rotation."""
    m1 = _popcount(z & gx)
    anti = ((m1 + _popcount(x & gz)) & 1).astype(bool)
    zp, xp = z[anti] ^ gz, x[anti] ^ gx
    k = (_popcount(zp & xp) - int(_popcount(gz & gx)[0]) - _popcount(z[anti] & x[anti]) + 2 * m1[anti]) & 3
    cp = (k - 2) * math.sin(th) * c[anti]
    c = np.where(anti, c * math.cos(th), c)
    return c, zp, xp, cp


def _propagate(N, obs, gens, ang, window=1, keep=None, local=0.0, budget=None, noise=None, per=0, after=None, limit=2e8):
    """evolve! by its definition: rotate, append, and every `window` rotations sum equal
    keys and truncate.  None when it would take too long."""
    z, x, c = obs
    spent = 0
    for i, (g, th) in enumerate(zip(gens, ang)):
        gz, gx = pp.pack_keys(N, [(g.z, g.x)])
        c, zp, xp, cp = _rotated(z, x, c, gz, gx, th)
        if local:
            on = np.abs(cp) > local
            zp, xp, cp = zp[on], xp[on], cp[on]
        z, x, c = np.concatenate([z, zp]), np.concatenate([x, xp]), np.concatenate([c, cp])
        spent += len(c)
        if spent > limit:
            return None
        if (i + 1) % window == 0 or i + 1 == len(gens):
            z, x, c = _combine(z, x, c)
            if budget is not None:
                cut = np.partition(np.abs(c), len(c) - 1 - budget)[len(c) - 1 - budget] if len(c) > budget else 1e-12
                on = np.abs(c) > cut
            else:
                on = keep(z, x, c)
            z, x, c = z[on], x[on], c[on]
        if noise and per and (i + 1) % per == 0:
            c = c * noise(z, x)
        if after and (i + 1) % per == 0:
            after(z, x, c)
    o = _order(z, x)
    return z[o], x[o], c[o]


def _ket(z, x, c, ket):
    k = np.array([[(ket >> (64 * w)) & M64 for w in range(z.shape[1])]], dtype=np.uint64)
    d = (x == 0).all(1)
    return math.fsum(np.where(_parity(z[d] & k), -c[d], c[d]).tolist())


def _filter(case):
    return lambda z, x, c: (np.abs(c) > case["thresh"]) & (_popcount(z | x) <= case["wmax"])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("circuit", "layers"):
        N, layer, ang, obs = _circuit(case, seed)
        series = []
        noise = None
        if case["noise"]:
            lam = 1.0 - 4.0 * case["noise"] / 3.0 if "graph_seed" not in case else 1.0 - 2.0 * case["noise"]
            noise = (lambda z, x: lam ** _popcount(z | x)) if "graph_seed" not in case else \
                (lambda z, x: lam ** _popcount(x))
        t = _propagate(N, _words(N, obs), layer * case["layers"], ang * case["layers"], keep=_filter(case), noise=noise,
                       per=len(layer), after=lambda z, x, c: series.append(_ket(z, x, c, 0)), limit=5e7)
        if t is None:
            return None
        return {"expect": series[-1] if kind == "circuit" else np.array(series), "z": None, "x": None, "c": t[2]}
    if kind == "step":
        if case["energy"]:
            return None
        N, obs, gens, ang = _step(case, seed)
        t = _propagate(N, obs, gens, ang, keep=_filter(case), limit=3e7)
        return None if t is None else {"z": None, "x": None, "c": t[2]}
    if kind in ("window", "adaptive"):
        N, gens, ang, obs = _chain(case, seed)
        kw = {"budget": case["budget"]} if kind == "adaptive" else \
            {"window": case["window"], "local": case["local"], "keep": lambda z, x, c: np.abs(c) > case["thresh"]}
        t = _propagate(N, _words(N, obs), gens, ang, limit=3e7, **kw)
        return None if t is None else {"expect": _ket(*t, 0), "z": None, "x": None, "c": t[2]}
    if kind == "product":
        N, a, b = _product(case, seed)
        parts = []
        for i in range(len(a[2])):
            az, ax = a[0][i:i + 1], a[1][i:i + 1]
            z, x = az ^ b[0], ax ^ b[1]
            # phase of P_a P_b as a power of i; odd powers cancel in the anticommutator
            k = (_popcount(z & x) - _popcount(az & ax) - _popcount(b[0] & b[1]) + 2 * _popcount(ax & b[0])) & 3
            on = (k & 1) == 0
            parts.append((z[on], x[on], 2.0 * np.where(k[on] == 0, 1.0, -1.0) * a[2][i] * b[2][on]))
        z, x, c = _combine(*(np.concatenate(p) for p in zip(*parts)))
        o = _order(z, x)
        return {"z": None, "x": None, "c": c[o]}
    if kind == "measure":
        N, (z, x, c), ket = _measure(case, seed)
        e = _ket(z, x, c, ket)
        k = np.array([[(ket >> (64 * w)) & M64 for w in range(z.shape[1])]], dtype=np.uint64)
        ph = ((4 - (_popcount(z & x) & 3)) % 4 + 2 * (_popcount(z & (x ^ k)) & 1)) & 3
        o = np.argsort(_mix(x, x), kind="stable")
        head = np.ones(len(c), dtype=bool)
        head[1:] = (x[o][1:] != x[o][:-1]).any(1)
        at = np.flatnonzero(head)
        sg = np.where(ph >= 2, -c, c)[o]
        im = (ph & 1).astype(bool)[o]
        re = np.add.reduceat(np.where(im, 0.0, sg), at)
        ii = np.add.reduceat(np.where(im, sg, 0.0), at)
        return {"expect": e, "variance": math.fsum((re * re + ii * ii).tolist()) - e * e,
                "norm": math.sqrt(math.fsum((c * c).tolist()))}
    return None
