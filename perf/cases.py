"""The work this framework is measured on: what a program that estimates
Clifford+T probabilities has it do, through the package's public entry points.

Kinds of case (`kind`):
  samples  Backend.singleProjectorSample: one projector's sampled estimator, the
           bulk of every probability() call
  exact    Backend.exactProjector on a query's two projectors: the estimator
           without sampling, which the backend takes by itself when the
           decomposition has few terms
  queries  Backend.run_queries(batched): many probability queries at once, as a
           server or a sampleQubits chain sends them
  inner    Backend.innerProductExact on stabilizer states a program holds
  states   Backend.randomStabilizerState, then Backend.measurePauli on them

Projectors come from seeded random Clifford+T circuits (H/S/X/Z 0.55, CNOT 0.30,
T 0.15) through the package's front end, so they have the row counts, weights
and phases that a user's circuits give.
"""
import math

import numpy as np

from circuitsimulator_gb300 import backend, frontend

_gpu = None


def _backend():
    """The one Backend a program keeps open."""
    global _gpu
    if _gpu is None:
        _gpu = backend.Backend(0)
    return _gpu


# ---------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call: a few states on a small decomposition, all latency
        {"name": "samples_t8", "kind": "samples", "t": 8, "n": 6, "k": 4, "exact": False, "count": 32,
         "libc": False},
        # the plain method: 12 T gates, exact decomposition (64 terms), 2000 states, the C library's draws
        {"name": "samples_h12", "kind": "samples", "t": 12, "n": 10, "k": 0, "exact": True, "count": 2000,
         "libc": True},
        # an ordinary sparsified query, odd sizes
        {"name": "samples_t27", "kind": "samples", "t": 27, "n": 13, "k": 11, "exact": False, "count": 3001,
         "libc": True},
        # the plain method at scale: 40 T gates, 2^16 terms, 4096 states (the largest)
        {"name": "samples_t40", "kind": "samples", "t": 40, "n": 24, "k": 16, "exact": False, "count": 4096,
         "libc": True},
        # many terms and few states, counter-based draws (a rank's share of a sharded query)
        {"name": "samples_t57", "kind": "samples", "t": 57, "n": 29, "k": 18, "exact": False, "count": 256,
         "libc": False},
        # one conditional of a sampleQubits chain at the widest rows
        {"name": "samples_t64", "kind": "samples", "t": 64, "n": 32, "k": 14, "exact": False, "count": 2048,
         "libc": True},
        # few enough terms that the backend sums all pairs: exact decomposition, 256 terms
        {"name": "exact_h16", "kind": "exact", "t": 16, "n": 4, "k": 0, "exact": True},
        # the same on a sparsified decomposition, 2048 terms
        {"name": "exact_t21", "kind": "exact", "t": 21, "n": 6, "k": 11, "exact": False},
        # light queries of mixed size in one batch (t 8..23)
        {"name": "queries_light", "kind": "queries", "count": 24, "tmin": 8, "tmax": 23, "samples": 8000,
         "force": False},
        # sampled queries of mixed size in one batch (t 24..64)
        {"name": "queries_sampled", "kind": "queries", "count": 12, "tmin": 24, "tmax": 64, "samples": 200,
         "force": True},
        # inner products of states that the program holds
        {"name": "inner_n40", "kind": "inner", "n": 40, "count": 4096},
        # random states, each projected by one Pauli
        {"name": "states_n31", "kind": "states", "n": 31, "count": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["samples"] * 5 + ["exact", "exact", "queries", "queries", "inner", "states"])
    if kind == "samples":
        if rng.random() < 0.2:
            t = rng.randint(8, 18)
            return {"kind": kind, "t": t, "n": rng.randint(6, 24), "k": 0, "exact": True,
                    "count": _log_int(rng, 16, 4096), "libc": rng.random() < 0.5}
        t = rng.randint(8, 64)
        k = rng.randint(min(4, t // 2), min(18, t - 2))
        most = max(16, min(4096, (1 << 28) >> k))
        return {"kind": kind, "t": t, "n": rng.randint(6, 32), "k": k, "exact": False,
                "count": _log_int(rng, 16, most), "libc": rng.random() < 0.5}
    if kind == "exact":
        if rng.random() < 0.5:
            return {"kind": kind, "t": rng.randint(10, 18), "n": rng.randint(3, 5), "k": 0, "exact": True}
        t = rng.randint(12, 22)
        return {"kind": kind, "t": t, "n": rng.randint(4, 8), "k": rng.randint(4, min(11, t - 1)), "exact": False}
    if kind == "queries":
        if rng.random() < 0.5:
            return {"kind": kind, "count": _log_int(rng, 2, 24), "tmin": 8, "tmax": rng.randint(12, 23),
                    "samples": 8000, "force": False}
        return {"kind": kind, "count": _log_int(rng, 2, 12), "tmin": rng.randint(18, 30),
                "tmax": rng.randint(31, 64), "samples": _log_int(rng, 20, 200), "force": True}
    return {"kind": kind, "n": rng.randint(5, 64), "count": _log_int(rng, 64, 4096)}


# ---------------------------------------------------------------- inputs
def _circuit(n, t, rs):
    """A compiled random circuit with t T gates: one gate per line, one symbol per qubit."""
    lines = []

    def gate(ops):
        lines.append("".join(ops.get(q, "_") for q in range(n)))

    while t > 0:
        r = rs.random_sample()
        if r < 0.55:
            q = int(rs.randint(n))
            g = "HSXZ"[rs.randint(4)]
            for c in ("HXH" if g == "Z" else g):
                gate({q: c})
        elif r < 0.85:
            a, b = (int(v) for v in rs.choice(n, size=2, replace=False))
            gate({a: "C", b: "X"})
        else:
            q = int(rs.randint(n))
            for c in ("SSST" if rs.randint(2) else "T"):
                gate({q: c})
            t -= 1
    return "\n".join(lines) + "\n"


def _projectors(n, t, rs):
    """G' and H' of a random circuit's random outcome on some qubits, as the
    protocol's (phases, x rows, z rows, width); retried until neither is trivial."""
    while True:
        circ = _circuit(n, t, rs)
        qubits = sorted(int(q) for q in rs.choice(n, size=min(n, int(rs.randint(1, 5))), replace=False))
        measure = {q: int(rs.randint(2)) for q in qubits}
        try:
            G, H, nq, width = frontend.projectors(circ, measure, rng=rs)
        except SyntaxError:  # two T gates in a row on one qubit
            continue
        if width != t:
            continue
        Gp, _ = frontend.truncate(nq, G)
        Hp, _ = frontend.truncate(nq, H)
        if not Gp[0] or not Hp[0] or any(p == 2 and x == 0 and z == 0 for p, x, z in zip(*Gp)):
            continue
        return (list(Gp[0]), list(Gp[1]), list(Gp[2]), t), (list(Hp[0]), list(Hp[1]), list(Hp[2]), t)


def _code(t, k, rs):
    return [int.from_bytes(rs.bytes(8), "little") & ((1 << t) - 1) for _ in range(k)]


def _rs(case, seed):
    return np.random.RandomState((int(seed) * 1000003 + 7919) % (1 << 32))


def _k_for(t):
    """Rows of the sparsified decomposition at fidelity bound 0.02, 2^18 terms at most."""
    return min(18, int(math.ceil(1 - 2 * t * math.log2(math.cos(math.pi / 8)) - math.log2(0.02))))


def _queries(case, rs):
    out = []
    span = case["tmax"] - case["tmin"]
    for i in range(case["count"]):
        t = case["tmin"] + (i * span) // max(1, case["count"] - 1)
        exact = t <= 16
        cfg = dict(quiet=1, verbose=0, noapprox=0, samples=case["samples"], bins=1, t=t,
                   k=0 if exact else min(_k_for(t), 16), exact=int(exact), fidbound=0.02, fidelity=0, rank=0, forceL=0,
                   forceSample=int(case["force"]))
        n = int(rs.randint(max(4, min(t // 2, 12)), 17))
        out.append({"cfg": cfg, "projs": list(_projectors(n, t, rs)), "seed": int(rs.randint(1, 1 << 30)),
                    "rng": backend.RNG_LIBC})
    return out


def prepare(case, seed):
    rs = _rs(case, seed)
    gpu = _backend()
    kind = case["kind"]
    st = {"gpu": gpu, "case": case}
    if kind in ("samples", "exact"):
        st["P"], st["P2"] = (backend.projector(*p) for p in _projectors(case["n"], case["t"], rs))
        st["L"] = None if case["exact"] else _code(case["t"], case["k"], rs)
        st["seed"] = int(rs.randint(1, 1 << 30))
    elif kind == "queries":
        st["queries"] = _queries(case, rs)
    elif kind == "inner":
        st["a"] = gpu.randomStabilizerState(case["n"], case["count"], int(rs.randint(1 << 30)))
        st["b"] = gpu.randomStabilizerState(case["n"], case["count"], int(rs.randint(1 << 30)))
    else:
        st["seed"] = int(rs.randint(1 << 30))
        full = (1 << case["n"]) - 1
        st["m"] = rs.randint(4, size=case["count"]).astype(np.int32)
        st["z"] = np.array([int.from_bytes(rs.bytes(8), "little") & full for _ in range(case["count"])], dtype=np.uint64)
        st["x"] = np.array([int.from_bytes(rs.bytes(8), "little") & full for _ in range(case["count"])], dtype=np.uint64)
        # a Pauli with real eigenvalues: i^m matches the parity of its Y factors
        par = np.array([bin(int(a) & int(b)).count("1") & 1 for a, b in zip(st["z"], st["x"])])
        st["m"] = ((st["m"] & 2) | par).astype(np.int32)
    return st


# ---------------------------------------------------------------- one pass
def run(state):
    gpu, case = state["gpu"], state["case"]
    kind = case["kind"]
    if kind == "samples":
        return gpu.singleProjectorSample(state["P"], state["L"], case["exact"], case["count"],
                                         backend.RNG_LIBC if case["libc"] else backend.RNG_PHILOX, state["seed"])
    if kind == "exact":
        return [gpu.exactProjector(P, state["L"], case["exact"], 1.0) for P in (state["P"], state["P2"])]
    if kind == "queries":
        return [[r["numerator"], r["denominator"]] for r in gpu.run_queries(state["queries"], batched=True)]
    if kind == "inner":
        return list(gpu.innerProductExact(state["a"], state["b"]))
    s = gpu.randomStabilizerState(case["n"], case["count"], state["seed"])
    norm = gpu.measurePauli(s, state["m"], state["z"], state["x"])
    return [s.view(np.int64), norm]


# ---------------------------------------------------------------- work
def _terms(t, k, exact):
    return 1 << ((t + 1) // 2) if exact else 1 << k


def work(case):
    """Bytes: the states, projector rows, codes and words that go in and the
    values that come out.  Operations: every (state, term) pair's value is added
    into a sum of four integer coordinates; an inner product or a projection of
    stored states touches each row of the form once per eliminated variable."""
    kind = case["kind"]
    if kind == "samples":
        t, c = case["t"], case["count"]
        chi = _terms(t, case["k"], case["exact"])
        words = (1 + 3 * ((t + 7) // 8) + t * (t - 1) // 2) if case["libc"] else 0
        return {"bytes": 4 * words * c + 8 * c + 8 * case["k"] + 20 * t, "flops": 4 * c * chi}
    if kind == "exact":
        chi = _terms(case["t"], case["k"], case["exact"])
        return {"bytes": 8 * case["k"] + 40 * case["t"] + 16, "flops": 4 * chi * (chi + 1)}
    if kind == "queries":
        b = f = 0
        span = case["tmax"] - case["tmin"]
        for i in range(case["count"]):
            t = case["tmin"] + (i * span) // max(1, case["count"] - 1)
            exact = t <= 16
            chi = _terms(t, min(_k_for(t), 16), exact)
            if not case["force"] and 2 * case["samples"] > chi - 1:
                f += 2 * 4 * chi * (chi + 1) // 2
                b += 40 * t + 16
            else:
                f += 2 * 4 * case["samples"] * chi
                b += 40 * t + 16 + 2 * case["samples"] * 4 * (1 + 3 * ((t + 7) // 8) + t * (t - 1) // 2)
        return {"bytes": b, "flops": f}
    n, c = case["n"], case["count"]
    state = 40 + 3 * 8 * n
    if kind == "inner":
        return {"bytes": c * (2 * state + 12), "flops": c * n * n}
    return {"bytes": c * (2 * state + 8 + 20), "flops": c * n * n}


# ---------------------------------------------------------------- exact values
def _project(psi, P):
    """(1 + i^phase Z(z) X(x))/2 for every row, in order, on a state vector."""
    y = np.arange(len(psi), dtype=np.uint64)
    for ph, x, z in zip(*P[:3]):
        sign = 1.0 - 2.0 * (np.bitwise_count(y & np.uint64(z)) & np.uint8(1))
        psi = 0.5 * (psi + (1j ** ph) * sign * psi[y ^ np.uint64(x)])
    return psi


def _magic(t):
    """The sum of the exact decomposition's terms: |H>^t times decompose()'s norm."""
    v = math.cos(math.pi / 8)
    h = np.array([v, math.sin(math.pi / 8)])
    psi = np.ones(1)
    for _ in range(t):
        psi = np.kron(h, psi)
    return psi * 2 ** ((t // 2) / 2) * (2 * v if t % 2 else 1.0)


def _code_state(t, L):
    """Sum over the codewords x of the product of |0> (x_c = 0) and |+> (x_c = 1)."""
    cw = np.zeros(1, dtype=np.uint64)
    for row in L:
        cw = np.concatenate([cw, cw ^ np.uint64(row)])
    amp = np.bincount(cw.astype(np.int64), weights=2.0 ** (-0.5 * np.bitwise_count(cw)), minlength=1 << t)
    for c in range(t):  # amplitude at y: every codeword with ones at all of y's ones
        a = amp.reshape(-1, 2, 1 << c)
        a[:, 0, :] += a[:, 1, :]
    return amp


def _norm2(psi, P):
    return float(abs(np.vdot(psi, _project(psi.astype(complex), P))))


def exact(case, seed):
    kind = case["kind"]
    if kind == "exact" and case["t"] <= 22:
        rs = _rs(case, seed)
        Ps = _projectors(case["n"], case["t"], rs)
        psi = _magic(case["t"]) if case["exact"] else _code_state(case["t"], _code(case["t"], case["k"], rs))
        return [_norm2(psi, P) for P in Ps]
    if kind == "queries" and not case["force"]:
        # the sparsified queries' codes are the backend's own draws: no value for them
        return [[_norm2(_magic(q["cfg"]["t"]), P) for P in q["projs"]] if q["cfg"]["exact"] else [None, None]
                for q in _queries(case, _rs(case, seed))]
    return None  # whole numbers, or estimates on the backend's own random states
