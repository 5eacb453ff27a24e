"""The tree sum over all terms of |L> (csim_tree.cuh, csim_tree_plan.h),
compiled for the host, against the oracle: the exact Z[w] coordinates of
sum_j <theta|phi_j> are whole numbers, so they are equal, not close."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from helpers import phase_m, rand_word, random_projector_rows

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "tree_host_check.cpp")
SO = os.path.join(HERE, "native", "_build", "libtreehost.so")
CSRC = os.path.join(os.path.dirname(HERE), "circuitsimulator_gb300", "csrc")
DEPS = [SRC] + [os.path.join(CSRC, f) for f in ("csim_tree.cuh", "csim_tree_plan.h", "csim_pair_core.cuh")]


@pytest.fixture(scope="module")
def tree_sums():
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    if not os.path.exists(SO) or os.path.getmtime(SO) < max(os.path.getmtime(f) for f in DEPS):
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", SRC, "-o", SO])
    lib = C.CDLL(SO)
    lib.tree_host_sums.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_int64, C.c_void_p, C.c_void_p]

    def run(thetas, L, t, count):
        thetas = np.ascontiguousarray(thetas)
        k = 0 if L is None else len(L)
        Lw = None if L is None else np.array([int(x) for x in L] or [0], dtype=np.uint64)
        out = np.zeros((len(thetas), 4, 2), dtype=np.uint64)
        info = np.zeros(80, dtype=np.int32)
        assert lib.tree_host_sums(thetas.ctypes.data, len(thetas), None if L is None else Lw.ctypes.data, k, t, count,
                                  out.ctypes.data,
                                  info.ctypes.data) == 0
        vals = [[(int(w[0]) | (int(w[1]) << 64)) - ((1 << 128) if int(w[1]) >> 63 else 0) for w in row] for row in out]
        return vals, info

    return run


def _exact_sum(eps, p, m, P):
    """sum of eps 2^{p/2} w^m as Z[w] coordinates scaled by 2^{P/2}."""
    z = [0, 0, 0, 0]
    for e, pp, mm in zip(eps.tolist(), p.tolist(), m.tolist()):
        if not e:
            continue
        q, mm = pp + P, mm % 8
        terms = [(mm, 1 << (q // 2))] if q % 2 == 0 else [((mm + 1) % 8, 1 << (q // 2)), ((mm + 7) % 8, 1 << (q // 2))]
        for k, c in terms:
            z[k & 3] += -c if k >= 4 else c
    return z


def _thetas(oracle, rs, t, rows, count):
    r = oracle.rng(1000 + t)
    out = []
    for _ in range(20 * count):
        s = oracle.random_state(t, r)
        pf = 1.0
        for q in range(len(rows[0])):
            pf *= oracle.measure_pauli(s, phase_m(rows[0][q]), rows[2][q], rows[1][q])
            if pf == 0:
                break
        if pf:
            out.append(s[0])
        if len(out) == count:
            break
    return np.array(out)


def _check(tree_sums, oracle, t, L, thetas):
    k = 0 if L is None else len(L)
    got, info = tree_sums(thetas, L, t, 4096)
    assert tree_sums(thetas, L, t, 1)[0] == got  # fewer levels for a single state
    Lw = np.array([int(x) for x in L or [0]] or [0], dtype=np.uint64)
    chi = 2 ** ((t + 1) // 2) if L is None else 2 ** k
    for a in range(len(thetas)):
        e, p, m = oracle.term_products(t, int(L is None), Lw, k, thetas[a:a + 1], 0, chi, threads=4)
        assert got[a] == _exact_sum(e, p, m, 2 * t), (t, k, a)
    return info


@pytest.mark.parametrize("t,k", [(1, 0), (1, 1), (2, 2), (5, 2), (7, 5), (8, 8), (15, 4), (16, 7), (17, 6), (24, 10),
                                 (31, 8), (32, 7), (33, 8), (40, 9), (48, 8), (57, 7), (63, 6), (64, 7)])
@pytest.mark.parametrize("frac", [0.0, 0.3, 0.8])
def test_tree_sum_equals_oracle(tree_sums, oracle, t, k, frac):
    """Random codes and projected states (few to many non-pivot coordinates)."""
    rs = np.random.RandomState(100 * t + k)
    L = [rand_word(rs, t) for _ in range(k)]
    rows = random_projector_rows(rs, t, int(frac * t))
    thetas = _thetas(oracle, rs, t, rows, 3)
    assert len(thetas)
    _check(tree_sums, oracle, t, L, thetas)


@pytest.mark.parametrize("t", [1, 2, 3, 4, 7, 8, 12, 15, 16, 17, 18, 21])
@pytest.mark.parametrize("frac", [0.0, 0.5])
def test_tree_sum_of_magic_state_terms(tree_sums, oracle, t, frac):
    """Terms of |H^t>, products of two-qubit states (a single qubit left over for odd t)."""
    rs = np.random.RandomState(t)
    thetas = _thetas(oracle, rs, t, random_projector_rows(rs, t, int(frac * t)), 6)
    _check(tree_sums, oracle, t, None, thetas)


@pytest.mark.parametrize("t", [36])
def test_tree_sum_of_many_pairs(tree_sums, oracle, t):
    """Wide rows: 2^18 terms of |H^36> sum to <theta|H^36> for theta a product state,
    known in closed form: theta = |0>^36 meets the first kind in 1/2 and the second
    in 1/sqrt2 per pair, |+>^36 both kinds in 1/2 and 1/sqrt2 as well."""
    s = oracle.state(t)
    for plus in (True, False):
        st = s.copy()
        if not plus:
            for q in range(t):
                oracle.shrink(st, 1 << q, 0)
        got, _ = tree_sums(st, None, t, 1)
        # <0|a> = 1/2, <0|b> = 1/sqrt2 and <++|a> = 1/2, <++|b> = 1/sqrt2: (1/2 + 1/sqrt2)^18, scaled by 2^36
        z = [1, 0, 0, 0]
        for _ in range(t // 2):  # times 4 (1/2 + 1/sqrt2) = 2 + 2 sqrt2, sqrt2 = w - w^3
            r = [z[1] - z[3], z[0] + z[2], z[1] + z[3], z[2] - z[0]]
            z = [2 * a + 2 * b for a, b in zip(z, r)]
        assert got[0] == z


@pytest.mark.parametrize("t", [6, 16, 20, 33, 64])
def test_tree_sum_of_unusual_codes(tree_sums, oracle, t):
    """No rows; a zero row; repeated rows (each codeword several times); rows
    that leave coordinates 0 in every codeword; unit vectors; the all-ones word."""
    rs = np.random.RandomState(t)
    full = (1 << t) - 1
    a, b = rand_word(rs, t), rand_word(rs, t)
    low = full >> (t // 2)
    codes = [[], [0], [full], [a, a, b, a ^ b, 0], [a & low, b & low, rand_word(rs, t) & low],
             [1 << i for i in range(0, t, max(1, t // 6))], [full, 1 << (t - 1), 3 & full]]
    thetas = _thetas(oracle, rs, t, random_projector_rows(rs, t, t // 3), 4)
    ranks = [int(_check(tree_sums, oracle, t, L, thetas)[0]) for L in codes]
    assert ranks[:4] == [0, 0, 1, 2]


def test_tree_sum_on_extreme_states(tree_sums, oracle):
    """States of every dimension k = 0..n of the affine space, and D, J of one kind only."""
    rs = np.random.RandomState(8)
    for t in (12, 20, 40):
        r = oracle.rng(t)
        base = oracle.random_state(t, r)
        while int(base[0]["k"]) < t - 1:
            base = oracle.random_state(t, r)
        L = [rand_word(rs, t) for _ in range(7)]
        states = [base[0].copy()]
        s = base.copy()
        for q in range(t):
            oracle.shrink(s, 1 << q, int(rs.randint(2)))
            states.append(s[0].copy())
        for zero in ("D1", "D2", "J"):
            w = base[0].copy()
            w[zero] = 0
            if zero in ("D1", "J"):  # J's diagonal is D1
                w["D1"] = 0
                for x in range(int(w["k"])):
                    w["J"][x] = int(w["J"][x]) & ~(1 << x)
            states.append(w)
        _check(tree_sums, oracle, t, L, np.array(states))


@pytest.mark.parametrize("t,k,count", [(40, 16, 4096), (57, 18, 256), (24, 8, 60), (64, 18, 1)])
@pytest.mark.parametrize("room", [1 << 40, 1 << 32, (1 << 30) + 4096, 100 << 20, 1 << 20])
def test_scratch_of_the_memory_there_is(t, k, count, room):
    """Chunks fit the memory that the allocator finds, in quarters of the largest budget
    down to the smallest; then a run of more than one state fails, as one state's planes do."""
    src, so = os.path.join(HERE, "native", "tree_layout_check.cpp"), os.path.join(HERE, "native", "_build", "liblayout.so")
    os.makedirs(os.path.dirname(so), exist_ok=True)
    deps = [src] + [os.path.join(CSRC, f) for f in ("csim_tree.h", "csim_tree_host.h", "csim_tree.cuh", "csim_tree_plan.h")]
    if not os.path.exists(so) or os.path.getmtime(so) < max(os.path.getmtime(f) for f in deps):
        subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I/usr/local/cuda/include", src, "-o", so])
    lib = C.CDLL(so)
    rs = np.random.RandomState(t)
    L = np.array([int(rand_word(rs, t)) for _ in range(k)], dtype=np.uint64)
    out = np.zeros(5, dtype=np.int64)
    lib.tree_layout(C.c_void_p(L.ctypes.data), k, t, C.c_int64(count), C.c_int64(room), C.c_void_p(out.ctypes.data))
    status, used, tried, first, per = out.tolist()
    budget = (4 << 30) >> (2 * (tried - 1))
    assert 1 <= tried <= 4 and budget >= 64 << 20
    assert used <= max(budget, per) + 1024 and first == min(count, max(1, -(-count // max(1, -(-count // max(1, budget // per))))))
    assert (status == 0) == (used <= room)
    assert status == 0 or budget == 64 << 20


def _native(name, headers):
    src, so = os.path.join(HERE, "native", name + ".cpp"), os.path.join(HERE, "native", "_build", "lib%s.so" % name)
    os.makedirs(os.path.dirname(so), exist_ok=True)
    deps = [src] + [os.path.join(CSRC, f) for f in headers]
    if not os.path.exists(so) or os.path.getmtime(so) < max(os.path.getmtime(f) for f in deps):
        subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I/usr/local/cuda/include", src, "-o", so])
    return C.CDLL(so)


@pytest.mark.parametrize("t,k,count", [(64, 30, 3), (64, 26, 5), (64, 22, 40), (57, 24, 7), (48, 30, 2), (60, -1, 2),
                                       (40, 16, 4096), (24, 8, 60), (9, 3, 5), (64, 0, 3)])
@pytest.mark.parametrize("room", [1 << 40, (1 << 30) + 4096, 65 << 20])
@pytest.mark.parametrize("rows", [0, 1])
def test_any_tree_fits_the_smallest_scratch(t, k, count, room, rows):
    """Node planes of up to 2^30 terms: a state of many terms is several trees, so the
    smallest scratch will do; every tree is made once, every partial sum written once,
    no launch writes what another one still reads or beyond the scratch, and rows'
    leaves know the number of their first node."""
    lib = _native("tree_jobs_check", ("csim_tree.h", "csim_tree_host.h", "csim_tree.cuh", "csim_tree_plan.h"))
    rs = np.random.RandomState(t + k)
    L = np.array([int(rand_word(rs, t)) for _ in range(max(k, 1))], dtype=np.uint64)
    out = np.zeros(7, dtype=np.int64)
    lib.tree_jobs(C.c_void_p(L.ctypes.data if k >= 0 else None), max(k, 0), t, C.c_int64(count), C.c_int64(room), rows,
                  C.c_void_p(out.ctypes.data))
    status, used, jobs, violations, trees, written, parts = out.tolist()
    assert status == 0 and used <= room
    assert violations == 0 and written == parts
    assert (trees > 1) == (k > 21 or k < 0)
    assert jobs <= 12 * (1 + 2 * trees * count * (64 << 20) // min(room, 4 << 30))
