"""The tree sum's kernels (csim_tree.cu) against the pair kernels on the same
draws: every sampled value is an exact sum in Z[w], so they are equal."""
import numpy as np
import pytest

from circuitsimulator_gb300 import backend
from helpers import rand_word, random_projector_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    g = backend.Backend(0)
    g.set_option(backend.OPT_AUTOTUNE, 0)
    yield g
    g.close()


def _values(gpu, kernel, *args):
    try:
        gpu.set_option(backend.OPT_PAIR_KERNEL, kernel)
        return gpu.singleProjectorSample(*args)
    finally:
        gpu.set_option(backend.OPT_PAIR_KERNEL, 0)


def _code(kind, t, k, rs):
    L = [rand_word(rs, t) for _ in range(k)]
    if kind == "repeated":  # rank below k: each codeword several times
        L[1::2] = L[0::2][:len(L[1::2])]
    if kind == "low":  # coordinates that are 0 in every codeword
        L = [v & ((1 << (t // 2)) - 1) for v in L]
    return L


@pytest.mark.parametrize("t,k,count,kind", [
    (1, 0, 3, "random"), (1, 1, 5, "random"), (7, 5, 64, "random"), (8, 8, 33, "random"), (9, 3, 300, "random"),
    (16, 6, 129, "random"), (17, 6, 128, "low"), (23, 11, 500, "random"), (27, 9, 70, "repeated"),
    (32, 12, 40, "random"), (33, 12, 40, "random"), (40, 14, 300, "random"), (47, 8, 31, "low"),
    (56, 13, 20, "random"), (64, 11, 65, "random"), (64, 2, 200, "random"), (64, 0, 9, "random")])
def test_tree_sampler_equals_pair_kernel(gpu, t, k, count, kind):
    rs = np.random.RandomState(17 * t + k)
    L = _code(kind, t, k, rs)
    rows = random_projector_rows(rs, t, max(1, t // 3))
    P = backend.projector(rows[0], rows[1], rows[2], t)
    for rng in (backend.RNG_PHILOX, backend.RNG_LIBC):
        a = _values(gpu, 0, P, L, False, count, rng, 91)
        b = _values(gpu, 2, P, L, False, count, rng, 91)
        assert (a == b).all(), np.nonzero(a != b)[0][:8]


def test_tree_sampler_in_chunks(gpu):
    """More states than the scratch memory takes at once, more than one batch of
    states, and a code change between calls."""
    rs = np.random.RandomState(3)
    rows = random_projector_rows(rs, 40, 12)
    P = backend.projector(rows[0], rows[1], rows[2], 40)
    L = [rand_word(rs, 40) for _ in range(16)]
    a = _values(gpu, 0, P, L, False, 2100, backend.RNG_LIBC, 5)
    b = _values(gpu, 0, P, L[:4], False, 17000, backend.RNG_PHILOX, 5)
    assert (a == _values(gpu, 5, P, L, False, 2100, backend.RNG_LIBC, 5)).all()
    assert (b == _values(gpu, 5, P, L[:4], False, 17000, backend.RNG_PHILOX, 5)).all()


@pytest.mark.parametrize("t,count", [(1, 40), (2, 33), (3, 64), (8, 70), (9, 300), (15, 40), (16, 129), (17, 20), (24, 5)])
def test_tree_sampler_of_magic_state_terms(gpu, t, count):
    rs = np.random.RandomState(40 + t)
    rows = random_projector_rows(rs, t, max(1, t // 3))
    P = backend.projector(rows[0], rows[1], rows[2], t)
    for rng in (backend.RNG_PHILOX, backend.RNG_LIBC):
        a = _values(gpu, 0, P, None, True, count, rng, 12)
        assert (a == _values(gpu, 1, P, None, True, count, rng, 12)).all()


@pytest.mark.parametrize("t,k,kind", [(1, -1, ""), (2, -1, ""), (3, -1, ""), (8, -1, ""), (13, -1, ""), (16, -1, ""),
                                      (1, 1, "random"), (6, 4, "random"), (9, 9, "random"), (17, 6, "random"),
                                      (21, 8, "random"), (33, 7, "random"), (40, 9, "low"), (64, 5, "random"),
                                      (20, 6, "repeated"), (12, 0, "random")])
def test_tree_rows_equal_pair_kernel(gpu, t, k, kind):
    """exactProjector's rows (one term per row left out of the sum, the diagonal apart),
    whole and in ranges."""
    rs = np.random.RandomState(t + 50 * (k + 1))
    L = None if k < 0 else _code(kind, t, k, rs)
    chi = 1 << ((t + 1) // 2 if k < 0 else k)
    rows = random_projector_rows(rs, t, max(1, t // 2))
    P = backend.projector(rows[0], rows[1], rows[2], t)
    out = []
    for kernel in (0, 1):
        try:
            gpu.set_option(backend.OPT_PAIR_KERNEL, kernel)
            re, im = gpu.exactProjectorRows(P, L, k < 0, 0, chi)
            cut = chi // 3
            parts = [gpu.exactProjectorRows(P, L, k < 0, a, b) for a, b in ((0, cut), (cut, chi))]
            st = gpu.last_stats()
            out.append((re, im, gpu.exactProjector(P, L, k < 0, 1.0), st.pairs, st.states_live))
        finally:
            gpu.set_option(backend.OPT_PAIR_KERNEL, 0)
        assert (np.concatenate([p[0] for p in parts]) == re).all()
        assert (np.concatenate([p[1] for p in parts]) == im).all()
    (re0, im0, v0, n0, l0), (re1, im1, v1, n1, l1) = out
    assert (re0 == re1).all() and (im0 == im1).all() and v0 == v1
    assert (n0, l0) == (n1, l1)


def test_inner_product_of_any_symmetric_or_asymmetric_form(gpu, oracle):
    """A J that no state has (asymmetric, or with a diagonal other than D's) takes the steps that keep
    the whole form, as the reference does."""
    rs = np.random.RandomState(11)
    for n in (2, 5, 17, 31, 33, 40, 64):
        a, b = gpu.randomStabilizerState(n, 6, n), gpu.randomStabilizerState(n, 6, n + 1000)
        for i in range(6):
            st = (a, b)[i % 2]
            k = max(1, int(st["k"][i]))
            x, y = (int(v) for v in rs.randint(k, size=2))
            st["J"][i][x] ^= np.uint64(1 << (y if i < 4 else x))
        for i in range(6):
            want = oracle.inner_product(a[i:i + 1], b[i:i + 1])
            got = tuple(int(v[0]) for v in gpu.innerProductExact(a[i:i + 1], b[i:i + 1]))
            assert got == tuple(want), (n, i)


@pytest.mark.parametrize("t,k,kind,count", [(64, 23, "random", 5), (57, 22, "random", 3), (48, 23, "low", 3),
                                            (64, 24, "repeated", 3)])
def test_tree_sampler_in_several_trees(gpu, t, k, kind, count):
    """States of so many terms that each is several trees."""
    rs = np.random.RandomState(t + k)
    rows = random_projector_rows(rs, t, t // 2)
    P = backend.projector(rows[0], rows[1], rows[2], t)
    L = _code(kind, t, k, rs)
    for rng in (backend.RNG_PHILOX, backend.RNG_LIBC):
        a = _values(gpu, 0, P, L, False, count, rng, 19)
        assert a.any()
        assert (a == _values(gpu, 2, P, L, False, count, rng, 19)).all()


def test_batched_queries_in_several_trees(gpu):
    rs = np.random.RandomState(2)
    qs = []
    for i, (t, k, s) in enumerate([(64, 22, 3), (57, 23, 2), (24, 9, 200), (64, 22, 2)]):
        g = random_projector_rows(rs, t, 4)
        cfg = dict(quiet=1, verbose=0, noapprox=0, samples=s, bins=1, t=t, k=k, exact=0, fidbound=1e-5, fidelity=0,
                   rank=0, forceL=0, forceSample=1)
        qs.append({"cfg": cfg, "projs": [(*g, t), (g[0][1:], g[1][1:], g[2][1:], t)], "seed": 5 + i,
                   "rng": backend.RNG_LIBC if i % 2 else backend.RNG_PHILOX})
    for a, b in zip(gpu.run_queries(qs, batched=True), gpu.run_queries(qs, batched=False)):
        assert a["status"] == 0
        assert (a["numerator"], a["denominator"], a["pairs"]) == (b["numerator"], b["denominator"], b["pairs"])


def test_tree_sampler_across_chunks(gpu):
    """Node planes of 4200 states (40 qubits, 2^16 terms) are 4.9 GB, more than the scratch
    takes at once: planes written again for later states, and partial sums from there on."""
    rs = np.random.RandomState(3)
    rows = random_projector_rows(rs, 40, 12)
    P = backend.projector(rows[0], rows[1], rows[2], 40)
    L = [rand_word(rs, 40) for _ in range(16)]
    for rng in (backend.RNG_LIBC, backend.RNG_PHILOX):
        assert (_values(gpu, 0, P, L, False, 4200, rng, 5) == _values(gpu, 5, P, L, False, 4200, rng, 5)).all()


@pytest.mark.parametrize("t,lo", [(48, 0), (40, 1000)])
def test_tree_rows_across_chunks(gpu, t, lo):
    """The rows of 2^14 terms: 9 and 12 GB of node planes."""
    rs = np.random.RandomState(3)
    L = [rand_word(rs, t) for _ in range(14)]
    rows = random_projector_rows(rs, t, 2)
    P = backend.projector(rows[0], rows[1], rows[2], t)
    out = []
    try:
        for kernel in (0, 1):
            gpu.set_option(backend.OPT_PAIR_KERNEL, kernel)
            out.append(gpu.exactProjectorRows(P, L, False, lo, 1 << 14))
    finally:
        gpu.set_option(backend.OPT_PAIR_KERNEL, 0)
    assert out[0][0].any()
    assert (out[0][0] == out[1][0]).all() and (out[0][1] == out[1][1]).all()


@pytest.mark.parametrize("t,count", [(33, 5), (34, 4), (36, 3), (41, 3), (44, 2)])
def test_tree_sampler_of_many_pairs(gpu, t, count):
    """Terms of |H^t> with rows above 32 vertices, where the stages copy them past the registers."""
    rs = np.random.RandomState(t)
    rows = random_projector_rows(rs, t, 3)
    P = backend.projector(rows[0], rows[1], rows[2], t)
    for rng in (backend.RNG_PHILOX, backend.RNG_LIBC):
        a = _values(gpu, 0, P, None, True, count, rng, 12)
        assert a.any() and (a == _values(gpu, 1, P, None, True, count, rng, 12)).all()


def _block(rs, n):
    """n commuting independent Pauli rows (phases, x, z) of a random graph state with random
    local Cliffords, and its state vector."""
    while True:
        adj = np.triu(rs.randint(2, size=(n, n)), 1)
        adj = adj + adj.T
        x, z = [1 << a for a in range(n)], [sum(1 << b for b in range(n) if adj[a][b]) for a in range(n)]
        for q in range(n):
            for _ in range(rs.randint(3)):  # X -> Z -> Y -> X
                for a in range(n):
                    xb, zb = (x[a] >> q) & 1, (z[a] >> q) & 1
                    x[a] ^= (xb ^ (xb ^ zb)) << q
                    z[a] ^= (zb ^ xb) << q
        ph = [(bin(a & b).count("1") & 1) + 2 * int(rs.randint(2)) for a, b in zip(x, z)]
        psi = rs.standard_normal(1 << n) + 1j * rs.standard_normal(1 << n)
        y = np.arange(1 << n)
        for p, a, b in zip(ph, x, z):
            sign = 1.0 - 2.0 * (np.array([bin(v & b).count("1") for v in y]) & 1)
            psi = 0.5 * (psi + 1j ** p * sign * psi[y ^ a])
        if np.linalg.norm(psi) > 1e-6:
            return (ph, x, z), psi / np.linalg.norm(psi)


@pytest.mark.parametrize("t", [16, 33, 42, 49, 57, 60])
def test_tree_sampler_of_pairs_in_closed_form(gpu, t):
    """A projector onto one state, a product of states of six qubits: a sample is 0 or
    2^t 2^-c |sum|^2, the sum over all 2^(t/2) terms of |H^t> a product of the blocks' sums.
    Up to 2^30 terms and rows of 60 vertices, beyond what a pair kernel can check."""
    rs = np.random.RandomState(t)
    pair = 0.5 * np.array([1, 1, 1, -1]) + np.array([1, 0, 0, 1]) / np.sqrt(2)  # CZ|++> and (|00> + |11>) / sqrt2
    one = np.array([1, 1]) / np.sqrt(2) + np.array([1, 0])                      # |+> and |0>
    ph, xs, zs, amp, q = [], [], [], 1.0, 0
    while q < t:
        n = min(6, t - q)
        terms = np.ones(1)
        for i in range(0, n - 1, 2):
            terms = np.kron(pair, terms)
        if n % 2:
            terms = np.kron(one, terms)
        s = 0.0
        while abs(s) < 1e-9:
            rows, psi = _block(rs, n)
            s = np.vdot(psi, terms)
        amp *= abs(s) ** 2
        ph += rows[0]
        xs += [v << q for v in rows[1]]
        zs += [v << q for v in rows[2]]
        q += n
    P = backend.projector(ph, xs, zs, t)
    vals = gpu.singleProjectorSample(P, None, True, 12, backend.RNG_PHILOX, 1)
    assert vals.any()
    for v in vals[vals != 0]:
        c = t - np.log2(v / amp)
        assert abs(c - round(c)) < 1e-9 and 0 <= round(c) <= t, (v, amp, c)
