"""The C library's draws on the device (csim_rand.cu): the states' places in the
generator's sequence are the same however many states a call draws."""
import numpy as np
import pytest

from circuitsimulator_gb300 import backend
from helpers import rand_word, random_projector_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    g = backend.Backend(0)
    yield g
    g.close()


# few words are made on the host, more on the device (a batch is 2^14 states); with few qubits
# many vectors are drawn again
@pytest.mark.parametrize("t,count", [(1, 700), (2, 513), (3, 3000), (5, 17000), (8, 512), (9, 1100), (31, 1500), (33, 600),
                                     (64, 1300)])
def test_draws_of_one_call_equal_those_of_several(gpu, t, count):
    rs = np.random.RandomState(t)
    rows = random_projector_rows(rs, t, max(1, t // 3))
    P = backend.projector(rows[0], rows[1], rows[2], t)
    L = [rand_word(rs, t) for _ in range(2)]
    whole = gpu.singleProjectorSample(P, L, False, count, backend.RNG_LIBC, 77)
    after = gpu.singleProjectorSample(P, L, False, 3, backend.RNG_LIBC)
    parts, left = [], count
    for i, n in enumerate([1, 2, 509, 1, 20, 513] * 40):
        n = min(n, left)
        if not n:
            break
        parts.append(gpu.singleProjectorSample(P, L, False, n, backend.RNG_LIBC, *([77] if i == 0 else [])))
        left -= n
    assert (np.concatenate(parts) == whole).all()
    assert (gpu.singleProjectorSample(P, L, False, 3, backend.RNG_LIBC) == after).all()


@pytest.mark.parametrize("count", [1, 5, 16, 17])
def test_batched_draws_on_the_device_equal_the_hosts(gpu, count):
    """Queries whose states all fit a round have their words made on the device (sixteen
    queries to a launch); in rounds of a few states the host draws them."""
    rs = np.random.RandomState(count)
    qs = []
    for i in range(count):
        t = int(rs.choice([5, 9, 17, 24, 33, 47, 64]))
        g = random_projector_rows(rs, t, int(rs.randint(2, 6)))
        h = (g[0][1:], g[1][1:], g[2][1:])
        cfg = dict(quiet=1, verbose=0, noapprox=0, samples=int(rs.choice([60, 300, 600])), bins=1, t=t, k=3, exact=0,
                   fidbound=1e-5, fidelity=0, rank=0, forceL=0, forceSample=1)
        qs.append({"cfg": cfg, "projs": [(*g, t), (*h, t)], "seed": 50 + i, "rng": backend.RNG_LIBC})
    batched = gpu.run_queries(qs, batched=True)
    plain = gpu.run_queries(qs, batched=False)
    srv = backend.Server(0, round_pairs=8 * 40)
    try:
        tickets = [srv.submit(q) for q in qs]
        rounds = [srv.wait(t) for t in tickets]
    finally:
        srv.close()
    for b, p, r in zip(batched, plain, rounds):
        assert b["numerator"] == p["numerator"] == r["numerator"]
        assert b["denominator"] == p["denominator"] == r["denominator"]


def test_the_most_draws_of_a_round(gpu):
    """2^16 states of 64 qubits, 1.3e8 words of one stream."""
    rs = np.random.RandomState(64)
    g = random_projector_rows(rs, 64, 3)
    cfg = dict(quiet=1, verbose=0, noapprox=0, samples=32768, bins=1, t=64, k=1, exact=0, fidbound=1e-5, fidelity=0,
               rank=0, forceL=0, forceSample=1)
    q = {"cfg": cfg, "projs": [(*g, 64), (g[0][1:], g[1][1:], g[2][1:], 64)], "seed": 9, "rng": backend.RNG_LIBC}
    b, p = gpu.run_queries([q], batched=True)[0], gpu.run_queries([q], batched=False)[0]
    assert b["numerator"] == p["numerator"] and b["denominator"] == p["denominator"]


# percent of the words that a batch needs: none of its states but the first have any; some; all but a few
@pytest.mark.parametrize("percent", [1, 60, 96])
@pytest.mark.parametrize("t,count,kernel", [(3, 3000, 0), (40, 700, 0), (64, 17000, 0), (24, 900, 5)])
def test_states_that_run_out_of_words(gpu, percent, t, count, kernel):
    """A batch whose words run out on the device is drawn again with the host's: the same
    values, and the stream goes on behind them."""
    rs = np.random.RandomState(t)
    rows = random_projector_rows(rs, t, max(1, t // 3))
    P = backend.projector(rows[0], rows[1], rows[2], t)
    L = [rand_word(rs, t) for _ in range(2)]
    out = []
    try:
        gpu.set_option(backend.OPT_PAIR_KERNEL, kernel)
        gpu.singleProjectorSample(P, L, False, 1, backend.RNG_PHILOX, 1)  # a pair kernel is tuned
        for p in (100, percent):
            gpu.set_option(backend.OPT_DRAW_WORDS, p)
            n0 = gpu.launches
            a = gpu.singleProjectorSample(P, L, False, count, backend.RNG_LIBC, 7)
            n1 = gpu.launches
            out.append((a, gpu.singleProjectorSample(P, L, False, count, backend.RNG_LIBC), n1 - n0))
    finally:
        gpu.set_option(backend.OPT_PAIR_KERNEL, 0)
        gpu.set_option(backend.OPT_DRAW_WORDS, 100)
    assert (out[0][0] == out[1][0]).all() and (out[0][1] == out[1][1]).all()
    if percent < 90:
        assert out[1][2] > out[0][2]  # it did run out


@pytest.mark.parametrize("percent", [1, 60, 97])
def test_a_query_out_of_words_leaves_the_others_alone(gpu, percent):
    """Queries of one round: those whose words run out on the device get their states
    in another round, with the host's words; all have their usual results."""
    rs = np.random.RandomState(percent)
    qs = []
    for i in range(12):
        t = int(rs.choice([5, 9, 24, 33, 64]))
        g = random_projector_rows(rs, t, 4)
        cfg = dict(quiet=1, verbose=0, noapprox=0, samples=400, bins=1, t=t, k=3, exact=0, fidbound=1e-5, fidelity=0,
                   rank=0, forceL=0, forceSample=1)
        if i % 4 == 3:
            cfg.update(noapprox=1, forceSample=0, samples=1000)
        qs.append({"cfg": cfg, "projs": [(*g, t), (g[0][1:], g[1][1:], g[2][1:], t)], "seed": 50 + i,
                   "rng": backend.RNG_LIBC if i % 3 else backend.RNG_PHILOX})
    want = gpu.run_queries(qs, batched=True)
    plain = gpu.run_queries(qs, batched=False)
    try:
        gpu.set_option(backend.OPT_DRAW_WORDS, percent)
        got = gpu.run_queries(qs, batched=True)
    finally:
        gpu.set_option(backend.OPT_DRAW_WORDS, 100)
    for a, b, c in zip(want, got, plain):
        assert b["status"] == 0
        assert (a["numerator"], a["denominator"], a["pairs"]) == (b["numerator"], b["denominator"], b["pairs"])
        assert (a["numerator"], a["denominator"]) == (c["numerator"], c["denominator"])
