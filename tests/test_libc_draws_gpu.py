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
