"""Calls on a device whose memory other programs hold: they say so, and the calls
behind them are not affected."""
import contextlib

import numpy as np
import pytest

from circuitsimulator_gb300 import backend
from helpers import rand_word, random_projector_rows

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _free():
    return torch.cuda.mem_get_info(0)[0]


@contextlib.contextmanager
def full_device(leave):
    """`leave` bytes of device memory are free, the others taken."""
    held = torch.empty(max(0, _free() - leave), dtype=torch.uint8, device="cuda:0")
    try:
        assert _free() < leave + (32 << 20)
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def _problem(t, k, seed=0):
    rs = np.random.RandomState(100 * t + k + seed)
    rows = random_projector_rows(rs, t, t // 3)
    return backend.projector(rows[0], rows[1], rows[2], t), [rand_word(rs, t) for _ in range(k)]


@pytest.mark.parametrize("rng", [backend.RNG_PHILOX, backend.RNG_LIBC])
def test_a_call_after_one_without_memory(rng):
    gpu = backend.Backend(0)
    try:
        P, L = _problem(64, 10)
        small = gpu.singleProjectorSample(P, L, False, 40, rng, 5)  # (its kernels are loaded)
        large = _problem(64, 20)  # 50 MB of node planes for a state
        with full_device(16 << 20):
            with pytest.raises(backend.CsimError) as e:
                gpu.singleProjectorSample(*large, False, 64, backend.RNG_PHILOX, 5)
            assert e.value.code == -4, e.value  # CSIM_ERR_NOMEM
            again = gpu.singleProjectorSample(P, L, False, 40, rng, 5)
        assert (again == small).all()
    finally:
        gpu.close()


def _query(t, k, samples, seed=1):
    rs = np.random.RandomState(t)
    g = random_projector_rows(rs, t, 6)
    cfg = dict(quiet=1, verbose=0, noapprox=0, samples=samples, bins=1, t=t, k=k, exact=0, fidbound=1e-5, fidelity=0,
               rank=0, forceL=0, forceSample=1)
    return {"cfg": cfg, "projs": [(*g, t), (g[0][1:], g[1][1:], g[2][1:], t)], "seed": seed, "rng": backend.RNG_PHILOX}


def test_scratch_of_a_context():
    """One scratch of 4 GB at most for the samplers and the query engine: 4096 states of
    2^16 terms on 40 qubits take 5.3 GB of node planes at once."""
    backend.Backend(0).close()
    warm = backend.Backend(0)  # (the kernels' own memory)
    warm.run_queries([_query(40, 16, 100)], batched=True)
    warm.close()
    before = _free()
    gpu = backend.Backend(0)
    try:
        P, L = _problem(40, 16)
        gpu.singleProjectorSample(P, L, False, 4096, backend.RNG_PHILOX, 5)
        one = before - _free()
        gpu.run_queries([_query(40, 16, 2048), _query(40, 15, 4096)], batched=True)
        both = before - _free()
        assert 4 << 30 > one > 2 << 30 and both < (4 << 30) + (200 << 20), (one, both)
    finally:
        gpu.close()


@pytest.mark.parametrize("budget", [1 << 30, 16 << 20])
def test_scratch_of_a_server(budget):
    """Node planes take half of the memory budget at most, or 64 MB."""
    gpu = backend.Backend(0)
    q = _query(40, 16, 3000)
    want = gpu.run_queries([q], batched=True)[0]
    gpu.close()
    before = _free()
    srv = backend.Server(0, hbm_budget_bytes=budget, round_pairs=1 << 29)
    try:
        tickets = [srv.submit(q) for _ in range(3)]
        got = [srv.wait(t) for t in tickets]
        held = before - _free()
    finally:
        srv.close()
    assert all((r["numerator"], r["denominator"]) == (want["numerator"], want["denominator"]) for r in got)
    assert held < max(budget // 2, 64 << 20) + (150 << 20), held


def _words_query(t, samples, rng):
    q = _query(t, 4, samples, seed=3)
    q["rng"] = rng
    return q


def test_a_round_without_memory_fails_its_queries_only():
    """A query whose round finds no memory fails; the server and the queries behind it go on."""
    small = _words_query(64, 700, backend.RNG_LIBC)
    gpu = backend.Backend(0)
    want = gpu.run_queries([small], batched=True)[0]
    gpu.close()
    srv = backend.Server(0)
    try:
        first = srv.wait(srv.submit(small))
        with full_device(64 << 20):
            big = srv.wait(srv.submit(_words_query(64, 20000, backend.RNG_LIBC)))
            again = srv.wait(srv.submit(small))
        after = srv.wait(srv.submit(_words_query(64, 20000, backend.RNG_LIBC)))
        for r in (first, again):
            assert (r["status"], r["numerator"], r["denominator"]) == (0, want["numerator"], want["denominator"])
        assert big["status"] == -4 and after["status"] == 0
    finally:
        srv.close()


@pytest.mark.parametrize("t,k,count,rng,leave", [(64, 6, 20000, backend.RNG_LIBC, 100), (40, 16, 2000, backend.RNG_LIBC, 90),
                                                 (57, 17, 300, backend.RNG_PHILOX, 90), (12, -1, 20000, backend.RNG_LIBC, 12)])
def test_a_sampler_in_the_memory_there_is(t, k, count, rng, leave):
    """Batches of fewer states where a batch of 2^14 finds no memory: the same values, and
    the streams go on behind them."""
    gpu = backend.Backend(0)
    try:
        P, L = _problem(t, max(k, 1))
        L = None if k < 0 else L
        want = gpu.singleProjectorSample(P, L, k < 0, count, rng, 5)
        more = gpu.singleProjectorSample(P, L, k < 0, 100, rng)
        gpu.close()
        gpu = backend.Backend(0)
        with full_device(leave << 20):
            got = gpu.singleProjectorSample(P, L, k < 0, count, rng, 5)
            assert gpu.last_stats().states == count
            assert (gpu.singleProjectorSample(P, L, k < 0, 100, rng) == more).all()
        assert (got == want).all()
    finally:
        gpu.close()
