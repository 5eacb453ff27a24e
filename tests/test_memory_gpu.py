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
        small = gpu.singleProjectorSample(P, L, False, 600, rng, 5)  # (its kernels are loaded)
        with full_device(128 << 20):
            with pytest.raises(backend.CsimError) as e:
                gpu.singleProjectorSample(P, L, False, 1 << 14, backend.RNG_LIBC, 5)
            assert e.value.code == -4, e.value  # CSIM_ERR_NOMEM
            again = gpu.singleProjectorSample(P, L, False, 600, rng, 5)
        assert (again == small).all()
    finally:
        gpu.close()
