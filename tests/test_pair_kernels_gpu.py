"""The pair kernels that the samplers run when one is asked for: their tuner and the
block-prefix kernel's ordered codewords."""
import subprocess
import sys

import numpy as np
import pytest

from circuitsimulator_gb300 import backend
from helpers import rand_word, random_projector_rows

pytestmark = pytest.mark.gpu


def _problem(t, k):
    rs = np.random.RandomState(t)
    rows = random_projector_rows(rs, t, max(2, t // 3))
    return backend.projector(rows[0], rows[1], rows[2], t), [rand_word(rs, t) for _ in range(k)]


def streams():
    """Run in a process of its own, whose table of tuned launches is empty."""
    a, b = backend.Backend(0), backend.Backend(0)
    b.set_option(backend.OPT_AUTOTUNE, 0)
    for rng in (backend.RNG_LIBC, backend.RNG_PHILOX):
        t0 = 20 if rng == backend.RNG_LIBC else 36
        out = []
        for g in (a, b):
            g.set_option(backend.OPT_PAIR_KERNEL, 5)
            vals, n = [], []
            # two t buckets, both tuned on their first use, then an explicit tuning in mid-stream
            for t, seed in ((t0, 5), (t0 + 4, backend.SEED_CONTINUE), (t0, backend.SEED_CONTINUE)):
                n0 = g.launches
                vals.append(g.singleProjectorSample(*_problem(t, 9), False, 40, rng, seed))
                n.append(g.launches - n0)
            st = g.last_stats()
            if g is a:
                g.autotune(t0 + 8)
                assert (g.last_stats().pairs, g.last_stats().states) == (st.pairs, st.states)
            vals.append(g.singleProjectorSample(*_problem(t0, 9), False, 40, rng, backend.SEED_CONTINUE))
            out.append((np.concatenate(vals), n))
        (va, na), (vb, nb) = out
        assert (va == vb).all()
        assert na[0] > 2 * nb[0] and na[1] > 2 * nb[1] and na[2] <= nb[2] + 4, (na, nb)
    print("ok")


def test_tuning_leaves_the_streams_where_they_are():
    """Contexts that tune and that do not give the same values, with each generator's stream
    continued across calls that tune."""
    code = "import sys; sys.path[:0] = %r; import test_pair_kernels_gpu as m; m.streams()" % (sys.path,)
    r = subprocess.run([sys.executable, "-c", code], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, timeout=600)
    assert r.returncode == 0 and r.stdout.decode().split()[-1] == "ok", r.stdout.decode()[-2000:]


@pytest.mark.parametrize("t,k,low", [(24, 13, 8), (40, 14, 24), (64, 13, 30)])
def test_shared_prefix_codes_through_every_kernel(t, k, low):
    """Codes whose rows but two leave the top bits alone, so that long runs of the ordered
    codewords agree on them: the tree, the block-prefix and the direct kernel."""
    gpu = backend.Backend(0)
    try:
        rs = np.random.RandomState(3000 + t)
        L = [rand_word(rs, t) & (-1 if r < 2 else (1 << low) - 1) for r in range(k)]
        rows = random_projector_rows(rs, t, max(1, t // 5))
        P = backend.projector(rows[0], rows[1], rows[2], t)
        out = []
        for kernel in (0, 1, 2, 3, 4, 5):
            gpu.set_option(backend.OPT_PAIR_KERNEL, kernel)
            out.append(gpu.singleProjectorSample(P, L, False, 30, backend.RNG_PHILOX, 17))
        assert out[0].any()
        for v in out[1:]:
            assert (v == out[0]).all()
    finally:
        gpu.close()
