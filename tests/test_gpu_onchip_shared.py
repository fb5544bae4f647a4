"""On-chip solves of several contexts at once: every solve is one cooperative launch
whose blocks wait for one another and that wants the whole chip, so two of them may
only follow each other.  Each thread drives a context of its own (a stream of its
own); the answers are those of the same calls made alone, bit for bit."""
import threading

import numpy as np
import pytest

from helpers import opts

pytestmark = pytest.mark.gpu

# (one block to an SM and every SM needed; a few SMs each)
PAIRS = [(("fp64", 1000, 1000), ("fp64", 1000, 1000)), (("fp64", 1000, 1000), ("mixed", 1000, 600)),
         (("mixed", 1000, 600), ("mixed", 1000, 600)), (("fp64", 128, 64), ("fp64", 1000, 1000)),
         (("fp64", 128, 64), ("mixed", 256, 100))]


def _run(precision, nx, ny, seed, calls, start=None):
    from cajitafluids_gb300 import Context
    rng = np.random.default_rng(seed)
    out = []
    with Context(nx, ny, hi=(1.0, ny * (1.0 / nx)), precision=precision) as c:
        c.set_density(0.3)
        c.project(0.01, opts(max_iter=1))  # (graphs are built here)
        u = rng.standard_normal(c.owned_shape("u"))
        v = rng.standard_normal(c.owned_shape("v"))
        u[:, 0] = u[:, -1] = 0.0
        v[0] = v[-1] = 0.0
        if start is not None:
            start.wait(60)
        for _ in range(calls):
            c.upload("u", u)
            c.upload("v", v)
            st = c.project(0.01, opts(tol=1e-12, max_iter=400, precon="Diagonal"))
            out.append((st, c.download("u"), c.download("v")))
    return out


@pytest.mark.parametrize("a,b", PAIRS)
def test_two_contexts_at_once(built, a, b):
    calls = 6
    alone = [_run(*a, 1, 1)[0], _run(*b, 2, 1)[0]]
    start, got, errors = threading.Barrier(2), [None, None], []

    def work(k, case):
        try:
            got[k] = _run(*case, 1 + k, calls, start)
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k, c)) for k, c in enumerate((a, b))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(240)
    assert not errors, errors
    for k in (0, 1):
        assert len(got[k]) == calls
        for st, u, v in got[k]:
            assert st == alone[k][0]
            assert np.array_equal(u, alone[k][1]) and np.array_equal(v, alone[k][2])
