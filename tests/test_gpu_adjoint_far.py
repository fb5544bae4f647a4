"""A trace of more than a cell fails the backward call as such, also when the
pressure solves of the meaningless adjoints that follow it fail (here by a NaN in the
seed)."""
import numpy as np
import pytest

from cajitafluids_gb300 import CfError, Context
from cajitafluids_gb300 import _lib as L
from helpers import opts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("precon", ["Diagonal", "PFMG"])
@pytest.mark.parametrize("graphs", [True, False])
def test_far_trace_is_reported_before_failed_solves(built, precision, precon, graphs):
    n = 32
    rng = np.random.default_rng(3)
    with Context(n, n, periodic=(True, True), precision=precision) as c:
        c.set_quirks(L.CF_FIX_Q1)
        c.set_graphs(graphs)
        for f in ("u", "v"):
            c.upload(f, rng.standard_normal((n, n)))
        c.upload("q", rng.uniform(0.0, 1.0, (n, n)))
        # (the last step's adjoint projection sees zero velocities; its traces are far)
        c.forward_checkpointed(3, 2, 2.0 / n, 3, opts(tol=1e-8, max_iter=3000, precon=precon))
        seed = rng.standard_normal((n, n))
        seed[5, 7] = np.nan
        with pytest.raises(CfError) as e:
            c.backward(seed)
        assert e.value.code == L.CF_ERR_UNSUPPORTED
        assert "trace" in str(e.value)
