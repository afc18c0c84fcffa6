"""GPU: one-kind single systems whose lists overflow (32 entries an atom): the
shares of a slot take turns on the stencil's candidates.  The same trajectory
as with full lists over 20 steps: 1e-9 A in binary64, 1e-6 A in mixed
precision (the sums group differently)."""
import numpy as np
import pytest

from fmd_gb300 import serve, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L(gpu_lib):
    return serve.bind(gpu_lib.L)


@pytest.fixture(scope="module")
def eam(L):
    return serve.eam_tables(L)


@pytest.mark.parametrize("cells", [5, 16])       # many shares; few or one
@pytest.mark.parametrize("pot", ["lj", "morse", "eam"])
@pytest.mark.parametrize("precision", [serve.PREC_FP64, serve.PREC_MIXED])
def test_overflow_matches_full_lists(L, eam, precision, pot, cells):
    P = serve.POTENTIALS[pot]
    x, v = workloads.fcc_state(cells, cells, cells, P["a"], 300.0, P["mass"], seed=61, disp=0.05)
    l = cells * P["a"]
    x -= l * np.floor(x / l)
    res = []
    for cap in (0, 32):
        one = serve.Single(L, pot, x, v, l, precision=precision, eam=eam, list_capacity=cap)
        one.steps(20)
        xs, vs, Fs, ids = one.state()
        res.append(xs[np.argsort(ids)])
        one.close()
    d = res[0] - res[1]
    d -= l * np.round(d / l)
    assert np.abs(d).max() <= (1e-9 if precision == serve.PREC_FP64 else 1e-6)
