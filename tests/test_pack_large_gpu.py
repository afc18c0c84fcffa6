"""Large packed systems, whose cells are refreshed by grid kernels instead of
one cluster each: the trajectory of the single-system path (binary64 positions
within 1e-9 A and forces within 1e-9 of max |F|, the bounds of the packs'
other comparisons), with list rebuilds on the way, in packs of their own
beside smaller jobs of the same potential."""
import numpy as np
import pytest

from fmd_gb300 import serve

pytestmark = pytest.mark.gpu
STEPS = 48


@pytest.fixture(scope="module")
def L(gpu_lib):
    return serve.bind(gpu_lib.L)


@pytest.fixture(scope="module")
def eam(L):
    return serve.eam_tables(L)


def _by_id(state):
    x, v, F, ids = state
    o = np.argsort(ids)
    return x[o], v[o], F[o]


def _served(L, eam, pot, cells):
    """kernels a step and the final states of jobs of cells^3 unit cells"""
    srv = serve.Server(L, chunk_steps=16, eam=eam)
    srv.set_tuning(128)
    ids, sizes = [], []
    for k, c in enumerate(cells):
        x, v, l = serve.job_atoms(dict(pot=pot, ncell=c, T=900.0, seed=40 + k))
        ids.append(srv.submit(pot, x, v, l, STEPS, precision=serve.PREC_FP64, keep_state=True))
        sizes.append(len(x))
    srv.drain()
    per_step = srv.stats().kernels / STEPS
    out = []
    for j, n in zip(ids, sizes):
        r = srv.result(j)
        assert r.state == 2 and r.errbits == 0
        out.append(_by_id(srv.state(j, n)))
    srv.close()
    return per_step, out


@pytest.mark.parametrize("pot", ["lj", "morse", "eam"])
def test_large_members_match_single(L, eam, pot):
    # 70 304 and 78 732 atoms, and one of 32 000
    cells = (26, 20, 27)
    _, got = _served(L, eam, pot, cells)
    for k, c in enumerate(cells):
        x, v, l = serve.job_atoms(dict(pot=pot, ncell=c, T=900.0, seed=40 + k))
        one = serve.Single(L, pot, x, v, l, precision=serve.PREC_FP64, eam=eam)
        one.steps(STEPS)
        xs, vs, Fs = _by_id(one.state())
        one.close()
        xp, vp, Fp = got[k]
        box = np.broadcast_to(np.asarray(l, float), (3,))
        dx = np.abs(xp - xs)
        dx = np.minimum(dx, np.abs(dx - box))       # (an atom at a periodic face)
        assert dx.max() <= 1e-9, dx.max()
        assert np.abs(Fp - Fs).max() <= 1e-9 * np.abs(Fs).max()


def test_which_kernels_refresh(L, eam):
    """start, refresh, list and force kernels a step: the refresh of a small
    job is one launch, that of a large one five (classify, scan, replay,
    arrivals, place over the whole chip)"""
    assert _served(L, eam, "lj", (20,))[0] == 4
    assert _served(L, eam, "lj", (26,))[0] == 8
