"""List walks split into shares and lanes (skin-list density and force
kernels): the share count of a system follows from its size alone, and how
many lanes walk the shares changes nothing."""
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


def _cube(pot, n, seed):
    P = serve.POTENTIALS[pot]
    x, v = workloads.fcc_state(n, n, n, P["a"], 300.0, P["mass"], seed=seed, disp=0.05)
    l = n * P["a"]
    return x - l * np.floor(x / l), v, l


def _forces(L, eam, pot, x, v, l, precision):
    one = serve.Single(L, pot, x, v, l, precision=precision, eam=eam)
    _, _, F, rows = one.state()
    th = one.th0
    one.close()
    out = np.zeros_like(F)
    out[rows] = F
    return out, th


# cells per edge on either side of each change of the share count (16 8 4 2 1)
SIZES = {serve.PREC_FP64: (4, 18, 19, 25, 30, 37), serve.PREC_MIXED: (5, 12, 15, 18, 21)}
# both binary64 paths carry ~48 significant bits per pair quantity: the
# parity bound of the forces, 1e-10 of the largest; mixed: 1e-5
BOUND = {serve.PREC_FP64: 1e-10, serve.PREC_MIXED: 1e-5}


@pytest.mark.parametrize("precision", [serve.PREC_FP64, serve.PREC_MIXED])
@pytest.mark.parametrize("pot,step", [("lj", 1), ("eam", 1), ("morse", 2)])
def test_shares_match_exact_list(L, eam, monkeypatch, pot, step, precision):
    for n in SIZES[precision][::step]:
        x, v, l = _cube(pot, max(n, 5) if pot != "lj" else n, 70 + n)
        F, th = _forces(L, eam, pot, x, v, l, precision)
        monkeypatch.setenv("FMD_SKIN", "0")           # the exact per-step list, one thread per atom
        R, tr = _forces(L, eam, pot, x, v, l, serve.PREC_FP64)
        monkeypatch.delenv("FMD_SKIN")
        assert np.abs(F - R).max() <= BOUND[precision] * np.abs(R).max(), n
        assert abs(th.potential - tr.potential) <= BOUND[precision] * abs(tr.potential), n


@pytest.mark.parametrize("precision", [serve.PREC_FP64, serve.PREC_MIXED])
@pytest.mark.parametrize("pot,n", [("lj", 6), ("eam", 8), ("morse", 5)])
def test_lanes_change_nothing(L, eam, pot, n, precision):
    """A small job alone (every share its own lane) and among enough others
    for a lane to walk several shares: the same bits."""
    x, v, l = _cube(pot, n, 81)
    got = []
    for others in (0, 40):
        srv = serve.Server(L, budget_bytes=8 << 30, max_jobs=64, chunk_steps=8, eam=eam)
        jid = srv.submit(pot, x, v, l, 24, precision=precision, keep_state=True)
        for k in range(others):
            p = ("lj", "eam", "morse")[k % 3]
            srv.submit(p, *_cube(p, 8 + k % 3, 90 + k), 24, precision=precision)
        srv.drain()
        got.append(srv.state(jid, len(x)))
        srv.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


def test_release_between_batches(L, eam):
    """Jobs released as soon as a batch is done, batch after batch on one
    server: a released job is gone from its pack too."""
    x, v, l = _cube("lj", 6, 99)
    srv = serve.Server(L, budget_bytes=8 << 30, max_jobs=64, chunk_steps=8, eam=eam)
    first = None
    for _ in range(6):
        ids = [srv.submit("lj", x, v, l, 16, precision=p, keep_state=True) for p in (0, 1, 0, 1, 0)]
        srv.drain()
        got = [srv.state(j, len(x))[0] for j in ids]
        for j in ids:
            srv.release(j)
        first = first or got
        for a, b in zip(first, got):
            np.testing.assert_array_equal(a, b)
    srv.close()
