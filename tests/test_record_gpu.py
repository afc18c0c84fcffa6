"""The thermo record is formed on the last step of a batch only (steps in
between leave at most the Berendsen scale): a batch of k steps equals k
batches of one, bit for bit, record included."""
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


@pytest.mark.parametrize("thermostat", [0, 1])
@pytest.mark.parametrize("skin", ["0", "0.5"])          # per-step list, skin list
@pytest.mark.parametrize("precision", [serve.PREC_FP64, serve.PREC_MIXED])
@pytest.mark.parametrize("pot,n", [("lj", 4), ("eam", 7), ("morse", 13)])
def test_batch_equals_single_steps(L, eam, monkeypatch, pot, n, precision, skin, thermostat):
    monkeypatch.setenv("FMD_SKIN", skin)
    P = serve.POTENTIALS[pot]
    x, v = workloads.fcc_state(n, n, n, P["a"], 300.0, P["mass"], seed=7)
    got = []
    for batches in ([6], [1] * 6, [4, 2]):
        one = serve.Single(L, pot, x, v, n * P["a"], precision=precision, eam=eam)
        for k in batches:
            serve.check(L, L.fmdg_vv_steps(one.h, k, one.dt, -1, thermostat, 0.1, 150.0), "vv_steps")
        t = one.thermo()
        got.append([*one.state(), np.array([t.kinetic, t.temperature, t.potential, t.virial, t.count])])
        one.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            np.testing.assert_array_equal(a, b)
