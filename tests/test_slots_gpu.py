"""A list build numbers the slots of a single system in the current cell
order: after it nothing depends on how the atoms lay when they were uploaded.
A run of hot atoms whose list is then rebuilt gives the same bits (forces, and
the energy and virial that the blocks of slots sum) as its state uploaded
afresh.  One thread a slot and several lanes, few shares and many."""
import ctypes as C

import numpy as np
import pytest

from fmd_gb300 import serve

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L(gpu_lib):
    L = serve.bind(gpu_lib.L)
    L.fmdg_set_state.argtypes = [C.c_void_p, C.POINTER(C.c_double), C.POINTER(C.c_double)]
    return L


@pytest.fixture(scope="module")
def eam(L):
    return serve.eam_tables(L)


@pytest.mark.parametrize("precision", [serve.PREC_FP64, serve.PREC_MIXED])
@pytest.mark.parametrize("pot,cells", [("lj", 5), ("eam", 7), ("morse", 13), ("lj", 21), ("eam", 26)])
def test_build_renumbers(L, eam, pot, cells, precision):
    x, v, l = serve.job_atoms(dict(pot=pot, ncell=cells, T=1100.0, seed=60))
    a = serve.Single(L, pot, x, v, l, precision=precision, eam=eam)
    a.steps(80)
    xa, va, _, ids = a.state()
    assert L.fmdg_set_state(a.h, xa.ctypes.data_as(C.POINTER(C.c_double)), None) == 0      # (the list is stale now)
    assert L.fmdg_compute_forces(a.h, -1) == 0
    fa, ta = a.state()[2], a.thermo()
    a.close()
    b = serve.Single(L, pot, xa, va, l, precision=precision, eam=eam)
    xb, _, fb, idb = b.state()
    tb = b.thermo()
    b.close()
    np.testing.assert_array_equal(idb, np.arange(len(xa)))      # (the same storage order)
    np.testing.assert_array_equal(fa, fb)
    assert (ta.potential, ta.virial) == (tb.potential, tb.virial)
