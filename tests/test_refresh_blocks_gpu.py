"""A small system's refresh by one cluster of eight blocks, the fallback of
devices without room for sixteen: the same bits as the default."""
import ctypes as C

import numpy as np
import pytest

from fmd_gb300 import serve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pot,n", [("lj", 4), ("eam", 8), ("morse", 12)])
def test_eight_blocks(gpu_lib, pot, n):
    L = serve.bind(gpu_lib.L)
    L.fmdg_set_refresh_blocks.argtypes = [C.c_void_p, C.c_int]
    eam = serve.eam_tables(L)
    x, v, l = serve.job_atoms(dict(pot=pot, ncell=n, T=900.0, seed=3))
    states = []
    for blocks in (0, 8):
        one = serve.Single(L, pot, x, v, l, precision=serve.PREC_FP64, eam=eam)
        assert L.fmdg_set_refresh_blocks(one.h, blocks) == 0
        assert L.fmdg_set_refresh_blocks(one.h, 5) != 0
        one.steps(60)
        states.append(one.state())
        one.close()
    for a, b in zip(*states):
        np.testing.assert_array_equal(a, b)
