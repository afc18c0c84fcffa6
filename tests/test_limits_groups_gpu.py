"""GPU: fmd_matt_findLimits of a group number that no atom has, a negative one
among them: the starting values, as before the atoms are distributed (only
FMD_GROUP_ALL, -1, means every atom)."""
import ctypes as C

import numpy as np
import pytest

from fmd_gb300 import api

pytestmark = pytest.mark.gpu


def test_groups_without_atoms(gpu_lib):
    lib = gpu_lib
    md = C.c_void_p(lib.fmd_create())
    lib.fmd_io_setShowErrorMessages(md, False)
    lib.fmd_box_setSubdomains(md, 1, 1, 1)
    lib.fmd_box_setSize(md, 60.0, 60.0, 60.0)
    lib.fmd_box_setPBC(md, True, True, True)
    api.set_atom_kinds(lib, md, ["Ar"], [39.948])
    lib.fmd_pot_lj_apply(md, 0, 0, 3.405, 0.0104, 8.5125)
    lib.fmd_matt_makeCuboidFCC(md, 0.0, 0.0, 0.0, 4, 4, 4, 5.26, 0, 3, 100.0)
    lo, hi = (C.c_double * 3)(), (C.c_double * 3)()
    groups = (-1, 3, 0, -2, -7)
    found = []
    lib.L.fmdx_distribute.argtypes = [C.c_void_p]
    for distributed in (False, True):
        if distributed:
            assert lib.L.fmdx_distribute(md) == 0
        for g in groups:
            lib.fmd_matt_findLimits(md, g, lo, hi)
            found.append(list(lo) + list(hi))
    assert found[:len(groups)] == found[len(groups):]
    nobody = [np.finfo(float).max] * 3 + [np.finfo(float).tiny] * 3
    assert [f == nobody for f in found[:len(groups)]] == [False, False, True, True, True]
    lib.fmd_free(md)
