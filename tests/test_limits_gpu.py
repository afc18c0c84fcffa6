"""GPU: the extent of a group's atoms equals the extent of the dumped
positions exactly, for one atom, partial warps, several blocks and a group
without atoms (the starting values: largest and smallest positive double)."""
import ctypes as C

import numpy as np
import pytest

from fmd_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 257, 70001])
def test_group_limits(gpu_lib, tmp_path, n):
    lib, box = gpu_lib, np.array([60.0, 70.0, 80.0])
    rng = np.random.default_rng(n)
    x = rng.uniform(0.01, 0.99, (n, 3)) * box
    group = rng.integers(0, 3, n).astype(np.int32)
    md = C.c_void_p(lib.fmd_create())
    lib.fmd_io_setShowErrorMessages(md, False)
    lib.fmd_box_setSubdomains(md, 1, 1, 1)
    lib.fmd_box_setSize(md, *box)
    lib.fmd_box_setPBC(md, True, True, True)
    api.set_atom_kinds(lib, md, ["Ar"], [39.948])
    lib.fmd_pot_lj_apply(md, 0, 0, 0.1, 1e-6, 3.0)
    path = str(tmp_path / "s.stt")
    api.write_state(path, 0.0, box, (1, 1, 1), ["Ar"], np.zeros(n, np.uint32), group, x, np.zeros((n, 3)))
    lib.fmd_io_loadState(md, path.encode(), False)
    lib.L.fmdx_distribute.argtypes = [C.c_void_p]
    assert lib.L.fmdx_distribute(md) == 0
    d = lib.dump(md)
    lo, hi = (C.c_double * 3)(), (C.c_double * 3)()
    for g in (-1, 0, 1, 2, 7):
        lib.fmd_matt_findLimits(md, g, lo, hi)
        y = d["x"] if g < 0 else d["x"][d["group"] == g]
        if len(y):
            np.testing.assert_array_equal(np.array(lo), y.min(axis=0))
            np.testing.assert_array_equal(np.array(hi), y.max(axis=0))
        else:
            assert list(lo) == [np.finfo(float).max] * 3 and list(hi) == [np.finfo(float).tiny] * 3
    lib.fmd_free(md)
