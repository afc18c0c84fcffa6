"""The electron solver at the cell counts where its launch changes form: one
to many warps of cells, the last grid whose arrays fit the staging in shared
memory and the first that does not, a block of the largest size, and more
cells than threads.  The first update (one launch, 400 substeps) of a slab at
rest against the oracle, within the 1e-10 of the other TTM comparisons."""
import ctypes as C
import tempfile

import numpy as np
import pytest

import cases
import test_parity_oracle_gpu as parity
from fmd_gb300 import workloads

pytestmark = pytest.mark.gpu

A = 3.615
RATIO = 400         # (the explicit substeps of a 3.6 A cell are stable)
STAGED = (48 * 1024 - 8 * RATIO) // 68 - 2      # 68 bytes a cell, two margin cells


@pytest.mark.parametrize("cells", [20, 63, 64, 65, STAGED, STAGED + 1, 1023, 1024, 1100])
@pytest.mark.parametrize("cat", [1, 2])
def test_first_update(gpu_lib, cat, cells):
    lib = gpu_lib
    x, v = workloads.fcc_state(4, 4, cells, A, 300.0, 63.546, seed=7, origin=(0.0, 0.0, 20.0), disp=0.03)
    x = np.column_stack([np.mod(x[:, :2], 4 * A), x[:, 2]])
    spec = dict(box=(4 * A, 4 * A, cells * A + 40.0), pbc=(1, 1, 0), kinds=[("Cu", 63.546)], pots=[("eam", 0, 0)],
                x=x, v=v, kind=np.zeros(len(x), np.uint32), group=np.zeros(len(x), np.int32), dt=0.001)
    turi = dict(cat=cat, dims=(1, 1, cells), gamma=96.6, K=400.0, G=1e17, zhigilei=(1.57e6, 2.66e6, 2.41e11),
                Te=300.0, ratio=RATIO, frac=0.1, laser=(500.0, 0.0, 0.0, 100e-15, 15e-9))
    with tempfile.TemporaryDirectory() as work:
        md, o = parity.build_both(lib, spec, work)
        lib.fmd_matt_getTemperature(md)
        cases.setup_turi(lib, md, turi, work)
        lib.fmd_dync_integrate(md, -1, 0.0, spec["dt"])
        g = lib.ttm_1d(md, cells + 2)
        # the engine's derived parameters (equal to the reference's:
        # test_ttm_setup_matches_reference)
        pd, pk, tabs = np.zeros(17), np.zeros(9, np.int32), (C.c_void_p * 6)()
        f = lib.L.fmdx_ttm_params
        f.argtypes = [C.c_void_p] * 4
        assert f(md, pd.ctypes.data, pk.ctypes.data, tabs) == 0
        tables = {}
        if cat == 2:
            for w, key in enumerate(("T_C", "Ct", "C_DD", "T_G", "Gt", "G_DD")):
                n = int(pk[3] if w < 3 else pk[4])
                tables[key] = np.ctypeslib.as_array(C.cast(tabs[w], C.POINTER(C.c_double)), shape=(n,)).copy()
        o.ttm_setup(pd, pk, turi["Te"], tables)
        o.set_time(0.0, spec["dt"])
        o.turi_update()
        r = o.ttm_1d(cells + 2)
        lib.fmd_free(md)
        o.close()
    np.testing.assert_array_equal(g["num"], r["num"])
    assert r["Te"].max() > 400.0 and (r["num"] >= pk[2]).sum() > cells - 16
    for name in ("Te", "xi"):
        assert np.abs(g[name] - r[name]).max() <= 1e-10 * np.abs(r[name]).max(), name
