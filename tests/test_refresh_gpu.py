"""Cell refresh at the sizes where its kernels change: one to eight blocks of
512 in the cluster of a small system, the grid kernels beyond 8192 atoms, and
cell counts that are no multiple of a block.  Order, cells and positions equal
the oracle's, refresh after refresh."""
import os
import sys

import numpy as np
import pytest

from fmd_gb300 import api, workloads

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))
import pyoracle  # noqa: E402

pytestmark = pytest.mark.gpu
A = 5.26


@pytest.mark.parametrize("cells,open_z", [((4, 4, 4), False), ((5, 5, 5), True), ((6, 7, 8), False),
                                          ((10, 11, 12), True), ((12, 13, 13), False), ((13, 13, 13), False),
                                          ((25, 24, 23), True), ((40, 39, 9), False)])
def test_refresh_matches_oracle(gpu_lib, tmp_path, cells, open_z):
    box = np.array(cells) * A
    if open_z:
        box[2] += 20.0
    x, v = workloads.fcc_state(*cells, A, 100.0, 39.948, seed=5, origin=(0.0, 0.0, 10.0 if open_z else 0.0))
    n = len(x)
    kind, group = np.zeros(n, np.uint32), np.zeros(n, np.int32)
    lib, pbc = gpu_lib, (1, 1, 0 if open_z else 1)
    import ctypes as C
    md = C.c_void_p(lib.fmd_create())
    lib.fmd_io_setShowErrorMessages(md, False)
    lib.fmd_box_setSubdomains(md, 1, 1, 1)
    lib.fmd_box_setSize(md, *box)
    lib.fmd_box_setPBC(md, *[bool(p) for p in pbc])
    api.set_atom_kinds(lib, md, ["Ar"], [39.948])
    lib.fmd_pot_lj_apply(md, 0, 0, 3.405, 0.0104, 8.5125)
    path = str(tmp_path / "s.stt")
    api.write_state(path, 0.0, box, pbc, ["Ar"], kind, group, x, v)
    lib.fmd_io_loadState(md, path.encode(), False)
    lib.fmd_dync_integrate(md, -1, 0.0, 0.002)
    d = lib.dump(md)
    nc, cellh, l, _ = lib.grid(md)
    o = pyoracle.Oracle()
    o.setup(l, pbc, nc, cellh, [("Ar", 39.948)], [("lj", 0, 0, 3.405, 0.0104, 8.5125)])
    o.upload(d["cell"], d["x"], d["v"], d["kind"], d["group"], d["id"], int(np.prod(nc)))
    rng = np.random.default_rng(n)
    for _ in range(3):
        # up to a cell's width, so every cell has departures (open faces: a few atoms leave)
        y = d["x"] + rng.uniform(-0.9, 0.9, d["x"].shape) * cellh.min()
        lib.set_state(md, y, None)
        lib.wb("refresh")(md)
        o.set_state(y, None)
        assert o.refresh() == 0
        d, e = lib.dump(md), o.dump()
        for key in ("id", "cell", "x"):
            np.testing.assert_array_equal(d[key], e[key], err_msg=key)
    lib.fmd_free(md)
    o.close()
