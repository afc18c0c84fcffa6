"""GPU: refresh of cells at the sizes where the replay of a source cell
changes: up to 1024 atoms and arrivals a cell by a warp's masks, more by one
thread, in the cluster kernel (8064 atoms) and in the grid kernels (8640).
Order, cells and positions equal the oracle's (exactly), refresh after
refresh; every cell has departures and arrivals."""
import tempfile

import numpy as np
import pytest

from fmd_gb300 import workloads
from test_parity_oracle_gpu import build_both

pytestmark = pytest.mark.gpu
A = 5.26


@pytest.mark.parametrize("cells,rc", [((12, 12, 14), 31.0), ((12, 12, 15), 31.0), ((12, 12, 14), 20.0),
                                      ((12, 12, 15), 20.0)])
@pytest.mark.parametrize("share", [0.02, 1.0])       # of the atoms that are displaced
def test_large_cells(gpu_lib, cells, rc, share):
    x, v = workloads.fcc_state(*cells, A, 100.0, 39.948, seed=51, disp=0.05)
    n = len(x)
    spec = dict(box=tuple(c * A for c in cells), pbc=(1, 1, 1), kinds=[("Ar", 39.948)],
                pots=[("lj", 0, 0, 3.405, 0.0104, rc)], x=np.mod(x, np.array(cells) * A), v=v,
                kind=np.zeros(n, np.uint32), group=np.zeros(n, np.int32))
    rng = np.random.default_rng(n)
    with tempfile.TemporaryDirectory() as work:
        md, o = build_both(gpu_lib, spec, work)
        d = gpu_lib.dump(md)
        _, cellh, _, _ = gpu_lib.grid(md)
        for _ in range(3):
            move = rng.uniform(-0.9, 0.9, d["x"].shape) * (rng.random(n) < share)[:, None]
            y = d["x"] + move * cellh.min()
            gpu_lib.set_state(md, y, None)
            gpu_lib.wb("refresh")(md)
            o.set_state(y, None)
            assert o.refresh() == 0
            d, e = gpu_lib.dump(md), o.dump()
            for key in ("id", "cell", "x"):
                np.testing.assert_array_equal(d[key], e[key], err_msg=key)
        gpu_lib.fmd_free(md)
        o.close()
