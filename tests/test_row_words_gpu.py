"""GPU: the last words of the slots' position rows carry F'(rho) in a step
over every atom and the kinds in a step over one group: runs over all atoms
and over a group that holds them all take turns on one EAM system (one
element), against the CPU oracle.

Tolerances (those of the oracle parity tests): binary64 forces 1e-10 of max
|F|, energy 1e-10, positions and velocities 1e-9; mixed forces 1e-5, energy
1e-6."""
import tempfile

import numpy as np
import pytest

from fmd_gb300 import workloads
from test_parity_oracle_gpu import build_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [6, 14])       # shares of the list walk; one thread per atom
@pytest.mark.parametrize("precision", [0, 1])
def test_group_and_all_in_turn(gpu_lib, precision, cells):
    x, v = workloads.fcc_state(cells, cells, cells, 3.615, 300.0, 63.546, seed=41, disp=0.04)
    n, dt = len(x), 0.001
    spec = dict(box=(cells * 3.615,) * 3, pbc=(1, 1, 1), kinds=[("Cu", 63.546)], pots=[("eam", 0, 0)], x=x, v=v,
                kind=np.zeros(n, np.uint32), group=np.zeros(n, np.int32), dt=dt)
    f, e = (1e-10, 1e-10) if precision == 0 else (1e-5, 1e-6)
    with tempfile.TemporaryDirectory() as work:
        md, o = build_both(gpu_lib, spec, work, precision=precision)
        for group in (-1, 0, -1, 0):
            gpu_lib.fmd_dync_integrate(md, group, 0.0, dt)       # forces only
            o.forces(group)
            g, r = gpu_lib.dump(md), o.dump()
            np.testing.assert_array_equal(g["id"], r["id"])
            assert np.abs(g["F"] - r["F"]).max() <= f * np.abs(r["F"]).max()
            assert abs(g["pe"] - r["pe"]) <= e * abs(r["pe"])
            if precision == 0:
                gpu_lib.fmd_dync_integrate(md, group, 2.5 * dt, dt)
                o.vv(3, dt, group)
                g, r = gpu_lib.dump(md), o.dump()
                np.testing.assert_array_equal(g["id"], r["id"])
                assert np.abs(g["x"] - r["x"]).max() <= 1e-9
                assert np.abs(g["v"] - r["v"]).max() <= 1e-9
        gpu_lib.fmd_free(md)
        o.close()
