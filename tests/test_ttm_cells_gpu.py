"""The electron solver of the 1-D two-temperature model on a slab at rest: the
first update (one launch, `ratio` substeps) against the oracle, src/ttm.c:194-383.
"""
import tempfile

import numpy as np
import pytest

import cases
import test_parity_oracle_gpu as parity
from fmd_gb300 import workloads

pytestmark = pytest.mark.gpu

A = 3.615


def _first_update(lib, work, nz, cells, Te, K, fluence, depth, ratio):
    """A copper slab of nz unit cells with vacuum at both ends under a type-1
    turi of `cells` cells, after fmd_dync_integrate over no time: the
    engine's and the oracle's 1-D fields."""
    x, v = workloads.fcc_state(4, 4, nz, A, 300.0, 63.546, seed=5, origin=(0.0, 0.0, 20.0), disp=0.03)
    box = (4 * A, 4 * A, nz * A + 40.0)
    x = np.column_stack([np.mod(x[:, :2], 4 * A), x[:, 2]])
    spec = dict(box=box, pbc=(1, 1, 0), kinds=[("Cu", 63.546)], pots=[("eam", 0, 0)], x=x, v=v,
                kind=np.zeros(len(x), np.uint32), group=np.zeros(len(x), np.int32), dt=0.001)
    md, o = parity.build_both(lib, spec, work)
    laser = (fluence, 0.3, 0.0, 1e-13, depth)
    lib.fmd_matt_getTemperature(md)     # (the set-up reads the group's atom count)
    cases.setup_turi(lib, md, dict(cat=1, dims=(1, 1, cells), gamma=96.6, K=K, G=1e17, Te=Te, ratio=ratio, frac=0.1,
                                   laser=laser), work)
    lib.fmd_dync_integrate(md, -1, 0.0, spec["dt"])
    g = lib.ttm_1d(md, cells + 2)
    pd, pk = parity.pyoracle.ttm1_params(box, cells, x, 96.6, K, 1e17, laser, 0.1, ratio)
    o.ttm_setup(pd, pk, Te)
    o.set_time(0.0, spec["dt"])
    o.turi_update()
    r = o.ttm_1d(cells + 2)
    lib.fmd_free(md)
    o.close()
    return g, r


def _close(g, r, tol):
    np.testing.assert_array_equal(g["num"], r["num"])
    for name in ("Te", "xi"):
        # (xi of cells without atoms is not a number on either side)
        ok = np.isfinite(r[name])
        np.testing.assert_array_equal(np.isfinite(g[name]), ok)
        if ok.any():
            assert np.abs(g[name][ok] - r[name][ok]).max() <= tol * np.abs(r[name][ok]).max(), name


# (ratio, K, fluence) of slabs whose first substeps overshoot: cells go below
# zero and stand still while their neighbours go on.  A relative change of
# 1e-13 per substep moves the result by up to 1.3e-7 of its largest value
# (numpy restatement); the engine's substeps differ from the oracle's by less
# than 1e-14, so 1e-7 leaves a margin of 8.
@pytest.mark.parametrize("ratio,K,fluence", [(5, 1000.0, 100.0), (6, 400.0, 1000.0), (6, 1000.0, 100.0)])
def test_cells_that_pass_zero(gpu_lib, ratio, K, fluence):
    with tempfile.TemporaryDirectory() as work:
        g, r = _first_update(gpu_lib, work, 40, 40, 300.0, K, fluence, 1e-9, ratio)
    assert (r["Te"][r["num"] > 6] < 0.0).any()
    _close(g, r, 1e-7)


def test_cells_that_are_not_a_number(gpu_lib):
    with tempfile.TemporaryDirectory() as work:
        g, r = _first_update(gpu_lib, work, 40, 40, float("nan"), 400.0, 100.0, 1e-8, 10)
    assert np.isnan(r["Te"]).any() and np.isnan(r["xi"][r["num"] > 6]).all()
    _close(g, r, 1e-10)
