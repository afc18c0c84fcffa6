"""Atoms that leave through open faces between two list builds: their slots
stay in their neighbours' lists, out of reach, until the next build.  Step by
step while atoms leave (and no atom has moved far enough to rebuild a list):
count, order, forces, energy and virial against the oracle, in the bounds of
the other comparisons with it."""
import ctypes as C
import tempfile

import numpy as np
import pytest

import test_parity_oracle_gpu as parity
from fmd_gb300 import serve, workloads

pytestmark = pytest.mark.gpu

POTS = {"lj": (5.26, ("Ar", 39.948), [("lj", 0, 0, 3.405, 0.0104, 8.5125)], 0.002),
        "morse": (3.615, ("Cu", 63.546), [("morse", 0, 0, 0.3429, 1.3588, 2.866, 8.0)], 0.001),
        "eam": (3.615, ("Cu", 63.546), [("eam", 0, 0)], 0.001)}
STEPS = 10


def _slab(pot, cells):
    """A cold slab with its surfaces 0.7 a from the open faces, and atoms over
    hollow sites that cross a face in one to nine steps."""
    a, kind, pots, dt = POTS[pot]
    gap = 0.7 * a
    x, v = workloads.fcc_state(*cells, a, 5.0, kind[1], seed=11, disp=0.02)
    sites = workloads.fcc_sites(*cells, a)
    x[:, 2] += gap - sites[:, 2].min()
    sites[:, 2] += gap - sites[:, 2].min()
    top = sites[:, 2].max()
    lz = top + gap
    rng = np.random.default_rng(4)
    out, vel = [], []
    for face, layer in ((lz, top - a / 2), (0.0, gap + a / 2)):
        hollow = sites[np.abs(sites[:, 2] - layer) < 0.1]
        for k, s in enumerate(hollow[rng.permutation(len(hollow))[:18]]):
            sign = 1.0 if face else -1.0
            out.append([s[0], s[1], face - sign * (0.01 + 0.02 * (k % 9))])
            vel.append([0.0, 0.0, sign * 0.02 / dt])
    x, v = np.concatenate([x, out]), np.concatenate([v, vel])
    box = (cells[0] * a, cells[1] * a, lz)
    x[:, :2] = np.mod(x[:, :2], box[:2])
    return dict(box=box, pbc=(1, 1, 0), kinds=[kind], pots=pots, x=x, v=v, kind=np.zeros(len(x), np.uint32),
                group=np.zeros(len(x), np.int32), dt=dt)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("cells", [(8, 8, 6), (16, 17, 10)])
@pytest.mark.parametrize("pot", list(POTS))
def test_forces_over_dead_slots(gpu_lib, pot, cells, precision):
    lib, spec = gpu_lib, _slab(pot, cells)
    L = serve.bind(lib.L)
    lib.L.fmdx_device.argtypes, lib.L.fmdx_device.restype = [C.c_void_p], C.c_void_p
    tf, te, tw = (1e-10, 1e-10, 1e-10) if precision == 0 else (1e-5, 1e-6, 1e-5)
    with tempfile.TemporaryDirectory() as work:
        md, o = parity.build_both(lib, spec, work, precision)
        lib.fmd_dync_integrate(md, -1, 0.0, spec["dt"])
        o.forces(-1)
        dev = C.c_void_p(lib.L.fmdx_device(md))
        d0 = lib.dump(md)
        z0 = dict(zip(d0["id"].tolist(), d0["x"]))
        counts = [len(d0["id"])]
        for _ in range(STEPS):
            assert L.fmdg_vv_steps(dev, 1, spec["dt"], -1, 0, 1.0, 0.0) == 0
            o.vv(1, spec["dt"])
            g, r, th = lib.dump(md), o.dump(), serve.Thermo()
            assert L.fmdg_get_thermo(dev, C.byref(th)) == 0
            np.testing.assert_array_equal(g["id"], r["id"])
            counts.append(len(g["id"]))
            assert th.count == counts[-1]
            assert np.abs(g["F"] - r["F"]).max() <= tf * np.abs(r["F"]).max()
            assert abs(th.potential - r["pe"]) <= te * abs(r["pe"])
            assert abs(th.virial - r["virial"]) <= tw * max(abs(r["virial"]), abs(r["pe"]))
        # atoms left step after step, and no list was due (skin / 2 = 0.25 A)
        assert counts[-1] == counts[0] - 36 and len(set(counts)) >= 8
        move = np.array([g["x"][k] - z0[i] for k, i in enumerate(g["id"].tolist())])
        move[:, :2] -= np.round(move[:, :2] / np.array(spec["box"][:2])) * np.array(spec["box"][:2])
        assert np.linalg.norm(move, axis=1).max() < 0.24
        lib.fmd_free(md)
        o.close()
