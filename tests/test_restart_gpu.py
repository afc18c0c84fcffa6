"""A run continued from a saved state repeats the run that saved it, bit for
bit: saved between two runs and inside one (an event handler), binary64 and
mixed, small systems (cluster refresh, many shares) and larger ones.  Saving
changes nothing else: the run up to there, and the file, are those of a run
without it."""
import ctypes as C
import os

import numpy as np
import pytest

from fmd_gb300 import api, workloads

pytestmark = pytest.mark.gpu

POTS = {"lj": ("Ar", 39.948, 5.26, 0.002), "morse": ("Cu", 63.546, 3.615, 0.001), "eam": ("Cu", 63.546, 3.615, 0.001)}
FMD_EVENT_TIMER_TICK = 0


def _system(lib, work, pot, cells, precision, state=None):
    name, mass, a, dt = POTS[pot]
    md = C.c_void_p(lib.fmd_create())
    lib.fmd_io_setShowErrorMessages(md, False)
    lib.fmd_io_setSaveDirectory(md, (str(work) + "/").encode())
    lib.fmd_box_setSubdomains(md, 1, 1, 1)
    if state is None:
        lib.fmd_box_setSize(md, cells * a, cells * a, cells * a)
        lib.fmd_box_setPBC(md, True, True, True)
    api.set_atom_kinds(lib, md, [name], [mass])
    if pot == "lj":
        lib.fmd_pot_lj_apply(md, 0, 0, 3.405, 0.0104, 8.5125)
    elif pot == "morse":
        lib.fmd_pot_morse_apply(md, 0, 0, 0.3429, 1.3588, 2.866, 8.0)
    else:
        path = os.path.join(str(work), "a.eam.alloy")
        if not os.path.exists(path):
            workloads.write_analytic_eam(path)
        lib.fmd_pot_apply(md, 0, 0, lib.fmd_pot_eam_alloy_load(md, path.encode()))
    lib.L.fmdx_set_precision.argtypes = [C.c_void_p, C.c_int]
    lib.L.fmdx_set_precision(md, precision)
    if state is None:
        lib.L.fmdx_set_seed.argtypes = [C.c_void_p, C.c_ulonglong]
        lib.L.fmdx_set_seed(md, 3)
        lib.fmd_matt_makeCuboidFCC(md, 0.0, 0.0, 0.0, cells, cells, cells, a, 0, 0, 900.0)
    else:
        lib.fmd_io_loadState(md, str(state).encode(), True)
    return md, dt


def _run(lib, md, dt, steps):
    lib.fmd_dync_integrate(md, -1, (steps - 0.5) * dt, dt)


def _same(a, b):
    for key in ("cell", "kind", "x", "v", "F"):
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)


CASES = [("lj", 8), ("morse", 6), ("eam", 8), ("lj", 16), ("eam", 14)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("pot,cells", CASES)
def test_saved_between_runs(gpu_lib, tmp_path, pot, cells, precision):
    lib = gpu_lib
    md, dt = _system(lib, tmp_path, pot, cells, precision)
    _run(lib, md, dt, 77)
    lib.fmd_io_saveState(md, b"s.stt")
    _run(lib, md, dt, 50)
    went_on = lib.dump(md)
    lib.fmd_free(md)
    md, dt = _system(lib, tmp_path, pot, cells, precision, state=tmp_path / "s.stt")
    _run(lib, md, dt, 50)
    _same(lib.dump(md), went_on)
    lib.fmd_free(md)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("pot,cells", CASES)
def test_saved_inside_a_run(gpu_lib, tmp_path, pot, cells, precision):
    lib = gpu_lib
    md, dt = _system(lib, tmp_path, pot, cells, precision)
    saved = []

    def handler(mdp, event, user, params):
        if event == FMD_EVENT_TIMER_TICK:
            t = lib.fmd_dync_getTime(mdp)
            if t > dt and not saved:
                lib.fmd_io_saveState(mdp, b"s.stt")
                saved.append(t)

    keep = api.EventHandler(handler)
    lib.fmd_setEventHandler(md, None, keep)
    lib.fmd_timer_makeSimple(md, 0.0, 70 * dt, -1.0)
    _run(lib, md, dt, 120)
    went_on = lib.dump(md)
    lib.fmd_free(md)
    assert len(saved) == 1 and abs(saved[0] / dt - 70) < 1e-6
    md, dt = _system(lib, tmp_path, pot, cells, precision, state=tmp_path / "s.stt")
    _run(lib, md, dt, 50)
    _same(lib.dump(md), went_on)
    lib.fmd_free(md)


def test_saving_changes_nothing_before_it(gpu_lib, tmp_path):
    """77 steps in one run and in two, without a save: the same bits."""
    lib = gpu_lib
    out = []
    for parts in ((77,), (40, 37)):
        md, dt = _system(lib, tmp_path, "lj", 8, 0)
        for k in parts:
            _run(lib, md, dt, k)
        out.append(lib.dump(md))
        lib.fmd_free(md)
    _same(*out)
