"""A device call that fails becomes an error event of the fmd.h API: the host
sources over an engine whose functions do nothing but the one that fails."""
import ctypes as C
import glob
import os
import re
import subprocess

import pytest

from fmd_gb300 import api

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FMD_EVENT_ERROR = 2         # enum fmd_event_t (include/fmd.h)
FMD_ERR_FUNCTION_FAILED = 8     # enum fmd_error_t


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    """The host sources over a stand-in engine; `failing` names the call
    that returns a status."""
    work = tmp_path_factory.mktemp("host")
    inc, hdr = os.path.join(ROOT, "include"), open(os.path.join(ROOT, "include", "fmdg.h")).read()
    names = sorted(set(re.findall(r"\bint (fmdg_\w+)\(", hdr)) - {"fmdg_create"})
    fake = ["#include <string.h>", "const char *failing = \"\";",
            "const char *fmdg_last_error(void) { return \"stand-in\"; }", "void fmdg_destroy(void *s) { }",
            "int fmdg_create(void **s, int device) { static int one; *s = &one; return 0; }"]
    fake += ['int %s() { return strcmp(failing, "%s") ? 0 : -1; }' % (n, n) for n in names]
    (work / "fake.c").write_text("\n".join(fake) + "\n")
    so = work / "libhost.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-I" + inc, "-I/usr/local/cuda/include",
                    *sorted(glob.glob(os.path.join(ROOT, "fmd_gb300", "csrc", "host", "*.c"))), str(work / "fake.c"),
                    "-o", str(so), "-lm"], check=True)
    return api.Lib(str(so))


def test_find_limits_reports_a_failed_call(host):
    errors = []

    def handler(md, event, user, params):
        if event == FMD_EVENT_ERROR:
            errors.append(C.cast(params, C.POINTER(api.ErrorParams)).contents.error)

    keep = api.EventHandler(handler)
    md = C.c_void_p(host.fmd_create())
    host.fmd_io_setShowErrorMessages(md, False)
    host.fmd_setEventHandler(md, None, keep)
    host.fmd_box_setSubdomains(md, 1, 1, 1)
    host.fmd_box_setSize(md, 60.0, 60.0, 60.0)
    host.fmd_box_setPBC(md, True, True, True)
    api.set_atom_kinds(host, md, ["Ar"], [39.948])
    host.fmd_pot_lj_apply(md, 0, 0, 3.405, 0.0104, 8.5125)
    host.fmd_matt_makeCuboidFCC(md, 0.0, 0.0, 0.0, 4, 4, 4, 5.26, 0, 0, 100.0)
    host.L.fmdx_distribute.argtypes = [C.c_void_p]
    assert host.L.fmdx_distribute(md) == 0 and errors == []
    lo, hi = (C.c_double * 3)(), (C.c_double * 3)()
    failing = C.c_char_p.in_dll(host.L, "failing")
    host.fmd_matt_findLimits(md, -1, lo, hi)
    assert errors == []
    failing.value = b"fmdg_find_limits"
    host.fmd_matt_findLimits(md, -1, lo, hi)
    failing.value = b""
    assert errors == [FMD_ERR_FUNCTION_FAILED]
    host.fmd_free(md)
