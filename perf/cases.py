"""Workloads of the engine, each with its inputs, one pass through the public
entry points, its smallest possible work and its outputs in 64 bits.

A pass is what a program does between two looks at its results:

  dynamics  a run of `steps` time steps of one system through the fmd.h API
            (fmd_dync_integrate / fmd_dync_equilibrate) and the state read
            back; the next pass goes on from there, as a program's next call
            does
  snapshot  the same number of steps from a stored snapshot: positions and
            velocities in, cell refresh, initial forces, steps, state out
            (ensembles of short runs from one configuration; the analytic
            EAM's crystals collapse after about a thousand steps, so its
            passes start over)
  ttm       a run under the 1-D two-temperature model through fmd.h, its
            grid fields and the state read back
  served    jobs submitted to a live server, drained, and their results and
            final states fetched
  forces    one allocation-free force evaluation on the caller's device
            buffers

Positions, velocities and forces come back by atom number, as a program that
follows its atoms keeps them, beside the storage order itself.  A run in mixed
precision rests on binary32 pair arithmetic, and what it returns is kept in
binary32.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import random
import tempfile

import numpy as np
import torch

import fmd_gb300
from fmd_gb300 import api, serve, workloads

KB = 8.6173303e-5                 # eV/K
MASS_UNIT = 9.6485332907e+03      # Da per internal mass unit

# pair potentials of the configurations: LJ argon (2.5 sigma), Morse copper
# (8 A), the analytic copper EAM (5.5 A, smoothly cut)
POTS = {
    "lj": dict(a=5.26, mass=39.948, dt=0.002, rc=8.5125, kind="Ar", cells=4),
    "morse": dict(a=3.615, mass=63.546, dt=0.001, rc=8.0, kind="Cu", cells=5),
    "eam": dict(a=3.615, mass=63.546, dt=0.001, rc=5.5, kind="Cu", cells=4),
}
LJ_EPS, LJ_SIG = 0.0104, 3.405
MORSE = (0.3429, 1.3588, 2.866)
# the copper-argon jobs of the served mode (LJ copper-argon pairs)
CUAR = dict(ar=(3.4, 0.0104, 8.5), mix=(2.87, 0.0652, 7.175), dt=0.001, rc=8.5, masses=(63.546, 39.948))
VACUUM = 20.0                     # A on either side of an open face
# flops of one pair (half shell), by the formulas of each potential
PAIR_FLOPS = {"lj": 27, "morse": 40, "eam": 94}
FCC = np.array([[0.0, 0.0, 0.0], [0.0, 0.5, 0.5], [0.5, 0.0, 0.5], [0.5, 0.5, 0.0]])


def listed():
    return [
        # the smallest: a thermostatted box of the test suite's size, where a
        # step is launches and latency
        dict(name="argon_256_equilibrate", do="dynamics", pot="lj", nx=4, ny=4, nz=4, T=100.0, steps=50,
             precision="fp64", open_z=False, tau=0.1),
        # the argon example program: 10^3 cells, NVE in the drop-in precision
        dict(name="argon_4000", do="dynamics", pot="lj", nx=10, ny=10, nz=10, T=100.0, steps=100,
             precision="fp64", open_z=False, tau=0.0),
        # a free-standing plate with odd edges and open faces
        dict(name="morse_plate_4004", do="dynamics", pot="morse", nx=13, ny=11, nz=7, T=300.0, steps=50,
             precision="fp64", open_z=True, tau=0.0),
        # a small metal crystal, many short runs from one snapshot
        dict(name="eam_2048_snapshot", do="snapshot", pot="eam", nx=8, ny=8, nz=8, T=300.0, steps=50,
             precision="fp64", open_z=False, tau=0.0),
        # a mid-size liquid-like box in mixed precision
        dict(name="argon_32000_mixed", do="dynamics", pot="lj", nx=20, ny=20, nz=20, T=400.0, steps=50,
             precision="mixed", open_z=False, tau=0.0),
        # the EAM configuration, in both precisions
        dict(name="eam_256000", do="snapshot", pot="eam", nx=40, ny=40, nz=40, T=300.0, steps=40,
             precision="fp64", open_z=False, tau=0.0),
        dict(name="eam_256000_mixed", do="snapshot", pot="eam", nx=40, ny=40, nz=40, T=300.0, steps=60,
             precision="mixed", open_z=False, tau=0.0),
        # the Morse target slab at its full size: the largest system
        dict(name="morse_slab_512000_mixed", do="dynamics", pot="morse", nx=80, ny=80, nz=20, T=300.0, steps=20,
             precision="mixed", open_z=True, tau=0.0),
        # the laser-heated slab of the two-temperature configuration
        dict(name="ttm_slab_160000", do="ttm", pot="eam", nx=20, ny=20, nz=100, T=300.0, steps=50,
             precision="fp64", cells=50),
        # the serving loop: jobs of uneven sizes and potentials at once
        dict(name="served_mix", do="served", jobs=12, nmin=2000, nmax=60000, steps=128, precision="mixed", draw=5),
        # many small jobs, hybrid ones among them, in the drop-in precision
        dict(name="served_small", do="served", jobs=20, nmin=500, nmax=2500, steps=96, precision="fp64", draw=7),
        # forces alone, for hosts that own their device memory
        dict(name="forces_62100", do="forces", pot="morse", nx=27, ny=25, nz=23, T=300.0, open_z=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, pot, nmin, nmax, lean_z=False):
    """Cell counts of a box of about log-uniform(nmin, nmax) atoms, ragged."""
    least = POTS[pot]["cells"]
    n = _log_int(rng, nmin, nmax)
    side = (n / 4.0) ** (1.0 / 3.0)
    nx = max(least, int(round(side * rng.uniform(0.8, 1.25))))
    ny = max(least, int(round(side * rng.uniform(0.8, 1.25))))
    nz = max(1 if lean_z else least, int(round(n / 4.0 / (nx * ny))))
    while 4 * nx * ny * nz > nmax and nx > least:
        nx -= 1
    while 4 * nx * ny * nz > nmax and nz > least:
        nz -= 1
    return nx, ny, nz


def draw(rng):
    do = rng.choice(["dynamics", "dynamics", "dynamics", "snapshot", "snapshot", "served", "served", "ttm", "forces"])
    if do == "served":
        nmin = _log_int(rng, 500, 8000)
        return dict(do=do, jobs=rng.randint(2, 20), nmin=nmin, nmax=int(nmin * rng.uniform(1.5, 7.0)),
                    steps=rng.randint(40, 128), precision=rng.choice(["mixed", "mixed", "fp64"]),
                    draw=rng.randint(1, 1 << 20))
    if do == "ttm":
        nx, ny, nz = rng.randint(4, 14), rng.randint(4, 14), rng.randint(20, 90)
        return dict(do=do, pot="eam", nx=nx, ny=ny, nz=nz, T=rng.uniform(100.0, 600.0), steps=rng.randint(10, 40),
                    precision="fp64", cells=rng.randint(20, 60))
    if do == "forces":
        pot = rng.choice(["lj", "morse"])
        nx, ny, nz = _dims(rng, pot, 500, 60000)
        return dict(do=do, pot=pot, nx=nx, ny=ny, nz=nz, T=rng.uniform(50.0, 600.0), open_z=rng.random() < 0.3)
    pot = "eam" if do == "snapshot" else rng.choice(["lj", "morse"])
    open_z = rng.random() < 0.3
    nx, ny, nz = _dims(rng, pot, 256, 200000, open_z)
    n = 4 * nx * ny * nz
    return dict(do=do, pot=pot, nx=nx, ny=ny, nz=nz, T=rng.uniform(50.0, 600.0),
                steps=max(3, min(60, int(2e6 / n))), precision=rng.choice(["fp64", "mixed"]), open_z=open_z,
                tau=0.1 if do == "dynamics" and rng.random() < 0.25 else 0.0)


# ------------------------------------------------------------------- inputs
def _lattice(nx, ny, nz, a, origin=(0.0, 0.0, 0.0)):
    """FCC sites in the order the lattice builder makes them."""
    i, j, k = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij")
    cells = np.stack([i.ravel(), j.ravel(), k.ravel()], axis=1).astype(np.float64)
    return ((cells[:, None, :] + 0.25 + FCC[None]) * a).reshape(-1, 3) + np.asarray(origin)


def _velocities(n, mass, T, rng):
    v = rng.standard_normal((n, 3)) * math.sqrt(KB * T / (mass / MASS_UNIT))
    return v - v.mean(axis=0)


def _system(case, seed):
    """Box, positions (thermally displaced sites) and velocities."""
    P = POTS[case["pot"]]
    rng = np.random.default_rng([seed, 17])
    a, open_z = P["a"], case.get("open_z") or case["do"] == "ttm"
    box = np.array([case["nx"] * a, case["ny"] * a, case["nz"] * a + (2 * VACUUM if open_z else 0.0)])
    x = _lattice(case["nx"], case["ny"], case["nz"], a, (0.0, 0.0, VACUUM if open_z else 0.0))
    x = x + np.clip(rng.standard_normal(x.shape) * 0.04, -0.15, 0.15)
    v = _velocities(len(x), P["mass"], case["T"], rng)
    return box, (True, True, not open_z), x, v


def _served_jobs(case, seed):
    """(potential, x, v, box lengths, kinds) of every job: sizes log-uniform,
    the potentials in turn; small fleets hold copper-argon jobs too."""
    pick = random.Random(case["draw"])
    kinds = ["lj", "morse", "eam"] + (["cuar"] if case["nmax"] <= 4000 else [])
    jobs = []
    for k in range(case["jobs"]):
        pot = kinds[k % len(kinds)]
        n = math.exp(pick.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        T = pick.uniform(50.0, 600.0)
        rng = np.random.default_rng([seed, 29, k])
        if pot == "cuar":
            c = max(5, int(round((n / 5.5) ** (1.0 / 3.0))))
            lc = c * POTS["eam"]["a"]
            m = max(1, int(round(lc / POTS["lj"]["a"])))
            xc, xa = _lattice(c, c, c, lc / c), _lattice(m, m, m, lc / m, (lc + 2.0, 0.0, 0.0))
            x = np.concatenate([xc, xa])
            kind = np.concatenate([np.zeros(len(xc), np.uint32), np.ones(len(xa), np.uint32)])
            v = np.concatenate([_velocities(len(xc), CUAR["masses"][0], T, rng),
                                _velocities(len(xa), CUAR["masses"][1], T, rng)])
            box = np.array([2.0 * lc + 4.0, lc, lc])
        else:
            P = POTS[pot]
            c = max(5, int(round((n / 4.0) ** (1.0 / 3.0))))
            x = _lattice(c, c, c, P["a"])
            kind = np.zeros(len(x), np.uint32)
            v = _velocities(len(x), P["mass"], T, rng)
            box = np.full(3, c * P["a"])
        x = x + np.clip(rng.standard_normal(x.shape) * 0.04, -0.15, 0.15)
        jobs.append((pot, x, v, box, kind))
    return jobs


# ------------------------------------------------------------ library handles
_LOADED = {}


def _libs():
    """libfmd (fmd.h binding), the engine's binding and the EAM's files, once
    per process."""
    if not _LOADED:
        lib = fmd_gb300.load()
        vp, i, d = C.c_void_p, C.c_int, C.c_double
        for name, res, args in [("fmdx_device", vp, [vp]), ("fmdx_set_precision", None, [vp, i]),
                                ("fmdx_distribute", i, [vp]), ("fmdg_refresh", i, [vp]),
                                ("fmdg_compute_forces", i, [vp, i]), ("fmdg_get_thermo", i, [vp, vp]),
                                ("fmdg_run_host", i, [vp, i, d, i, vp, vp, vp, vp, vp, vp]),
                                ("fmdg_natoms", i, [vp, C.POINTER(i)])]:
            f = getattr(lib.L, name)
            f.restype, f.argtypes = res, args
        L = serve.bind(lib)
        L.fmdg_pair_forces_noalloc.restype = i
        L.fmdg_pair_forces_noalloc.argtypes = [i, C.POINTER(i), C.POINTER(i), C.POINTER(d), i, C.POINTER(serve.Pair)] + [vp] * 7
        work = tempfile.TemporaryDirectory()
        _LOADED.update(lib=lib, L=L, work=work,
                       setfl=workloads.write_analytic_eam(os.path.join(work.name, "analytic.eam.alloy")))
    return _LOADED


class _Md:
    """One fmd.h instance with its atoms on the device."""

    def __init__(self, case, box, pbc, x, v):
        G = _libs()
        self.lib, P = G["lib"], POTS[case["pot"]]
        lib, n = self.lib, len(x)
        self.md = md = C.c_void_p(lib.fmd_create())
        self.n, self.dt = n, P["dt"]
        lib.fmd_io_setShowErrorMessages(md, False)
        lib.fmd_box_setSubdomains(md, 1, 1, 1)
        lib.fmd_box_setSize(md, *box)
        lib.fmd_box_setPBC(md, *pbc)
        api.set_atom_kinds(lib, md, [P["kind"]], [P["mass"]])
        if case["pot"] == "lj":
            lib.fmd_pot_lj_apply(md, 0, 0, LJ_SIG, LJ_EPS, P["rc"])
        elif case["pot"] == "morse":
            lib.fmd_pot_morse_apply(md, 0, 0, *MORSE, P["rc"])
        else:
            lib.fmd_pot_apply(md, 0, 0, lib.fmd_pot_eam_alloy_load(md, G["setfl"].encode()))
        lib.L.fmdx_set_precision(md, 1 if case["precision"] == "mixed" else 0)
        lib.fmd_matt_makeCuboidFCC(md, 0.0, 0.0, 0.0 if pbc[2] else VACUUM, case["nx"], case["ny"], case["nz"],
                                   P["a"], 0, 0, case["T"])
        assert lib.L.fmdx_distribute(md) == 0, "the atoms could not be distributed"
        # positions and velocities of this seed, in the storage order
        ids = np.zeros(n, np.uint32)
        lib.wb("dump")(md, None, ids.ctypes.data, None, None, None, None, None, None)
        number = ids.astype(np.int64) - int(ids.min())
        self.first = int(ids.min())
        lib.set_state(md, x[number], v[number])
        lib.wb("refresh")(md)

    def device(self):
        return C.c_void_p(self.lib.L.fmdx_device(self.md))

    def __del__(self):
        try:
            self.lib.fmd_free(self.md)
        except Exception:
            pass


def _pinned(rows, n, dtype):
    return torch.empty((rows, n), dtype=dtype, pin_memory=True)


class _HostState:
    """Pinned host buffers of one system: state in and out."""

    def __init__(self, n):
        self.x, self.v = _pinned(3, n, torch.float64), _pinned(3, n, torch.float64)
        self.xin, self.vin = _pinned(3, n, torch.float64), _pinned(3, n, torch.float64)
        self.ids = _pinned(1, n, torch.int32)
        self.th = (C.c_double * 8)()


def _ck(rc, what):
    if rc:
        raise RuntimeError("%s: status %d" % (what, rc))


def _run_host(m, H, steps, read):
    L = m.lib.L
    p = lambda t: t.data_ptr()  # noqa: E731
    if read:
        _ck(L.fmdg_run_host(m.device(), steps, m.dt, -1, None, None, p(H.x), p(H.v), p(H.ids), C.addressof(H.th)),
            "fmdg_run_host")
    else:
        _ck(L.fmdg_run_host(m.device(), steps, m.dt, -1, p(H.xin), p(H.vin), None, None, None, None), "fmdg_run_host")


def _by_number(m, H, precision):
    """The pinned state by atom number (a row per atom), and the order."""
    number = H.ids[0].long() - m.first
    dtype = torch.float64 if precision == "fp64" else torch.float32
    x, v = torch.empty((m.n, 3), dtype=dtype), torch.empty((m.n, 3), dtype=dtype)
    x[number] = H.x.t().to(dtype)
    v[number] = H.v.t().to(dtype)
    return number, x, v


def _thermo(kinetic, temperature, potential, virial, precision):
    return np.array([kinetic, temperature, potential, virial], np.float64 if precision == "fp64" else np.float32)


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    do = case["do"]
    if do == "served":
        if "eam" not in _LOADED:
            _libs()["eam"] = serve.eam_tables(_libs()["L"])
        srv = serve.Server(_libs()["L"], budget_bytes=16 << 30, max_jobs=256, chunk_steps=32, eam=_LOADED["eam"])
        return dict(case=case, srv=srv, jobs=_served_jobs(case, seed), last=[])
    box, pbc, x, v = _system(case, seed)
    if do == "forces":
        return _prepare_forces(case, box, pbc, x)
    m = _Md(case, box, pbc, x, v)
    state = dict(case=case, m=m, host=_HostState(m.n))
    if do == "ttm":
        state["turi"] = _ttm_setup(m, case["cells"])
    else:
        m.lib.fmd_dync_integrate(m.md, -1, 0.0, m.dt)      # initial forces
    if do == "snapshot":
        state["x0"], state["v0"] = torch.from_numpy(x), torch.from_numpy(v)
        _run_host(m, state["host"], 0, True)
    return state


def _ttm_setup(m, cells):
    """Electron grid, material constants and pulse of the configuration."""
    lib, md = m.lib, m.md
    lib.fmd_matt_getTemperature(md)
    h = lib.fmd_turi_add(md, api.FMD_TURI_TTM_TYPE1, 1, 1, cells, 0.0, -1.0)
    lib._fmd_ttm_setHeatCapacity_linear(md, h, api.HeatCapacityLinear(96.6))
    lib._fmd_ttm_setHeatConductivity_constant1(md, h, 400.0)
    lib._fmd_ttm_setCouplingFactor_constant1(md, h, 1e17)
    lib.fmd_ttm_setElectronTemperature(md, h, 300.0)
    lib.fmd_ttm_setTimestepRatio(md, h, 100)
    lib.fmd_ttm_setCellActivationFraction(md, h, 0.1)
    lib._fmd_ttm_setLaserSource_gaussian(md, h, api.LaserGaussian(500.0, 0.0, 1e-12, 100e-15, 15e-9))
    return h


def _prepare_forces(case, box, pbc, x):
    P = POTS[case["pot"]]
    nc = (box / P["rc"]).astype(np.int64)
    ic = np.clip(np.floor(x / (box / nc)).astype(np.int64), 0, nc - 1)
    flat = ic[:, 2] + nc[2] * (ic[:, 1] + nc[1] * ic[:, 0])
    order = np.argsort(flat, kind="stable")
    start = np.concatenate([[0], np.cumsum(np.bincount(flat, minlength=int(nc.prod())))]).astype(np.int32)
    n = len(x)
    pair = (serve.Pair * 1)()
    pair[0].cat = serve.FMDG_POT_LJ if case["pot"] == "lj" else serve.FMDG_POT_MORSE
    for q, p in enumerate((4 * LJ_EPS, LJ_SIG ** 2, P["rc"] ** 2) if case["pot"] == "lj" else MORSE + (P["rc"] ** 2,)):
        pair[0].p[q] = p
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return dict(case=case, n=n, pair=pair, nc=(C.c_int * 3)(*[int(k) for k in nc]),
                pbc=(C.c_int * 3)(*[int(b) for b in pbc]), l=(C.c_double * 3)(*box), x=cuda(x[order].T),
                kind=torch.zeros(n, dtype=torch.int32, device="cuda"), start=cuda(start),
                cell=cuda(flat[order].astype(np.int32)), F=torch.empty((3, n), dtype=torch.float64, device="cuda"),
                pe=torch.empty(1, dtype=torch.float64, device="cuda"))


# --------------------------------------------------------------------- run
def run(state):
    return {"dynamics": _run_dynamics, "snapshot": _run_snapshot, "ttm": _run_ttm, "served": _run_served,
            "forces": _run_forces}[state["case"]["do"]](state)


DUMP_ATOMS = 50000   # up to here a program reads the forces too, through the per-atom dump


def _run_dynamics(s):
    case, m = s["case"], s["m"]
    lib, md, prec = m.lib, m.md, case["precision"]
    span = (case["steps"] - 0.5) * m.dt
    if case["tau"] > 0.0:
        lib.fmd_dync_equilibrate(md, -1, span, m.dt, case["tau"], case["T"])
    else:
        lib.fmd_dync_integrate(md, -1, span, m.dt)
    ke, T, e = lib.fmd_matt_getKineticEnergy(md), lib.fmd_matt_getTemperature(md), lib.fmd_matt_getTotalEnergy(md)
    th = _thermo(ke, T, e - ke, lib.wb("virial")(md), prec)
    if m.n > DUMP_ATOMS:
        _run_host(m, s["host"], 0, True)
        number, x, v = _by_number(m, s["host"], prec)
        return dict(order=number, x=x, v=v, thermo=th)
    d = lib.dump(md)
    number = d["id"].astype(np.int64) - m.first
    dtype = np.float64 if prec == "fp64" else np.float32
    out = dict(order=number, thermo=th)
    for key in ("x", "v", "F"):
        out[key] = np.zeros((m.n, 3), dtype)
        out[key][number] = d[key]
    return out


def _run_snapshot(s):
    case, m, H = s["case"], s["m"], s["host"]
    L, dev = m.lib.L, m.device()
    number = H.ids[0].long() - m.first
    H.xin.copy_(s["x0"][number].t())
    H.vin.copy_(s["v0"][number].t())
    _run_host(m, H, 0, False)
    _ck(L.fmdg_refresh(dev), "fmdg_refresh")
    _ck(L.fmdg_compute_forces(dev, -1), "fmdg_compute_forces")
    _run_host(m, H, case["steps"], True)
    number, x, v = _by_number(m, H, case["precision"])
    t = H.th                     # kinetic, temperature, momentum (3), potential, count, virial
    return dict(order=number, x=x, v=v, thermo=_thermo(t[0], t[1], t[5], t[7], case["precision"]))


def _run_ttm(s):
    case, m = s["case"], s["m"]
    m.lib.fmd_dync_integrate(m.md, -1, (case["steps"] - 0.5) * m.dt, m.dt)
    grid = m.lib.ttm_1d(m.md)
    _run_host(m, s["host"], 0, True)
    number, x, v = _by_number(m, s["host"], case["precision"])
    return dict(order=number, x=x, v=v, num=grid["num"].astype(np.int64), vcm=grid["vcm"][:, 2].copy(), Ti=grid["Ti"],
                Te=grid["Te"], xi=grid["xi"])


def _run_served(s):
    case, srv = s["case"], s["srv"]
    prec = serve.PREC_MIXED if case["precision"] == "mixed" else serve.PREC_FP64
    dtype = np.float32 if case["precision"] == "mixed" else np.float64
    ids = [srv.submit(pot, x, v, box, case["steps"], precision=prec, keep_state=True, kind=kind)
           for pot, x, v, box, kind in s["jobs"]]
    srv.drain()
    total = sum(len(j[1]) for j in s["jobs"])
    out = {key: np.empty((total, 3), dtype) for key in ("x", "v", "F")}
    order, th, at = [], [], 0
    for jid, job in zip(ids, s["jobs"]):
        n, r = len(job[1]), srv.result(jid)
        if r.state != 2 or r.errbits:
            raise RuntimeError("a served job failed (state %d, error bits %d)" % (r.state, r.errbits))
        x, v, F, number = srv.state(jid, n)
        rows = number.astype(np.int64) + at
        out["x"][rows], out["v"][rows], out["F"][rows] = x, v, F
        order.append(rows)
        for t in (r.first, r.last):
            th.append(_thermo(t.kinetic, t.temperature, t.potential, t.virial, case["precision"]))
        at += n
    # a batch's records are kept until the next batch is done
    for jid in s["last"]:
        srv.release(jid)
    s["last"] = ids
    return dict(out, order=np.concatenate(order), thermo=np.stack(th))


def _run_forces(s):
    p = lambda t: t.data_ptr()  # noqa: E731
    _ck(_libs()["L"].fmdg_pair_forces_noalloc(s["n"], s["nc"], s["pbc"], s["l"], 1, s["pair"], p(s["x"]), p(s["kind"]),
                                              p(s["start"]), p(s["cell"]), p(s["F"]), p(s["pe"]),
                                              torch.cuda.current_stream().cuda_stream), "fmdg_pair_forces_noalloc")
    return dict(F=s["F"], pe=s["pe"])


# -------------------------------------------------------------------- work
def _pairs_per_atom(pot):
    P = POTS[pot]
    return 0.5 * 4.0 / 3.0 * math.pi * P["rc"] ** 3 * 4.0 / P["a"] ** 3


def work(case):
    """State in and out once a pass (48 B each way per atom, forces 24 B where
    they come back); every pair inside the cutoff once a step."""
    if case["do"] == "served":
        b = f = 0.0
        for pot, x, _, _, _ in _served_jobs(case, 0):
            b += len(x) * (52 + 76)
            pot = "eam" if pot == "cuar" else pot
            f += len(x) * _pairs_per_atom(pot) * PAIR_FLOPS[pot] * (case["steps"] + 1)
        return dict(bytes=b, flops=f)
    n = 4 * case["nx"] * case["ny"] * case["nz"]
    evals = {"forces": 1, "snapshot": case.get("steps", 0) + 1}.get(case["do"], case.get("steps", 0) + 1)
    flops = n * _pairs_per_atom(case["pot"]) * PAIR_FLOPS[case["pot"]] * evals
    if case["do"] == "forces":
        return dict(bytes=n * (24 + 4 + 4 + 24), flops=flops)
    return dict(bytes=n * (48 + 4 + 48 + (24 if n <= DUMP_ATOMS and case["do"] == "dynamics" else 0)), flops=flops)


# -------------------------------------------------------------------- exact
def _natural_spline(y, h):
    """Second derivatives of the natural cubic spline of y on a uniform grid."""
    n = len(y)
    rhs = 6.0 * (y[2:] - 2.0 * y[1:-1] + y[:-2]) / (h * h)
    c, d = np.zeros(n - 2), np.zeros(n - 2)
    b = 4.0
    c[0], d[0] = 1.0 / b, rhs[0] / b
    for k in range(1, n - 2):
        m = 1.0 / (b - c[k - 1])
        c[k], d[k] = m, (rhs[k] - d[k - 1]) * m
    out = np.zeros(n)
    for k in range(n - 3, -1, -1):
        out[k + 1] = d[k] - c[k] * out[k + 2]
    return out


class _Table:
    """A natural cubic spline on a uniform grid, evaluated in torch."""

    def __init__(self, y, h):
        self.h, self.np = h, (y, _natural_spline(y, h))
        self.y, self.dd = (torch.from_numpy(t).cuda() for t in self.np)

    def __call__(self, x):
        q = x / self.h
        k = q.floor().long().clamp_(0, len(self.y) - 2)
        b = q - k
        a = 1.0 - b
        y0, y1, d0, d1 = self.y[k], self.y[k + 1], self.dd[k], self.dd[k + 1]
        h2 = self.h * self.h / 6.0
        return (a * y0 + b * y1 + ((a ** 3 - a) * d0 + (b ** 3 - b) * d1) * h2,
                (y1 - y0) / self.h + ((3 * b * b - 1) * d1 - (3 * a * a - 1) * d0) * self.h / 6.0)

    def host(self, x):
        k = np.clip(np.floor(x / self.h).astype(np.int64), 0, len(self.np[0]) - 2)
        b = x / self.h - k
        a = 1.0 - b
        y, dd = self.np
        return a * y[k] + b * y[k + 1] + ((a ** 3 - a) * dd[k] + (b ** 3 - b) * dd[k + 1]) * self.h * self.h / 6.0


_EAM = []


def _eam_functions():
    """The analytic EAM as its file defines it: f, phi, F on 10000 points,
    resampled by splines onto a grid of r^2 with two zero points beyond the
    cutoff; r phi is what the file holds, phi(0) a large number."""
    if not _EAM:
        rc, nr = 5.5, 10000
        dr = rc / (nr - 1)
        r = np.arange(nr) * dr
        t = np.clip((r - 5.0) / 0.5, 0.0, 1.0)
        cut = 1.0 - 3.0 * t * t + 2.0 * t ** 3
        e = np.exp(-1.36 * (r - 2.556))
        f = np.exp(-3.3 * (r / 2.556 - 1.0)) * cut
        phi = 0.35 * (e * e - 2.0 * e) * cut
        phi[0] = np.finfo(np.float32).max
        dr2 = ((nr + 1) * dr) ** 2 / (nr + 1)
        r2 = np.arange(nr + 2) * dr2
        tables = [_Table(_Table(np.concatenate([y, [0.0, 0.0]]), dr).host(np.sqrt(r2)), dr2) for y in (f, phi)]
        rho = np.arange(10000) * 0.012
        _EAM.extend(tables + [_Table(-1.1 * np.sqrt(rho), 0.012)])
    return _EAM


class _Exact:
    """Velocity-Verlet dynamics in 64 bits on plain torch: every pair once, on
    a list of radius cutoff + 0.7 A made anew when an atom has moved 0.3 A."""

    def __init__(self, pots, masses, box, pbc, x, v, kind=None):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.box, self.pbc, self.pots = t(box), torch.tensor(pbc, device="cuda"), pots
        self.x, self.v = t(x), t(v)
        self.kind = None if kind is None else t(kind.astype(np.int64))
        m = np.asarray(masses) / MASS_UNIT
        self.m = t((m[np.zeros(len(x), int)] if kind is None else m[kind])[:, None])
        self.rl = max(p[-1] for p in pots.values()) + 0.7
        self.x_list = None

    def _delta(self, i, j):
        d = self.x[i] - self.x[j]
        return torch.where(self.pbc, d - self.box * torch.round(d / self.box), d)

    def _list(self):
        w = torch.where(self.pbc, self.x - self.box * torch.floor(self.x / self.box), self.x)
        lo = torch.where(self.pbc, torch.zeros_like(self.box), w.min(0).values)
        span = torch.where(self.pbc, self.box, w.max(0).values - lo + 1e-9)
        nc = [max(1, int(s / self.rl)) for s in span.tolist()]
        n = len(w)
        if any(p and c < 3 for p, c in zip(self.pbc.tolist(), nc)):      # a short box: all pairs, in slices
            got = []
            for a in range(0, n, 2048):
                i = torch.arange(a, min(a + 2048, n), device="cuda")
                ii, jj = i.repeat_interleave(n), torch.arange(n, device="cuda").repeat(len(i))
                keep = ii < jj
                ii, jj = ii[keep], jj[keep]
                near = self._delta(ii, jj).square().sum(1) < self.rl ** 2
                got.append(torch.stack([ii[near], jj[near]]))
            self.pairs = torch.cat(got, 1)
        else:
            nct = torch.tensor(nc, device="cuda")
            ic = torch.minimum(((w - lo) / span * nct).long(), nct - 1)
            flat = (ic[:, 0] * nc[1] + ic[:, 1]) * nc[2] + ic[:, 2]
            order = torch.argsort(flat, stable=True)
            count = torch.bincount(flat, minlength=nc[0] * nc[1] * nc[2])
            start = torch.cumsum(count, 0) - count
            most = int(count.max())
            slot = torch.arange(n, device="cuda") - start[flat[order]]
            table = torch.full((len(count), most), -1, dtype=torch.long, device="cuda")
            table[flat[order], slot] = order
            got, me = [], torch.arange(n, device="cuda")
            for code in range(27):
                o = torch.tensor([code // 9 - 1, code // 3 % 3 - 1, code % 3 - 1], device="cuda")
                jc = ic + o
                inside = ((jc >= 0) & (jc < nct) | self.pbc).all(1)
                jc = torch.remainder(jc, nct)
                cand = table[(jc[:, 0] * nc[1] + jc[:, 1]) * nc[2] + jc[:, 2]]
                ok = (cand > me[:, None]) & inside[:, None]
                ii = me[:, None].expand_as(cand)[ok]
                jj = cand[ok]
                near = self._delta(ii, jj).square().sum(1) < self.rl ** 2
                got.append(torch.stack([ii[near], jj[near]]))
            self.pairs = torch.cat(got, 1)
        self.x_list = self.x.clone()

    def forces(self):
        if self.x_list is None or float((self.x - self.x_list).square().sum(1).max()) > 0.09:
            self._list()
        F = torch.zeros_like(self.x)
        pe, vir = 0.0, 0.0
        allow = self.pairs
        for (a, b), pot in self.pots.items():
            i, j = allow
            if self.kind is not None:
                ki, kj = self.kind[i], self.kind[j]
                pick = (ki == a) & (kj == b) | (ki == b) & (kj == a)
                i, j = i[pick], j[pick]
            d = self._delta(i, j)
            r2 = d.square().sum(1)
            near = r2 < pot[-1] ** 2
            i, j, d, r2 = i[near], j[near], d[near], r2[near]
            if pot[0] == "lj":
                s2 = pot[1] ** 2 / r2
                s6 = s2 ** 3
                f, e = 48.0 * pot[2] / r2 * (s6 * s6 - 0.5 * s6), 4.0 * pot[2] * (s6 * s6 - s6)
            elif pot[0] == "morse":
                r = r2.sqrt()
                e1 = torch.exp(-pot[2] * (r - pot[3]))
                f, e = 2.0 * pot[1] * pot[2] / r * (e1 * e1 - e1), pot[1] * (e1 * e1 - 2.0 * e1)
            else:
                tf, tphi, tF = _eam_functions()
                rho, drho = tf(r2)
                phi, dphi = tphi(r2)
                dens = torch.zeros(len(self.x), dtype=torch.float64, device="cuda")
                dens.index_add_(0, i, rho)
                dens.index_add_(0, j, rho)
                emb, demb = tF(dens)
                if self.kind is not None:
                    emb, demb = emb * (self.kind == a), demb * (self.kind == a)
                f, e = -2.0 * ((demb[i] + demb[j]) * drho + dphi), phi
                pe = pe + emb.sum()
            F.index_add_(0, i, f[:, None] * d)
            F.index_add_(0, j, -f[:, None] * d)
            pe, vir = pe + e.sum(), vir + (f * r2).sum()
        self.F, self.pe, self.virial = F, pe, vir

    def temperature(self):
        return float((self.m * self.v.square()).sum()) / (3.0 * len(self.x) * KB)

    def steps(self, count, dt, tau=0.0, T0=0.0):
        for _ in range(count):
            if tau > 0.0:
                self.v = self.v * math.sqrt(1.0 + dt / tau * (T0 / self.temperature() - 1.0))
            self.v = self.v + 0.5 * dt / self.m * self.F
            self.x = self.x + dt * self.v
            self.forces()
            self.v = self.v + 0.5 * dt / self.m * self.F

    def wrapped(self):
        """Positions as they are stored: inside the box along periodic axes."""
        w = torch.where(self.x < 0.0, self.x + self.box, self.x)
        w = torch.where(w >= self.box, w - self.box, w)
        return torch.where(self.pbc, w, self.x).cpu().numpy()

    def thermo(self):
        T = self.temperature()
        return np.array([1.5 * len(self.x) * KB * T, T, float(self.pe), float(self.virial)])


def _pots_of(pot):
    rc = POTS[pot]["rc"] if pot in POTS else 0.0
    if pot == "cuar":
        return {(0, 0): ("eam", 5.5), (1, 1): ("lj",) + CUAR["ar"], (0, 1): ("lj",) + CUAR["mix"]}, CUAR["masses"]
    return {(0, 0): {"lj": ("lj", LJ_SIG, LJ_EPS, rc), "morse": ("morse",) + MORSE + (rc,), "eam": ("eam", rc)}[pot]}, \
        (POTS[pot]["mass"],)


def exact(case, seed):
    """The same passes in 64 bits; no value for the storage order, and none
    for the two-temperature runs (their substeps are sequential)."""
    do = case["do"]
    if do == "ttm":
        return None
    if do == "served":
        out, th = {"x": [], "v": [], "F": []}, []
        for pot, x, v, box, kind in _served_jobs(case, seed):
            pots, masses = _pots_of(pot)
            e = _Exact(pots, masses, box, (True,) * 3, x, v, kind if pot == "cuar" else None)
            e.forces()
            th.append(e.thermo())
            e.steps(case["steps"], CUAR["dt"] if pot == "cuar" else POTS[pot]["dt"])
            th.append(e.thermo())
            out["x"].append(e.wrapped())
            out["v"].append(e.v.cpu().numpy())
            out["F"].append(e.F.cpu().numpy())
        return dict({k: np.concatenate(a) for k, a in out.items()}, order=None, thermo=np.stack(th))
    box, pbc, x, v = _system(case, seed)
    pots, masses = _pots_of(case["pot"])
    e = _Exact(pots, masses, box, pbc, x, v)
    e.forces()
    if do == "forces":
        P = POTS[case["pot"]]
        nc = (box / P["rc"]).astype(np.int64)
        ic = np.clip(np.floor(x / (box / nc)).astype(np.int64), 0, nc - 1)
        order = np.argsort(ic[:, 2] + nc[2] * (ic[:, 1] + nc[1] * ic[:, 0]), kind="stable")
        return dict(F=np.ascontiguousarray(e.F.cpu().numpy()[order].T), pe=np.array([float(e.pe)]))
    e.steps(case["steps"], POTS[case["pot"]]["dt"], case["tau"], case["T"])
    out = dict(order=None, x=e.wrapped(), v=e.v.cpu().numpy(), thermo=e.thermo())
    if do == "dynamics" and len(x) <= DUMP_ATOMS:
        out["F"] = e.F.cpu().numpy()
    return out
