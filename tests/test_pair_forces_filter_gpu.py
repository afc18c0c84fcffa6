"""fmdg_pair_forces_noalloc's candidate filter and queue against an all-pairs
sum: sizes around a warp, a block and an atom count per block of two, mixed
LJ / Morse tables, coordinates far from the origin's precision."""
import ctypes as C

import numpy as np
import pytest

from fmd_gb300 import serve

pytestmark = pytest.mark.gpu
LJ = (4 * 0.0104, 3.405 ** 2, 8.5 ** 2, 0.0)
MORSE = (0.3429, 1.3588, 2.866, 8.0 ** 2)


def _reference(x, kind, l, pbc, table):
    """Forces and energy over every pair's nearest image (l > 2 rc along
    periodic axes), in binary64."""
    F, pe = np.zeros_like(x), 0.0
    for i in range(len(x)):
        d = x[i] - x
        d = np.where(pbc, d - l * np.round(d / l), d)
        r2 = (d * d).sum(1)
        r2[i] = np.inf
        for k in range(2):
            cat, p = table[kind[i]][k]
            m = (kind == k) & (r2 < (p[2] if cat == 1 else p[3]))
            q = r2[m]
            if cat == 1:
                s6 = (p[1] / q) ** 3
                f, e = 12 * p[0] / q * (s6 * s6 - 0.5 * s6), p[0] * (s6 * s6 - s6)
            else:
                r = np.sqrt(q)
                e1 = np.exp(-p[1] * (r - p[2]))
                f, e = 2 * p[1] * p[0] / r * (e1 * e1 - e1), p[0] * (e1 * e1 - 2 * e1)
            F[i] += (f[:, None] * d[m]).sum(0)
            pe += 0.5 * e.sum()
    return F, pe


@pytest.mark.parametrize("n,l,open_z,shift", [(1, 18.0, False, 0.0), (31, 20.0, False, 0.0), (33, 25.9, True, 0.0),
                                              (512, 26.0, False, 0.0), (1500, 36.0, True, 0.0),
                                              (1500, 36.0, True, 5000.0)])
@pytest.mark.parametrize("table", [((1, LJ), (1, LJ)), ((3, MORSE), (3, MORSE)), ((1, LJ), (3, MORSE))])
def test_filtered_forces(gpu_lib, n, l, open_z, shift, table):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + int(shift))
    # no two atoms closer than 2 A: sites of a jittered grid
    g = int(np.ceil(n ** (1 / 3)))
    site = np.stack(np.unravel_index(rng.permutation(g ** 3)[:n], (g, g, g)), 1)
    x = (site + 0.5 + rng.uniform(-0.15, 0.15, (n, 3))) * (l / g)
    kind = rng.integers(0, 2, n).astype(np.int32)
    l3, pbc = np.full(3, l), np.array([True, True, not open_z])
    tab = [[table[0], table[1]], [table[1], table[0]]]
    nc = np.maximum(1, (l3 / 8.5).astype(int))
    ic = np.minimum((x / (l3 / nc)).astype(int), nc - 1)
    flat = ic[:, 2] + nc[2] * (ic[:, 1] + nc[1] * ic[:, 0])
    o = np.argsort(flat, kind="stable")
    x, kind, flat = x[o], kind[o], flat[o]
    F0, pe0 = _reference(x, kind, l3, pbc, tab)
    x = x + np.array([0.0, 0.0, shift])          # (open z: the cells do not depend on the origin)
    start = np.concatenate([[0], np.cumsum(np.bincount(flat, minlength=int(nc.prod())))]).astype(np.int32)
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    xs, ks, cs, fs = cuda(x.T), cuda(kind), cuda(start), cuda(flat.astype(np.int32))
    F, pe = torch.zeros((3, n), dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    pairs = (serve.Pair * 4)()
    for a in range(2):
        for b in range(2):
            pairs[2 * a + b].cat = tab[a][b][0]
            for q in range(4):
                pairs[2 * a + b].p[q] = tab[a][b][1][q]
    L = serve.bind(gpu_lib.L)
    L.fmdg_pair_forces_noalloc.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int] + [C.c_void_p] * 8
    p = lambda t: t.data_ptr()  # noqa: E731
    h = lambda a, t: np.ascontiguousarray(a, t).ctypes.data_as(C.c_void_p)  # noqa: E731
    nca, pba = np.ascontiguousarray(nc, np.int32), np.ascontiguousarray(pbc, np.int32)
    la = np.ascontiguousarray(l3, np.float64)
    rc = L.fmdg_pair_forces_noalloc(n, h(nca, np.int32), h(pba, np.int32), h(la, np.float64), 2, C.addressof(pairs), p(xs),
                                    p(ks), p(cs), p(fs), p(F), p(pe), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    # binary64 sums of at most ~300 terms; the shifted coordinates carry
    # 5000 * 2^-53 of rounding into every distance
    tol = 1e-12 if shift == 0.0 else 1e-9
    scale = max(np.abs(F0).max(), 1e-6)
    assert np.abs(F.cpu().numpy().T - F0).max() <= tol * scale
    assert abs(float(pe) - pe0) <= tol * max(abs(pe0), 1e-6)
