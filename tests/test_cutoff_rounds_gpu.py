"""GPU: pairs at the cutoff in mixed precision.  The list walk takes entries
in rounds of four, decides the cutoff in binary32 and corrects the entries
near it by binary64: clusters of a centre and m atoms (m = 1..9: full
rounds, remainders, one and several near entries a round) on a sphere whose
radius differs from the cutoff by 1e-9 to 3e-6 of it, either way.

Tolerances: forces 1e-5 of max |F|, energy 1e-6 relative (the mixed mode's).
One pair wrongly in or out is over half of max |F| and 1e-3 of the energy."""
import tempfile

import numpy as np
import pytest

from test_parity_oracle_gpu import build_both

pytestmark = pytest.mark.gpu

RC = 3.5


def _clusters(pot):
    rng = np.random.default_rng(71)
    x = []
    centres = [(i, j, k) for i in range(5) for j in range(5) for k in range(5)]
    for c, ijk in enumerate(centres):
        # the centres differ in their place within the cells
        o = 12.0 * np.array(ijk) + 6.0 + rng.uniform(-0.4, 0.4, 3)
        dirs = []
        while len(dirs) < 1 + c % 9:
            u = rng.standard_normal(3)
            u /= np.linalg.norm(u)
            if all(np.dot(u, w) < 0.7 for w in dirs):
                dirs.append(u)
        eps = 10.0 ** rng.uniform(-9.0, -5.5, len(dirs)) * rng.choice([-1.0, 1.0], len(dirs))
        x += [o] + [o + RC * (1.0 + e) * u for u, e in zip(dirs, eps)]
    x = np.array(x)
    n = len(x)
    return dict(box=(60.0,) * 3, pbc=(1, 1, 1), kinds=[("Cu", 63.546)], pots=[pot], x=x, v=np.zeros((n, 3)),
                kind=np.zeros(n, np.uint32), group=np.zeros(n, np.int32), dt=0.001)


@pytest.mark.parametrize("pot", [("lj", 0, 0, 2.4, 0.4, RC), ("morse", 0, 0, 0.3429, 1.3588, 2.866, RC)],
                         ids=["lj", "morse"])
def test_pairs_at_cutoff(gpu_lib, pot):
    spec = _clusters(pot)
    with tempfile.TemporaryDirectory() as work:
        md, o = build_both(gpu_lib, spec, work, precision=1)
        gpu_lib.fmd_dync_integrate(md, -1, 0.0, spec["dt"])
        g = gpu_lib.dump(md)
        o.forces(-1)
        r = o.dump()
        np.testing.assert_array_equal(g["id"], r["id"])
        assert np.abs(g["F"] - r["F"]).max() <= 1e-5 * np.abs(r["F"]).max()
        assert abs(g["pe"] - r["pe"]) <= 1e-6 * abs(r["pe"])
        gpu_lib.fmd_free(md)
        o.close()
