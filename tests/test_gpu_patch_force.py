"""Patch-force integral at the edges of its launch shapes (one block up to 512 faces, several blocks
with a cross-block combination beyond): every sum against the CPU oracle.

Tolerance, fixed before the first run: the sums differ from the oracle's serial ones by their order only,
so by at most n eps of the sum of absolute terms; with n < 5000 faces 5000 * 1.1e-16 < 1e-12 of that
scale."""
import numpy as np
import pytest

import anabasis_b200 as anb
import oracle
from tests.cases import channel, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz", [(1, 1), (4, 8), (3, 11), (16, 32), (19, 27), (32, 24), (40, 31), (50, 45)])
def test_inlet_force(ny, nz):
    m, bc, _ = channel(nx=3, ny=ny, nz=nz, jitter=0.1, seed=1)
    f = random_state(m, 2)
    s = anb.Solver(m, anb.default_params(mu=1e-3))
    s.set_bc(bc)
    s.set_state(*f)
    o = oracle.Oracle(m.topology())
    names = m.topology()["patch_names"]
    for name in ("patch_1_0", "patch_0_0"):
        k = names.index(name)
        a = s.patch_force(k, -1)
        b = o.patch_force(k, -1, 1e-3, *f)
        assert a["n_faces"] == int(m.topology()["patch_size"][k])
        scale = max(np.abs(f[3]).max() * a["area"], np.abs(a["Fv"]).max())
        for i, q in enumerate(("Fp", "Fv", "F")):
            assert np.abs(np.array(a[q]) - b[3 * i:3 * i + 3]).max() <= 1e-12 * scale, (name, q)
        assert abs(a["area"] - b[9]) <= 1e-12 * a["area"]
