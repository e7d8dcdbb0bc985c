"""Smoothed-aggregation preconditioner of the pressure CG: at the edges of its row and level sizes
(one coarsening step, tails of warps and blocks, jittered hexes and tets, FP64 and FP32 storage) it
must leave the solution of A x = b alone and converge about as fast as a multigrid does.

Tolerances, fixed before the first run: the solve stops at |r| <= 1e-13 |b|; the residual recomputed
here in FP64 from the assembled coefficients may differ from the recursive one by rounding, about
cond-free eps * sum |a| |x|, so 1e-11 |b| is asked.  A V-cycle-preconditioned CG gains a digit in about
three iterations on such grids; 60 for 13 digits is the bound (the Jacobi CG needs hundreds)."""
import numpy as np
import pytest

import anabasis_b200 as anb
from tests.cases import channel, random_state

pytestmark = pytest.mark.gpu

MESHES = [dict(nx=11, ny=4, nz=3), dict(nx=33, ny=4, nz=1), dict(nx=23, ny=9, nz=7, jitter=0.15, seed=1),
          dict(nx=41, ny=16, nz=17, jitter=0.1, seed=2), dict(nx=7, ny=5, nz=5, tets=True),
          dict(nx=19, ny=9, nz=8, jitter=0.12, seed=3, tets=True)]


@pytest.mark.parametrize("kw", MESHES)
def test_pressure_solve(kw):
    m, bc, _ = channel(**kw)
    C, I = m.n_cells, m.n_internal
    t = m.topology()
    o, n = t["owner"][:I], t["neighbour"]
    s = anb.Solver(m, anb.default_params(mu=1e-3, p_tol=0.0, p_rel_tol=1e-13))
    s.set_bc(bc)
    u, v, w, p = random_state(m, 4)
    rau = 1e-2 * (1 + 0.5 * np.random.default_rng(5).random(C))
    a = s.debug_pressure(u, v, w, p, rau)
    b = np.random.default_rng(6).standard_normal(C) * a["diag"].mean()
    x, its, _ = s.debug_pressure_solve(b, np.zeros(C))
    r = b - a["diag"] * x
    np.subtract.at(r, o, a["a_pn"] * x[n])
    np.subtract.at(r, n, a["a_pn"] * x[o])
    assert np.linalg.norm(r) <= 1e-11 * np.linalg.norm(b), (C, its)
    assert its <= 60 or C <= 160, (C, its)


@pytest.mark.parametrize("kw", MESHES[2:])
def test_mixed_precision_fields(kw):
    # FP32 storage of the same hierarchy inside the FP64 defect correction: 1e-5 as in test_gpu_mixed
    m, bc, _ = channel(**kw)
    out = []
    for precision in (0, 1):
        s = anb.Solver(m, anb.default_params(mu=1e-3, u_relax=0.7, p_relax=0.3, precision=precision))
        s.set_bc(bc)
        s.set_state(*(0.2 * f for f in random_state(m, 7)))
        s.iterate(3)
        out.append(s.get_state())
    scale = max(np.abs(out[0][k]).max() for k in "uvw")
    for k in "uvw":
        assert np.abs(out[0][k] - out[1][k]).max() <= 1e-5 * scale, k


@pytest.mark.parametrize("precision", [0, 1])
def test_stale_hierarchy(precision):
    """Coarse levels kept for four steps under a matrix that changes every step: the preconditioner must stay
    symmetric (the finest Q follows the matrix), so the fields are those of a refresh every step and the
    iterations grow mildly.  Both solve to 1e-14: 1e-8 as in test_gpu_parity; a stale V-cycle costs a few
    iterations a solve, twice the fresh count is the bound."""
    m, bc, _ = channel(nx=41, ny=16, nz=17, jitter=0.1, seed=2)
    u, v, w, p = random_state(m, 7)
    got = []
    for every in (1, 4):
        s = anb.Solver(m, anb.default_params(mu=1e-3, u_relax=0.7, p_relax=0.3, vel_tol=1e-14, p_tol=1e-14,
                                             vel_maxit=2000, precision=precision, p_amg_rebuild_every=every))
        s.set_bc(bc)
        s.set_state(0.2 * u, 0.2 * v, 0.2 * w, 0.2 * p)
        _, st = s.iterate(6)
        got.append((s.get_state(), sum(x["its_p_total"] for x in st), [x["status"] for x in st]))
    scale = max(np.abs(got[0][0][k]).max() for k in "uvw")
    for k in "uvw":
        assert np.abs(got[0][0][k] - got[1][0][k]).max() <= 1e-8 * scale, k
    assert got[1][1] <= 2 * got[0][1] and not any(got[1][2]), got
