"""Pressure and scalar solves on stretched grids and with spread coefficients, smoothed aggregation (its refusals
and grouped levels among them) against the plain aggregation (ANB_AMG_SMOOTHED=0).

Tolerances, fixed before the first run: the CG stops at |r| <= 1e-11 |b|; the recursive residual leaves the true
one by rounding, at most a few eps of | |A| |x| | an iteration, for which 8 eps its is taken.  Two solutions whose
residuals are that small differ by no bound free of the condition number, so the scalar solves compare residuals
too, through the matrix of the plain run's own assembly.  Iterations: with spread coefficients the smoothed
hierarchy needs up to 1.4 times those of the plain one, so twice and five more are allowed."""
import os

import numpy as np
import pytest

import anabasis_b200 as anb
from tests.cases import random_state

pytestmark = pytest.mark.gpu


def _mesh(nx, ny, nz, ax, az, tets=False):
    """Cells ax times as long and az times as deep as high."""
    h = 0.41 / ny
    return anb.HostMesh.channel(nx, ny, nz, lx=ax * h * nx, ly=0.41, lz=az * h * nz, jitter=0.02, seed=1, tets=tets)


def _bc(m, tmp_path):
    f = tmp_path / "c.bc"
    f.write_text("velocity patch_0_0 wall_noslip\nvelocity patch_1_0 wall_noslip\nvelocity patch_2_0 zero_gradient\n"
                 "pressure patch_0_0 zero_gradient\npressure patch_1_0 zero_gradient\npressure patch_2_0 fixed_value 0.0\n")
    return m.evaluate_bc(f)


def _pressure(m, bc, spread, smoothed):
    os.environ["ANB_AMG_SMOOTHED"] = smoothed
    try:
        s = anb.Solver(m, anb.default_params(mu=1e-3, p_tol=0.0, p_rel_tol=1e-11, p_maxit=2000))
        s.set_bc(bc)
        C, I = m.n_cells, m.n_internal
        rau = 1e-2 * spread ** np.random.default_rng(5).random(C)
        a = s.debug_pressure(*random_state(m, 4), rau)
        b = np.random.default_rng(6).standard_normal(C) * np.abs(a["diag"])
        x, its, _ = s.debug_pressure_solve(b, np.zeros(C))
    finally:
        del os.environ["ANB_AMG_SMOOTHED"]
    t = m.topology()
    o, n = t["owner"][:I], t["neighbour"]
    r, size = b - a["diag"] * x, np.abs(a["diag"] * x)
    for i, j in ((o, n), (n, o)):
        np.subtract.at(r, i, a["a_pn"] * x[j])
        np.add.at(size, i, np.abs(a["a_pn"] * x[j]))
    tol = 1e-11 * np.linalg.norm(b) + 8 * its * 2.2e-16 * np.linalg.norm(size)
    assert np.linalg.norm(r) <= tol, (its, np.linalg.norm(r), tol)
    return its


# (ax, az): needles, pancakes (30 x 30: the second level is refused)
@pytest.mark.parametrize("grid", [(30, 26, 26), (52, 47, 46)])
@pytest.mark.parametrize("ax,az", [(5, 1), (10, 1), (30, 1), (5, 5), (10, 10), (30, 30)])
def test_stretched(grid, ax, az, tmp_path):
    m = _mesh(*grid, ax, az)
    bc = _bc(m, tmp_path)
    assert _pressure(m, bc, 1.0, "1") <= 2 * _pressure(m, bc, 1.0, "0") + 5


@pytest.mark.parametrize("n", [17, 26, 48])
@pytest.mark.parametrize("spread", [1e3, 1e4, 1e5])
def test_spread_coefficients(n, spread, tmp_path):
    m = _mesh(n, n, n, 1, 1)
    bc = _bc(m, tmp_path)
    assert _pressure(m, bc, spread, "1") <= 2 * _pressure(m, bc, spread, "0") + 5


@pytest.mark.parametrize("tets", [False, True])
@pytest.mark.parametrize("spread", [1e3, 1e5])
def test_elliptic_with_spread_gamma(tets, spread):
    m = _mesh(12, 12, 12, 1, 1, tets) if tets else _mesh(30, 30, 30, 1, 1)
    F = m.n_faces
    rng = np.random.default_rng(3)
    args = dict(cell_source=rng.standard_normal(m.n_cells), bc_type=np.zeros(F, np.int32), bc_value=np.zeros(F),
                gamma_face=spread ** rng.random(F), laplacian_nonorth=False, abs_tol=0.0, rel_tol=1e-11)
    out = {}
    for smoothed in ("1", "0"):
        os.environ["ANB_AMG_SMOOTHED"] = smoothed
        try:
            out[smoothed] = anb.Solver(m, anb.default_params()).scalar_elliptic_solve(**args)
        finally:
            del os.environ["ANB_AMG_SMOOTHED"]
        assert out[smoothed][1]["converged"]
    assert out["1"][1]["iterations"] <= 2 * out["0"][1]["iterations"] + 5
    # gamma >= 1: the error is at most |r| / (the smallest eigenvalue of the Laplacian with gamma = 1 times the
    # cell volume), 1e-11 |b| h^-2 / pi^2 / 3 < 1e-8 of the solution's scale on 30 cells a side
    x, y = out["1"][0], out["0"][0]
    assert np.linalg.norm(x - y) <= 1e-7 * np.linalg.norm(y)
