"""Levels of the smoothed-aggregation hierarchy read back from the device and compared with their definitions."""
import numpy as np
import pytest

import anabasis_b200 as anb
from tests.cases import channel, random_state

pytestmark = pytest.mark.gpu


def hierarchy(mesh, spread=1.0, seed=1, **kw):
    """(levels, Solver, system) of the pressure matrix for an rAU that spreads over `spread`."""
    m, bc, _ = mesh
    s = anb.Solver(m, anb.default_params(mu=1e-3, p_tol=0.0, p_rel_tol=1e-10, **kw))
    s.set_bc(bc)
    rau = 1e-2 * spread ** np.random.default_rng(seed).random(m.n_cells)
    a = s.debug_pressure(*random_state(m, 4), rau)
    b = np.random.default_rng(6).standard_normal(m.n_cells) * a["diag"].mean()
    x, its, _ = s.debug_pressure_solve(b, np.zeros(m.n_cells))
    return s.debug_hierarchy(), s, (a, b, x, its)


@pytest.mark.parametrize("spread", [1.0, 1e3, 1e6])
def test_smoother_weights_are_bounded(spread):
    """w <= 0.9 / a_ii and w sum_j |a_ij| <= 1.99 on every coarse level: then w A < 2 and the cycle is positive
    definite.  The weights are one division each, the row sums n additions: 1e-12 covers both roundings."""
    levels, _, _ = hierarchy(channel(41, 16, 17, jitter=0.1, seed=2), spread)
    assert len(levels) >= 3
    for k, lv in enumerate(levels):
        rows = np.repeat(np.arange(len(lv["diag"])), np.diff(lv["off"]))
        size = np.abs(lv["diag"]) + np.bincount(rows, np.abs(lv["val"]), len(lv["diag"]))
        want = 0.9 / lv["diag"]
        if k > 0:
            want = np.minimum(want, 1.99 / size)
        assert np.abs(lv["weight"] / want - 1).max() <= 1e-12, k
        assert (lv["weight"] * size).max() <= 1.99 * (1 + 1e-12) or k == 0
