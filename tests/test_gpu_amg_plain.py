"""Launch-saving forms that their first tests no longer reach, each on and off where the forms differ in their launches:
the plain aggregation's V-cycle (ANB_AMG_SMOOTHED=0 for the pressure; mom_amg), the smoothed aggregation's cluster
tail, and the FP64 momentum loop above the one-kernel limit.

The plain forms do the per-level kernels' arithmetic in the same order, so the fields must be equal bit for bit;
SELL-32 coarse levels and the smoothed tail sum a row in another order: the preconditioner is the same to
rounding and every solve reaches 1e-10, which leaves the fields equal to 1e-7 (FP64) and 1e-5 (mixed, whose
FP32 inner solves round differently), as in test_gpu_amg_tail."""
import os

import numpy as np
import pytest

import anabasis_b200 as anb
from tests.cases import channel, initial_state

pytestmark = pytest.mark.gpu

PRM = dict(rho=1.0, mu=1e-3, u_relax=0.7, p_relax=0.3, n_nonorth_corr=1)
HUGE = 1 << 30


@pytest.fixture(scope="module")
def case():
    # 36k cells: five or six plain levels, so 3000 rows splits the CSR levels between launches and tail
    m, bc, _ = channel(nx=60, ny=25, nz=24, jitter=0.15, seed=3, obstacle=True)
    return m, bc, initial_state(m, bc)


def run(case, steps=4, env=None, **kw):
    """Fields, pressure iterations a step, and the launches of one extra step (ungraphed V-cycles)."""
    m, bc, init = case
    env = {k: str(v) for k, v in (env or {}).items()}
    os.environ.update(env)
    try:
        s = anb.Solver(m, anb.default_params(**PRM, **kw))
        s.set_bc(bc)
        s.set_state(*init)
        _, st = s.iterate(steps)
        g = s.get_state()
        n0 = anb.lib().anb_launch_count()
        s.iterate(1)
        return g, [x["its_p_total"] for x in st], anb.lib().anb_launch_count() - n0
    finally:
        for k in env:
            os.environ.pop(k)


def same(a, b):
    return all(np.array_equal(a[0][k], b[0][k]) for k in ("u", "v", "w", "p", "phi")) and a[1] == b[1]


@pytest.mark.parametrize("kw", [dict(), dict(precision=1), dict(mom_amg=1)])
def test_plain_tail_and_fused_forms(case, kw):
    base = dict(ANB_AMG_SMOOTHED=0, ANB_NO_GRAPH=1, ANB_NO_LOOP_GRAPH=1)
    ref = run(case, env=dict(base, ANB_AMG_TAIL_ROWS=0, ANB_AMG_FUSED_DOWN_ROWS=0), **kw)
    launches = {ref[2]}
    for tail, fused in ((3000, 0), (HUGE, 0), (0, HUGE), (3000, HUGE), (1024, 65536)):
        got = run(case, env=dict(base, ANB_AMG_TAIL_ROWS=tail, ANB_AMG_FUSED_DOWN_ROWS=fused), **kw)
        assert same(got, ref), (tail, fused)
        assert got[2] < ref[2], (tail, fused)  # the form did run
        launches.add(got[2])
    assert len(launches) >= 4


@pytest.mark.parametrize("kw", [dict(), dict(precision=1), dict(mom_amg=1)])
def test_plain_sell_levels(case, kw):
    base = dict(ANB_AMG_SMOOTHED=0, ANB_AMG_TAIL_ROWS=1024)
    ref = run(case, env=dict(base, ANB_AMG_SELL_MIN_ROWS=HUGE), **kw)
    got = run(case, env=dict(base, ANB_AMG_SELL_MIN_ROWS=1000), **kw)
    assert got[2] != ref[2]  # the form did run (its sums may round to the same bits in FP32)
    assert all(abs(a - b) <= 2 for a, b in zip(got[1], ref[1]))
    scale = max(np.abs(ref[0][k]).max() for k in "uvw")
    tol = 1e-5 if kw.get("precision") else 1e-7
    for k in "uvw":
        assert np.abs(got[0][k] - ref[0][k]).max() <= tol * scale, k


@pytest.mark.parametrize("precision", [0, 1])
def test_smoothed_tail(case, precision):
    base = dict(ANB_NO_GRAPH=1, ANB_NO_LOOP_GRAPH=1)
    ref = run(case, env=dict(base, ANB_SA_TAIL_ROWS=0), precision=precision)
    scale = max(np.abs(ref[0][k]).max() for k in "uvw")
    tol = 1e-5 if precision else 1e-7
    for rows in (100, 1024, HUGE):
        got = run(case, env=dict(base, ANB_SA_TAIL_ROWS=rows), precision=precision)
        assert got[2] < ref[2] or rows == 100, rows
        assert all(abs(a - b) <= 2 for a, b in zip(got[1], ref[1])), rows
        for k in "uvw":
            assert np.abs(got[0][k] - ref[0][k]).max() <= tol * scale, (rows, k)
    # one settles into the graphs as well: the same kernels, the same bits
    a = run(case, env=dict(ANB_SA_TAIL_ROWS=1024), precision=precision)
    b = run(case, env=dict(base, ANB_SA_TAIL_ROWS=1024), precision=precision)
    assert same(a, b)


def test_fp64_momentum_loop_graph():
    # above the one-kernel limit of 101,000 rows (three components on 148 SMs) the momentum solve is a loop graph,
    # which replays the kernels of the host loop: the same bits and iterations
    m, bc, _ = channel(nx=104, ny=33, nz=33, jitter=0.15, seed=2, obstacle=True)
    assert m.n_cells > 102000
    c = (m, bc, initial_state(m, bc))
    assert same(run(c, 3), run(c, 3, dict(ANB_NO_LOOP_GRAPH=1)))
