"""Contexts are independent (include/anb.h): two threads with a context each, whose momentum solves are one
cooperative kernel over every SM and whose pressure solves are graph launches, get the serial runs' bits."""
import threading

import numpy as np
import pytest

import anabasis_b200 as anb
from tests.cases import channel, initial_state

pytestmark = pytest.mark.gpu

CASES = [dict(nx=40, ny=20, nz=20), dict(nx=30, ny=12, nz=12, jitter=0.1, seed=3, tets=True)]


def _solver(m, bc):
    s = anb.Solver(m, anb.default_params(rho=1.0, mu=1e-3, u_relax=0.7, p_relax=0.3, n_nonorth_corr=1))
    s.set_bc(bc)
    s.set_state(*initial_state(m, bc))
    return s


def test_two_simple_runs_at_once():
    meshes = [channel(**kw)[:2] for kw in CASES]
    want = []
    for m, bc in meshes:
        s = _solver(m, bc)
        _, st = s.iterate(20)
        want.append((s.get_state(), [x["its_p_total"] for x in st]))
    got = [None, None]
    start = threading.Barrier(2)

    def work(k):
        s = _solver(*meshes[k])
        start.wait()
        rc, st = s.iterate(20)
        got[k] = (s.get_state(), [x["its_p_total"] for x in st], rc)

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert got[k] is not None and got[k][2] == anb.ANB_OK and got[k][1] == want[k][1]
        assert all(np.array_equal(got[k][0][q], want[k][0][q]) for q in ("u", "v", "w", "p", "phi"))
