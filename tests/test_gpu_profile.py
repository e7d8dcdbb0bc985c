"""Kernel families of the BiCGSTAB are timed in every solve that has one (anb_profile_select)."""
import ctypes as ct

import numpy as np
import pytest

import anabasis_b200 as anb

pytestmark = pytest.mark.gpu

KF_BICG_SPMV, KF_BICG_VECTOR = 6, 12  # include/anb.h


@pytest.mark.parametrize("family", [KF_BICG_SPMV, KF_BICG_VECTOR])
def test_scalar_transport_is_timed(family):
    m = anb.HostMesh.channel(9, 8, 7, lx=1.0, ly=1.0, lz=1.0)
    F = m.n_faces
    args = dict(gamma_face=np.full(F, 0.1), su=np.ones(m.n_cells), bc_type=np.zeros(F, np.int32), bc_value=np.zeros(F),
                nonorth_corr=0)
    s = anb.Solver(m, anb.default_params())
    want = s.scalar_transport_solve(**args)[0]
    anb.lib().anb_profile_select(s._h, family)
    x, info = s.scalar_transport_solve(**args)
    n = ct.c_longlong(0)
    assert anb.lib().anb_profile_read(s._h, ct.byref(n), None, None) == anb.ANB_OK
    assert info["converged"] and n.value >= info["iterations"] > 0
    assert np.abs(x - want).max() <= 1e-7 * np.abs(want).max()  # both to |r| <= 1e-10, |x| about 0.1
