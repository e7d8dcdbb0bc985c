"""Device memory of contexts."""
import numpy as np
import pytest

import anabasis_b200 as anb

pytestmark = pytest.mark.gpu


def _free():
    import torch

    return torch.cuda.mem_get_info(0)[0]


def test_small_contexts_hold_little():
    # 12^3 cells need 2.6 MB for the context, 1.8 for the hierarchy and 0.4 for the scalar buffers; with the 2 MB
    # granularity of the allocations and the graphs 14 MB are allowed
    m = anb.HostMesh.channel(12, 12, 12, lx=1.0, ly=1.0, lz=1.0)
    F = m.n_faces

    def make():
        s = anb.Solver(m, anb.default_params())
        s.scalar_elliptic_solve(np.ones(m.n_cells), np.zeros(F, np.int32), np.zeros(F))
        return s

    first = make()  # modules and library state
    before = _free()
    held = [make() for _ in range(12)]
    assert before - _free() <= 12 * 14 * 2**20
    assert first.n_cells == held[0].n_cells
