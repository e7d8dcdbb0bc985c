"""The dynamic shared memory a kernel may have is an attribute of the function, which all contexts of a process
share, so a launch must never set it to its own need: allow_smem (csrc/device.cuh) takes it as a constant of the
kernel, and is the one place that sets it (CPU).  On the GPU two contexts whose refresh products need different
amounts of it, both above the default limit, solve at the same time and get the serial runs' bits."""
import threading
from pathlib import Path

import numpy as np
import pytest

import anabasis_b200 as anb

CSRC = Path(__file__).resolve().parents[1] / "anabasis_b200" / "csrc"


def test_one_place_sets_the_limit():
    users = [p.name for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh", ".hpp", ".cpp")
             and "cudaFuncAttributeMaxDynamicSharedMemorySize" in p.read_text()]
    assert users == ["device.cuh"]
    assert "template <size_t kBytes, class K>\ncudaError_t allow_smem(K* kern)" in (CSRC / "device.cuh").read_text()


@pytest.mark.gpu
def test_two_contexts_in_two_threads():
    cases = []
    for n in (64, 80):
        m = anb.HostMesh.channel(n, n, n, lx=1.0, ly=1.0, lz=1.0, jitter=0.1, seed=1)
        F = m.n_faces
        rng = np.random.default_rng(n)
        cases.append((m, dict(cell_source=rng.standard_normal(m.n_cells), bc_type=np.zeros(F, np.int32),
                              bc_value=np.zeros(F), gamma_face=np.ones(F), laplacian_nonorth=False)))
    want = [anb.Solver(m, anb.default_params()).scalar_elliptic_solve(**a)[0] for m, a in cases]
    got = [[], []]
    start = threading.Barrier(2)

    def work(k):
        m, a = cases[k]
        s = anb.Solver(m, anb.default_params())
        start.wait()
        for _ in range(6):
            got[k].append(s.scalar_elliptic_solve(**a)[0])

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert len(got[k]) == 6 and all(np.array_equal(x, want[k]) for x in got[k])
