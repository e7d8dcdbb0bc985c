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


class Hub:
    """A channel mesh with the cells of a box merged into one cell of many faces."""

    def __init__(self, m, lo, hi):
        t, g = m.topology(), m.geometry()
        cc = g["cc"].reshape(-1, 3)
        inside = ((cc > lo) & (cc < hi)).all(1)
        new = np.where(inside, 0, np.cumsum(~inside)).astype(np.int32)  # the hub is cell 0
        I, F = m.n_internal, m.n_faces
        own, nei = new[t["owner"]], new[t["neighbour"]]
        keep = np.concatenate([own[:I] != nei, np.ones(F - I, bool)])
        pts = [t["face_points"][a:b] for a, b in zip(t["face_offsets"][:-1], t["face_offsets"][1:])]
        swap = np.concatenate([own[:I] > nei, np.zeros(F - I, bool)])
        own[:I], nei = np.minimum(own[:I], nei), np.maximum(own[:I], nei)
        faces = [p[::-1] if s else p for p, s, k in zip(pts, swap, keep) if k]
        self.n_points, self.n_faces, self.n_patches = m.n_points, len(faces), m.n_patches
        self.n_internal, self.n_cells = int(keep[:I].sum()), int(new.max()) + 1
        self.hub_faces = int(((own[:I] == 0) & keep[:I]).sum())
        drop = I - self.n_internal
        self._t = dict(points=t["points"], face_offsets=np.cumsum([0] + [len(f) for f in faces]).astype(np.int32),
                       face_points=np.concatenate(faces).astype(np.int32), owner=own[keep].copy(),
                       neighbour=nei[keep[:I]].copy(), patch_start=t["patch_start"] - np.int32(drop),
                       patch_size=t["patch_size"], patch_names=t["patch_names"])
        self._keep = keep

    def topology(self):
        return self._t

    def bc(self, bc):
        return {k: v[self._keep] if k in "uvwp" else v for k, v in bc.items()}


def _hub():
    m, bc, d = channel(40, 24, 24)
    h = Hub(m, (0.55, 0.1, 0.1), (1.95, 0.31, 0.31))  # rows of hundreds of entries: tables and sorts overflow
    return h, h.bc(bc), d


def _csr(off, col, val, shape):
    from scipy.sparse import csr_matrix

    return csr_matrix((np.asarray(val, float), col, off), shape=shape)


def _pattern(a):
    a = a.tocsr()
    a.sort_indices()
    return a.indptr, a.indices


@pytest.mark.parametrize("name,spread", [("hex", 1.0), ("hex", 1e5), ("tets", 1.0), ("flat", 1.0), ("hub", 1.0)])
def test_levels_are_what_they_are_defined_to_be(name, spread):
    """Patterns exactly; values to 1e-11 of the largest of their row, a sum of at most thousands of products."""
    from scipy.sparse import diags, identity

    mesh = {"hex": lambda: channel(41, 16, 17, jitter=0.1, seed=2), "tets": lambda: channel(19, 9, 8, seed=3, tets=True),
            "flat": lambda: channel(20, 2, 61), "hub": _hub}[name]()
    if name == "hub":
        assert mesh[0].hub_faces > 500
    levels, s, (a, b, x, its) = hierarchy(mesh, spread)
    assert len(levels) >= 3
    kinds = set()
    for k, lv in enumerate(levels[:-1]):
        n, nc = len(lv["diag"]), int(lv["sizes"][2])
        A = (_csr(lv["off"], lv["col"], lv["val"], (n, n)) + diags(lv["diag"])).tocsr()
        ones = _csr(lv["off"], lv["col"], np.ones(len(lv["col"])), (n, n)) + identity(n)
        P0 = _csr(np.arange(n + 1), lv["agg"], np.ones(n), (n, nc))
        smooth = len(lv["p_col"]) > n
        kinds.add(smooth)
        pat = ones @ P0 if smooth else P0
        off, col = _pattern(pat)
        assert np.array_equal(off, lv["p_off"]) and np.array_equal(col, lv["p_col"]), k
        qat = ones @ pat
        off, col = _pattern(qat)
        assert np.array_equal(off, lv["q_off"]) and np.array_equal(col, lv["q_col"]), k
        assert lv["sizes"][3] == np.diff(off).max()
        P = P0 - (2 / 3) * (diags(1 / lv["diag"]) @ A @ P0) if smooth else P0
        got = _csr(lv["p_off"], lv["p_col"], lv["p_val"], (n, nc))
        assert abs(got - P).max() <= 1e-11
        Q = got - diags(lv["weight"]) @ A @ got
        R = _csr(lv["r_off"], lv["r_col"], lv["r_val"], (nc, n))
        off, col = _pattern((pat if k == 0 else qat).T)
        assert np.array_equal(off, lv["r_off"]) and np.array_equal(col, lv["r_col"]), k
        assert abs(R - (got if k == 0 else Q).T).max() <= 1e-11
        nxt = levels[k + 1]
        C = (got.T @ A @ got).tocsr()
        off, col = _pattern((pat.T @ qat))
        rows = np.repeat(np.arange(nc), np.diff(off))
        assert np.array_equal(col[rows != col], nxt["col"]) and np.array_equal(np.diff(nxt["off"]), np.diff(off) - 1), k
        D = _csr(nxt["off"], nxt["col"], nxt["val"], (nc, nc)) + diags(nxt["diag"])
        err = abs(D - C).max(axis=1).toarray().ravel()
        assert (err <= 1e-11 * nxt["diag"]).all(), k
    assert True in kinds


def test_row_too_long_is_refused():
    # spread coefficients break the hub's neighbours into aggregates of their own: a row of more than 787 entries,
    # which no block's shared memory holds; the plain aggregation serves
    with pytest.raises(anb.AnbError, match="no such array"):
        hierarchy(_hub(), 1e3)
