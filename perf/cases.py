"""The work that users of this library have it do, as cases that can be timed and compared.

Every case goes through the public Python mirror of the C ABI (include/anb.h): host arrays in, host
arrays out, one context per state.  The kinds are

  simple     anb_set_state, a few SIMPLE outer iterations, anb_get_state: what a host program does
             between two outputs.  The inner tolerances are 1e-15 absolute, as in the parity runs and in
             the runs that sensitivities start from: the fields are then those of the discrete
             equations, while at the default 1e-10 their eighth digit already depends on the order in
             which the solvers sum.
  force      anb_patch_force on the current state: the monitor that a run calls every few steps.
  adjoint    anb_adjoint_force_grad at a converged state: the gradient of the x-force on the obstacle
             with respect to every Dirichlet velocity value and the viscosity.
  elliptic   anb_scalar_elliptic_solve on a unit cube (the manufactured Poisson programs).
  transport  anb_scalar_transport_solve on a unit cube (the manufactured transport program).

Meshes are those of the library's own channel generator: the 2.5 x 0.41 x 0.41 channel of the
benchmark and the tests (hexes, jittered hexes, hexes split into six tets, with or without the
obstacle), and the unit cube of the scalar programs.
"""
from __future__ import annotations

import functools
import math
import os
import tempfile

import numpy as np

import anabasis_b200 as anb

BC_TEXT = """velocity patch_0_0 wall_noslip
velocity patch_1_0 parabolic_box_inlet 0.41 0.45 y z average_patch_normal
velocity patch_2_0 zero_gradient
pressure patch_0_0 zero_gradient
pressure patch_1_0 zero_gradient
pressure patch_2_0 fixed_value 0.0
"""
BC_OBSTACLE = "velocity patch_3_0 wall_noslip\npressure patch_3_0 zero_gradient\n"

_SIMPLE = dict(kind="simple", nx=0, ny=0, nz=0, jitter=0.15, obstacle=True, tets=False, mixed=False, tol=1e-15,
               n_nonorth=2, n_vel_nonorth=0, n_pressure_corr=0, steps=2)


def _simple(name, **kw):
    return {"name": name, **_SIMPLE, **kw}


def listed():
    return [
        # the force monitor on a coarse grid: one small launch and a read-back, all latency
        dict(name="force_obstacle", kind="force", nx=60, ny=25, nz=24, jitter=0.15, patch="patch_3_0"),
        # the same on the walls of the benchmark's grid (56,000 faces)
        dict(name="force_walls", kind="force", nx=200, ny=70, nz=70, jitter=0.15, patch="patch_0_0"),
        # the plain 16k-cell channel on an orthogonal grid, as its 300-step run works through it
        _simple("simple_16k", nx=40, ny=20, nz=20, jitter=0.0, obstacle=False, steps=10),
        # every corrector loop in use, on a mid-size grid: momentum re-solves and extra pressure passes
        _simple("simple_36k_correctors", nx=60, ny=25, nz=24, n_vel_nonorth=1, n_pressure_corr=1, steps=4),
        # a tetrahedral grid (rows of four), the shape of the scale study
        _simple("simple_tets", nx=90, ny=25, nz=25, tets=True, steps=2),
        # a jittered grid of odd sizes without the obstacle, one non-orthogonal corrector
        _simple("simple_250k", nx=127, ny=45, nz=43, obstacle=False, n_nonorth=1, steps=2),
        # the benchmark: the 970k-cell obstacle channel
        _simple("simple_970k", nx=200, ny=70, nz=70, steps=2),
        # the same grid with mixed precision (FP32 solves inside FP64 defect correction)
        _simple("mixed_970k", nx=200, ny=70, nz=70, mixed=True, steps=2),
        # the largest grid of one card's everyday use, twice the benchmark's
        _simple("simple_2m", nx=250, ny=91, nz=90, steps=1),
        # backward: the force gradient at a converged state
        dict(name="adjoint_36k", kind="adjoint", nx=60, ny=25, nz=24, jitter=0.15),
        # the scalar libraries' manufactured problems
        dict(name="elliptic_48", kind="elliptic", n=48, jitter=0.15, tets=False, n_nonorth=2),
        dict(name="transport_64", kind="transport", n=64, jitter=0.15, tets=False, n_nonorth=2, upwind=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["simple", "simple", "simple", "simple", "mixed", "force", "adjoint", "elliptic", "transport"])
    jitter = rng.choice([0.0, 0.1, 0.15])
    if kind == "elliptic":
        tets = rng.random() < 0.25
        return dict(kind=kind, n=int(_log(rng, 8, 24 if tets else 48)), jitter=jitter, tets=tets,
                    n_nonorth=rng.choice([0, 1, 2, 4]))
    if kind == "transport":
        tets = rng.random() < 0.25
        return dict(kind=kind, n=int(_log(rng, 8, 30 if tets else 64)), jitter=jitter, tets=tets,
                    n_nonorth=rng.choice([0, 1, 2]), upwind=rng.random() < 0.5)
    if kind == "adjoint":
        cells = _log(rng, 1500, 36000)
    else:
        cells = _log(rng, 2000, 1000000)
    ny = max(7, int((cells / 2.9) ** (1 / 3) * rng.uniform(0.85, 1.15)))
    nz = max(5, int((cells / 2.9) ** (1 / 3) * rng.uniform(0.85, 1.15)))
    nx = max(13, int(cells / (ny * nz)))
    if kind == "adjoint":
        return dict(kind=kind, nx=max(nx, 26), ny=max(ny, 9), nz=nz, jitter=jitter)
    if kind == "force":
        return dict(kind=kind, nx=max(nx, 26), ny=max(ny, 9), nz=nz, jitter=jitter,
                    patch=rng.choice(["patch_0_0", "patch_1_0", "patch_3_0"]))
    tets = rng.random() < 0.25
    if tets:
        nx = max(8, nx // 6)
    obstacle = nx >= 26 and ny >= 9 and rng.random() < 0.7
    return dict(_SIMPLE, nx=nx, ny=ny, nz=nz, jitter=jitter, obstacle=obstacle, tets=tets, mixed=kind == "mixed",
                n_nonorth=rng.choice([0, 1, 2]),
                n_vel_nonorth=rng.choice([0, 0, 1]) if kind == "simple" else 0,
                n_pressure_corr=rng.choice([0, 0, 1]), steps=rng.choice([1, 2]))


# ---- meshes (a user's grid lies on disk; it depends on the case alone) --------------------------


@functools.lru_cache(maxsize=2)
def _channel(nx, ny, nz, jitter, obstacle, tets):
    m = anb.HostMesh.channel(nx, ny, nz, jitter=jitter, seed=0, obstacle=obstacle, tets=tets)
    fd, path = tempfile.mkstemp(suffix=".bc")
    with os.fdopen(fd, "w") as f:
        f.write(BC_TEXT + (BC_OBSTACLE if obstacle else ""))
    bc = m.evaluate_bc(path)
    os.unlink(path)
    return m, bc, m.geometry()["cc"].reshape(-1, 3)


@functools.lru_cache(maxsize=2)
def _cube(n, jitter, tets):
    m = anb.HostMesh.channel(n, n, n, lx=1.0, ly=1.0, lz=1.0, jitter=jitter, seed=0, tets=tets)
    return m, m.geometry()


def _grid(case):
    if case["kind"] in ("elliptic", "transport"):
        return _cube(case["n"], case["jitter"], case["tets"])
    return _channel(case["nx"], case["ny"], case["nz"], case["jitter"], case.get("obstacle", True),
                    case.get("tets", False))


def _smooth(rng, x, modes=4):
    """A smooth random field of unit size: a few long waves over the box."""
    f = np.zeros(len(x))
    span = x.max(0) - x.min(0)
    for _ in range(modes):
        k = 2 * math.pi * rng.integers(1, 4, 3) / span
        f += rng.uniform(-1, 1) * np.sin(x @ k + rng.uniform(0, 2 * math.pi))
    return f / math.sqrt(modes)


def _channel_state(rng, bc, m, x):
    """The state that a run starts from, the mean inlet velocity, with smooth disturbances."""
    t = m.topology()
    k = t["patch_names"].index("patch_1_0")
    inlet = slice(int(t["patch_start"][k]), int(t["patch_start"][k] + t["patch_size"][k]))
    u = bc["u"][inlet].mean() * (1 + 0.1 * _smooth(rng, x))
    v = 0.01 * _smooth(rng, x)
    w = 0.01 * _smooth(rng, x)
    p = 0.05 * (1 - x[:, 0] / 2.5) * (1 + 0.1 * _smooth(rng, x))
    return u, v, w, p


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("elliptic", "transport"):
        m, g = _grid(case)
        cc, xf = g["cc"].reshape(-1, 3), g["xf"].reshape(-1, 3)
        s = anb.Solver(m, anb.default_params())
        F = m.n_faces
        bt = np.zeros(F, np.int32)
        bv = _smooth(rng, xf)
        if kind == "elliptic":
            args = dict(cell_source=3 * math.pi**2 * _smooth(rng, cc), bc_type=bt, bc_value=bv,
                        gamma_face=np.ones(F), laplacian_nonorth=True, nonorth_corr=case["n_nonorth"])
        else:
            vel = np.stack([1.0 + xf[:, 1], 0.5 - xf[:, 0], np.full(F, 0.25)], 1)
            flux = (vel * g["sf"].reshape(-1, 3)).sum(1)
            args = dict(gamma_face=np.full(F, 0.1), su=_smooth(rng, cc), bc_type=bt, bc_value=bv, face_flux=flux,
                        sp=np.zeros(m.n_cells), upwind=case["upwind"], diffusion_nonorth=True,
                        nonorth_corr=case["n_nonorth"], abs_tol=1e-13)
        return dict(kind=kind, s=s, args=args)
    m, bc, cc = _grid(case)
    par = dict(rho=1.0, mu=1e-3, u_relax=0.7, p_relax=0.3)
    if kind == "adjoint":
        par.update(n_nonorth_corr=2, vel_tol=1e-14, p_tol=1e-14, vel_maxit=1000)
    if kind == "simple":
        par.update(n_nonorth_corr=case["n_nonorth"], n_vel_nonorth_corr=case["n_vel_nonorth"],
                   n_pressure_corr=case["n_pressure_corr"], vel_tol=case["tol"], p_tol=case["tol"],
                   vel_maxit=5000, p_maxit=20000, precision=1 if case["mixed"] else 0)
    s = anb.Solver(m, anb.default_params(**par))
    names = m.topology()["patch_names"]
    if kind == "adjoint":
        # the inlet speed makes the state; the run to convergence is behind the program
        f = rng.uniform(0.6, 0.9)
        s.set_bc(dict(bc, u=f * bc["u"], v=f * bc["v"], w=f * bc["w"]))
        u, v, w, p = _channel_state(rng, bc, m, cc)
        s.set_state(f * u, f * v, f * w, f * f * p)
        s.iterate(400, 1e-12, 1e-11)
        return dict(kind=kind, s=s, patch=names.index("patch_3_0"))
    s.set_bc(bc)
    u, v, w, p = _channel_state(rng, bc, m, cc)
    s.set_state(u, v, w, p)
    if kind == "force":
        return dict(kind=kind, s=s, patch=names.index(case["patch"]))
    s.iterate(1)  # the multigrid hierarchy, built once in a run's first step
    out = dict(u=np.zeros(m.n_cells), v=np.zeros(m.n_cells), w=np.zeros(m.n_cells), p=np.zeros(m.n_cells))
    return dict(kind=kind, s=s, fields=(u, v, w, p), steps=case["steps"], out=out)


def run(state):
    s, kind = state["s"], state["kind"]
    if kind == "simple":
        s.set_state(*state["fields"])
        s.iterate(state["steps"])
        g = s.get_state(with_phi=False, out=state["out"])
        return {k: g[k] for k in ("u", "v", "w", "p")}
    if kind == "force":
        f = s.patch_force(state["patch"])
        return dict(n_faces=f["n_faces"], area=f["area"], Fp=np.array(f["Fp"]), Fv=np.array(f["Fv"]),
                    F=np.array(f["F"]))
    if kind == "adjoint":
        g, gmu, J, _ = s.adjoint_force_grad(state["patch"])
        return dict(dJ_dbc=g, dJ_dmu=gmu, J=J)
    if kind == "elliptic":
        return s.scalar_elliptic_solve(**state["args"])[0]
    return s.scalar_transport_solve(**state["args"])[0]


def work(case):
    """Lower bounds: every array of the grid and of the fields once per stage that needs it; the
    iterations of the linear solvers, whose number nothing fixes, are not counted."""
    m = _grid(case)[0]
    C, Fi, Fb = m.n_cells, m.n_internal, m.n_faces - m.n_internal
    kind = case["kind"]
    if kind == "force":
        t = m.topology()
        n = int(t["patch_size"][t["patch_names"].index(case["patch"])])
        return {"bytes": n * (4 + 56 + 32) + 120, "flops": 60 * n}
    system = 72 * Fi + 80 * Fb + 2 * 8 * Fi + 8 * C  # face geometry with its cells, a matrix
    if kind in ("elliptic", "transport"):
        per = 1 + case["n_nonorth"]
        return {"bytes": 24 * C + 16 * (Fi + Fb) + per * (system + 48 * C), "flops": per * (60 * Fi + 60 * C)}
    if kind == "adjoint":
        return {"bytes": 2 * system + 64 * C + 24 * (Fi + Fb), "flops": 600 * Fi}
    solves = 2 + case["n_nonorth"] + case["n_vel_nonorth"] + case["n_pressure_corr"]
    return {"bytes": 64 * C + case["steps"] * (solves * system + 300 * C),
            "flops": case["steps"] * solves * (150 * Fi + 100 * C)}


def exact(case, seed):
    """The force integral in plain numpy; nothing else here has a value without an iterative solve."""
    if case["kind"] != "force":
        return None
    rng = np.random.default_rng(seed)
    m, bc, cc = _grid(case)
    u, v, w, p = _channel_state(rng, bc, m, cc)
    t, g = m.topology(), m.geometry()
    k = t["patch_names"].index(case["patch"])
    f = np.arange(int(t["patch_start"][k]), int(t["patch_start"][k] + t["patch_size"][k]))
    c = t["owner"][f]
    area, n = g["af"][f], -g["nf"].reshape(-1, 3)[f]
    n = n / np.linalg.norm(n, axis=1)[:, None]
    d = cc[c] - g["xf"].reshape(-1, 3)[f]
    dn = np.abs((d * n).sum(1))
    vel = np.stack([u[c], v[c], w[c]], 1)
    ut = vel - (vel * n).sum(1)[:, None] * n
    Fp = (-p[c] * area)[:, None] * n
    Fv = (1e-3 * area / dn)[:, None] * ut
    return dict(n_faces=None, area=float(area.sum()), Fp=Fp.sum(0), Fv=Fv.sum(0), F=(Fp + Fv).sum(0))
