"""What is timed: the calls that a program using this package makes, over the sizes it makes them at.

Workloads come from ``pyvl_b200.workloads`` (the flat, swept pitching and flapping wings, the
jittered icosphere, the batch of uneven wings); every number that differs between two seeds --
incidence, sweep, motion, wake, jitter, points, training samples -- is drawn from the seed.

Kinds of case:

* ``run``     -- a whole ``run_solver`` call on a small wing: engine construction, a few free-wake
                 steps, results on the host.  What a user of the drop-in API starts with.
* ``matrix``  -- ``Mesh.induction_matrix3``: the normal influence matrix of a wing's rings.
* ``vectors`` -- ``Mesh.induction_matrix``: the vector influence of every ring at given points.
* ``field``   -- ``Mesh.induced_velocity``: the velocity a solved wing induces at the points of a
                 cross-plane survey behind it (flow fields, pressures, probes), FP64 or FP32.
* ``step``    -- one plain FP64 ``SolverEngine`` step of a moving wing with a full free wake:
                 assembly, wake corrections, LU, solve, advection, shedding.
* ``closed``  -- one ``SolverEngine`` step of a closed body (the zero-mean bordered system).
* ``mixed``   -- one ``MixedSolverEngine`` step of a flapping wing, seeded by the extrapolated warm
                 start: the path a long deforming-mesh run uses.
* ``batch``   -- one captured ``BatchEngine`` step of many uneven wings (parameter sweeps).
* ``train``   -- the warm-start network: one mini-batch gradient (forward and backward), and the
                 inference that a step runs.

``exact`` restates each of them in plain FP64 torch (the segment formula, the ring sums, the
no-penetration system with its wake terms, the dense solve, the Euler advection).
"""

from __future__ import annotations

import math

import numpy as np
import torch

import pyvl_b200 as pv
from pyvl_b200 import workloads
from pyvl_b200.batch import BatchEngine
from pyvl_b200.engine import MixedSolverEngine, SolverEngine, wake_spec_from_te
from pyvl_b200.learned import WarmStart, WarmStartMLP, drive_step, init_params

_F32 = 1  # precision code of induced_velocity
_PHASES = 32          # body positions kept per moving wing; the motion runs to and fro over them
_MIXED_PHASES = 96


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # a first run: the 16 x 4 flat wing, ten steps (the reference's smallest published example size)
        {"name": "run_small", "kind": "run", "ns": 16, "nc": 4, "steps": 10},
        # the matrix calls of a program that owns its solver loop: smallest, and the largest wing here
        {"name": "matrix_small", "kind": "matrix", "ns": 16, "nc": 4, "points": 64},
        {"name": "matrix_large", "kind": "matrix", "ns": 128, "nc": 32, "points": 4096},
        # ring vectors at an odd number of probe points, odd ring counts
        {"name": "vectors_odd", "kind": "vectors", "ns": 37, "nc": 13, "points": 1003},
        # a flow-field survey behind the largest wing
        {"name": "field_survey", "kind": "field", "ns": 128, "nc": 32, "points": 20011, "f32": False},
        # plain FP64 stepping: an odd wing, the pitching wing, the flapping wing with its full wake
        {"name": "step_odd", "kind": "step", "ns": 41, "nc": 11, "rows": 77, "motion": "flapping"},
        {"name": "step_pitching", "kind": "step", "ns": 64, "nc": 16, "rows": 200, "motion": "pitching"},
        {"name": "step_flapping", "kind": "step", "ns": 128, "nc": 32, "rows": 400, "motion": "flapping"},
        # the closed body: 5120 triangles and the zero-mean constraint
        {"name": "closed_sphere", "kind": "closed", "subdiv": 4, "jitter": 1e-3},
        # the fast path on the largest workload
        {"name": "mixed_flapping", "kind": "mixed", "ns": 128, "nc": 32, "rows": 400},
        # a sweep of uneven wings
        {"name": "batch_wings", "kind": "batch", "wings": 64, "p_min": 128, "p_max": 2048, "rows": 50, "sizes": 3},
        # one training iteration's gradient and one inference
        {"name": "train_batch", "kind": "train", "samples": 16384, "panels": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """An ns x nc grid of about lo .. hi rings, two to six times as many strips as rows."""
    p = _log(rng, lo, hi)
    ns = max(4, min(128, round(math.sqrt(p * rng.uniform(2.0, 6.0)))))
    return ns, max(2, min(32, p // ns))


def draw(rng):
    kind = rng.choice(["run", "matrix", "matrix", "vectors", "field", "step", "step", "closed", "mixed", "batch", "train"])
    if kind == "run":
        return {"kind": kind, "ns": rng.randint(8, 32), "nc": rng.randint(2, 8), "steps": rng.randint(5, 12)}
    if kind == "matrix":
        ns, nc = _grid(rng, 48, 4096)
        return {"kind": kind, "ns": ns, "nc": nc, "points": _log(rng, 16, 4096)}
    if kind == "vectors":
        ns, nc = _grid(rng, 32, 1024)
        return {"kind": kind, "ns": ns, "nc": nc, "points": _log(rng, 16, 4096)}
    if kind == "field":
        ns, nc = _grid(rng, 64, 4096)
        return {"kind": kind, "ns": ns, "nc": nc, "points": _log(rng, 100, 50000), "f32": rng.random() < 0.3}
    if kind == "step":
        ns, nc = _grid(rng, 64, 4096)
        return {"kind": kind, "ns": ns, "nc": nc, "rows": _log(rng, 4, 400),
                "motion": rng.choice(["flapping", "pitching"])}
    if kind == "closed":
        return {"kind": kind, "subdiv": rng.choice([2, 3, 3, 4]), "jitter": round(rng.uniform(2e-4, 2e-3), 6)}
    if kind == "mixed":
        ns, nc = _grid(rng, 256, 4096)  # an even strip count: the wing has a kink at its root
        return {"kind": kind, "ns": ns - ns % 2, "nc": nc, "rows": _log(rng, 40, 400)}
    if kind == "batch":
        return {"kind": kind, "wings": rng.randint(4, 64), "p_min": rng.randint(64, 256),
                "p_max": rng.randint(512, 2048), "rows": rng.randint(5, 50), "sizes": rng.randint(0, 10 ** 6)}
    return {"kind": kind, "samples": _log(rng, 128, 16384), "panels": _log(rng, 64, 4096)}


# --------------------------------------------------------------------------- inputs
def _dev():
    return torch.device("cuda")


def _moving_wing(case, seed):
    """A moving wing (workloads.Case), its first time and the seeded full wake behind it there."""
    rng = np.random.default_rng([seed, 1])
    ns, nc, rows = case["ns"], case["nc"], case["rows"]
    if case.get("motion", "flapping") == "pitching":
        c = workloads.swept_pitching(ns, nc, seed=int(rng.integers(1 << 30)), sweep_deg=float(rng.uniform(15, 30)),
                                     taper=float(rng.uniform(0.4, 0.7)), line_rows=rows)
    else:
        c = workloads.flapping(ns, nc, k=float(rng.uniform(0.15, 0.25)), alpha_deg=float(rng.uniform(3, 7)),
                               line_rows=rows)
    t0 = float(rng.uniform(0.0, 10.0))
    te = c.positions_at(t0)[np.asarray(c.te_node_pairs, np.int64)[:, ::-1]]  # shed line: strip s from node s+1 to s
    wpos, wcirc = workloads.synthetic_full_wake(te, rows, c.freestream, c.dt, int(rng.integers(1 << 30)))
    return c, t0, wpos, wcirc


def _phases(c, t0, n):
    """Positions and velocities at n consecutive times, then back again (velocities reversed)."""
    fwd = [(c.positions_at(t0 + i * c.dt), c.velocities_at(t0 + i * c.dt)) for i in range(n)]
    return fwd + [(p, -v) for p, v in fwd[-2:0:-1]]


def _static_wing(case, seed):
    rng = np.random.default_rng([seed, 2])
    c = workloads.swept_pitching(case["ns"], case["nc"], seed=int(rng.integers(1 << 30)),
                                 sweep_deg=float(rng.uniform(0, 35)), taper=float(rng.uniform(0.3, 1.0)))
    return c, c.positions_at(float(rng.uniform(0.0, 10.0)))


def _cp_choice(case, seed):
    """Which control points a matrix call asks for: all of them, or a seeded ascending choice."""
    rng = np.random.default_rng([seed, 3])
    p, n = case["ns"] * case["nc"], case["points"]
    return np.arange(p) if n == p else np.sort(rng.choice(p, n, replace=n > p))


def _probe_points(case, seed, span=8.0):
    """A survey of y-z planes behind the wing, plane by plane, line by line along y."""
    rng = np.random.default_rng([seed, 4])
    n = case["points"]
    planes = max(1, min(8, n // 64))
    per = -(-n // planes)
    nz = max(1, int(math.sqrt(per / 3)))
    ny = -(-per // nz)
    x, y, z = np.linspace(1.5, 6.0, planes), np.linspace(-0.75 * span, 0.75 * span, ny), np.linspace(-1.5, 1.5, nz)
    g = np.stack(np.meshgrid(x, z, y, indexing="ij"), -1)[..., [0, 2, 1]].reshape(-1, 3)[:n]
    return g + rng.uniform(-0.2, 0.2, 3)


def _circulation(case, seed):
    rng = np.random.default_rng([seed, 5])
    i = np.arange(case["ns"] * case["nc"], dtype=np.float64)
    return 0.1 + 0.05 * np.sin(0.01 * i + rng.uniform(0, 6)) + 0.005 * rng.standard_normal(i.size)


def _sphere(case, seed):
    return workloads.icosphere(case["subdiv"], seed=int(np.random.default_rng([seed, 6]).integers(1 << 30)),
                               jitter=case["jitter"])


def _flat_run(case, seed):
    rng = np.random.default_rng([seed, 7])
    c = workloads.flat_wing(case["ns"], case["nc"], alpha_deg=float(rng.uniform(2, 8)), nt=case["steps"],
                            line_rows=case["steps"])
    c.positions[:, 2] += 0.02 * rng.uniform(0.5, 1.5) * c.positions[:, 1] ** 2 / 16.0  # a little dihedral
    return c


def _batch_cases(case, seed):
    """Uneven wings whose sizes go with the case (``sizes``); incidence and dihedral go with the seed."""
    rng = np.random.default_rng([seed, 8])
    cases = workloads.batch_wings(case["wings"], case["sizes"], case["rows"], case["p_min"], case["p_max"])
    for c in cases:
        a = np.radians(rng.uniform(-8.0, 12.0))
        c.freestream = np.array([np.cos(a), 0.0, np.sin(a)])
        c.positions[:, 2] += rng.uniform(0.0, 0.1) * np.abs(c.positions[:, 1])
    return cases


def _batch_wakes(cases, seed):
    """A developed wake behind every wing of a batch."""
    return [workloads.synthetic_full_wake(c.positions_at(0.0)[np.asarray(c.te_node_pairs, np.int64)[:, ::-1]],
                                          c.line_rows, c.freestream, c.dt, seed + i) for i, c in enumerate(cases)]


def _train_data(case, seed):
    rng = np.random.default_rng([seed, 9])
    x = rng.standard_normal((case["samples"], 12)).astype(np.float32)
    w = rng.standard_normal(12).astype(np.float32) / 4
    t = (np.tanh(x @ w) + 0.1 * rng.standard_normal(case["samples"])).astype(np.float32)
    q = rng.standard_normal((case["panels"], 12)).astype(np.float32)
    return x, t, q, 0.1 * rng.standard_normal(case["panels"])


def _stepper(engine_cls, case, seed, phases, **kw):
    c, t0, wpos, wcirc = _moving_wing(case, seed)
    mesh = pv.Mesh(c.n_points, c.elements)
    eng = engine_cls(mesh, c.freestream, c.tol, wake_spec_from_te(mesh, c.te_node_pairs, c.line_rows, t0 - c.dt),
                     **{k: getattr(c, v) or None for k, v in kw.items()})
    eng.set_wake_state(wpos, wcirc, c.line_rows + 1, t0 - c.dt)
    eng.iteration = 1
    return {"engine": eng, "phases": _phases(c, t0, phases), "k": 0, "t0": t0, "dt": c.dt}


def prepare(case, seed):
    kind = case["kind"]
    f64 = dict(dtype=torch.float64, device=_dev())
    if kind == "run":
        c = _flat_run(case, seed)
        sim = pv.SimulationGeometry(pv.Geometry("wing", pv.ReferenceFrame(), pv.Mesh(c.n_points, c.elements),
                                                c.positions))
        spec = wake_spec_from_te(sim.mesh, c.te_node_pairs, c.line_rows, -c.dt)
        settings = pv.SolverSettings(pv.FlowConditionsUniform(*c.freestream), pv.ModelSettings(c.tol),
                                     pv.TimeSettings(c.nt, c.dt))
        return {"kind": kind, "sim": sim, "settings": settings, "spec": spec, "dt": c.dt, "rows": c.line_rows}
    if kind in ("matrix", "vectors", "field"):
        c, pos = _static_wing(case, seed)
        mesh = pv.Mesh(c.n_points, c.elements)
        p = torch.as_tensor(pos, **f64)
        s = {"kind": kind, "mesh": mesh, "tol": c.tol, "pos": p}
        if kind == "matrix":
            pick = torch.as_tensor(_cp_choice(case, seed), device=_dev())
            s["cps"], s["nrm"] = mesh.surface_average_vec3(p)[pick], mesh.surface_normal(p)[pick]
        else:
            s["pts"] = torch.as_tensor(_probe_points(case, seed), **f64)
        if kind == "field":
            s["gamma"], s["precision"] = torch.as_tensor(_circulation(case, seed), **f64), _F32 if case["f32"] else 0
        return s
    if kind == "step":
        return {"kind": kind, **_stepper(SolverEngine, case, seed, _PHASES)}
    if kind == "mixed":
        s = _stepper(MixedSolverEngine, case, seed, _MIXED_PHASES, cp_patches="smooth_patches",
                     wake_col_runs="wake_col_runs")
        return {"kind": kind, **s, "warm": WarmStart(s["engine"], None, jacobi=True)}
    if kind == "closed":
        c = _sphere(case, seed)
        eng = SolverEngine(pv.Mesh(c.n_points, c.elements), c.freestream, c.tol, None, [(0, c.n_surfaces)])
        return {"kind": kind, "engine": eng, "pos": c.positions, "vel": np.zeros_like(c.positions), "k": 0}
    if kind == "batch":
        cases = _batch_cases(case, seed)
        b = BatchEngine(cases)
        b.start(0.0)
        b.step()
        wakes = _batch_wakes(cases, seed)
        b.wpos.copy_(torch.as_tensor(np.concatenate([w.reshape(-1, 3) for w, _ in wakes])))
        b.wcirc.copy_(torch.as_tensor(np.concatenate([g.reshape(-1) for _, g in wakes])))
        b.rows.fill_(b.R)
        b.capture()
        return {"kind": kind, "batch": b}
    x, t, q, base = _train_data(case, seed)
    mlp = WarmStartMLP(_dev(), seed)
    mlp.out_scale = 0.5
    base = torch.as_tensor(base, **f64)
    return {"kind": kind, "mlp": mlp, "x": torch.as_tensor(x, device=_dev()), "t": torch.as_tensor(t, device=_dev()),
            "q": torch.as_tensor(q, device=_dev()), "base": base, "out": torch.empty_like(base)}


def run(s):
    kind = s["kind"]
    if kind == "run":
        spec = s["spec"]
        wake = pv.WakeModelLineExplicitUnsteady(spec.bordering_nodes, spec.shedding_lines, spec.adjacent_surfaces,
                                                s["settings"].model_settings.vortex_limit, -s["dt"], s["rows"])
        r = pv.run_solver(s["sim"], s["settings"], wake, None, verbose=False)
        return {"circulations": r.circulations, "wake": wake.wake_positions, "shed": wake.circulation}
    if kind == "matrix":
        return s["mesh"].induction_matrix3(s["tol"], s["pos"], s["cps"], s["nrm"])
    if kind == "vectors":
        return s["mesh"].induction_matrix(s["tol"], s["pos"], s["pts"])
    if kind == "field":
        return s["mesh"].induced_velocity(s["tol"], s["pos"], s["pts"], s["gamma"], s["precision"])
    if kind in ("step", "mixed"):
        eng, k = s["engine"], s["k"]
        s["k"] = k + 1
        pos, vel = s["phases"][k % len(s["phases"])]
        if kind == "step":
            eng.step(s["t0"] + k * s["dt"], pos, vel)
        else:
            drive_step(eng, s["warm"], s["t0"] + k * s["dt"], pos, vel)
        return {"gamma": eng.gamma, "wake": eng.wake_positions, "shed": eng.wake_circulation}
    if kind == "closed":
        s["k"] += 1
        return {"gamma": s["engine"].step(float(s["k"]), s["pos"], s["vel"])}
    if kind == "batch":
        b = s["batch"]
        b.step()
        return {"gamma": b.gamma, "wake": b.wpos, "shed": b.wcirc}
    mlp = s["mlp"]
    mlp.gradient(s["x"], s["t"])
    mlp.predict(s["q"], s["base"], s["out"])
    return {"grad": mlp.grad, "loss": mlp.loss, "prediction": s["out"]}


# --------------------------------------------------------------------------- work
_PAIR = 45  # operations of one segment-point pair (the reference's formula without its square root, division and atan2)


def _grid_lines(ns, nc):
    return ns * (nc + 1) + nc * (ns + 1)


def _step_work(ns, nc, rows, solve):
    """Distinct pairs of a step: every body line at every control point; every distinct wake line
    there too; every body line at every distinct wake node.  The matrix is written once and read
    once by the solve."""
    p = ns * nc
    pairs = _grid_lines(ns, nc) * p + (ns * (rows + 1) + (ns + 1) * rows) * p + _grid_lines(ns, nc) * (ns + 1) * rows
    return {"bytes": 16 * p * p + 2 * 24 * (ns + 1) * (rows + 1), "flops": _PAIR * pairs + solve}


def work(case):
    kind = case["kind"]
    if kind == "train":
        layers = 2 * (12 * 128 + 128 * 128 + 128)
        n, q, params = case["samples"], case["panels"], 18305
        return {"bytes": 4 * 13 * n + (4 * 12 + 16) * q + 12 * params, "flops": 3 * layers * n + layers * q}
    if kind == "closed":
        n = 20 * 4 ** case["subdiv"]
        return {"bytes": 16 * n * n, "flops": _PAIR * n * 3 * n // 2 + 2 * n ** 3 // 3}
    if kind == "batch":  # rings spread log-uniformly over [p_min, p_max], four strips to a row
        lo, hi = case["p_min"], case["p_max"]
        u = [(i + 0.5) / 16 for i in range(16)]
        sizes = [math.exp(math.log(lo) + x * math.log(hi / lo)) for x in u]
        parts = [_step_work(round(2 * math.sqrt(p)), max(1, round(math.sqrt(p) / 2)), case["rows"], 4 * p * p)
                 for p in sizes]
        return {k: int(sum(w[k] for w in parts) * case["wings"] / 16) for k in ("bytes", "flops")}
    ns, nc = case["ns"], case["nc"]
    p, lines = ns * nc, _grid_lines(ns, nc)
    if kind == "run":
        w = [_step_work(ns, nc, r, 2 * p ** 3 // 3) for r in range(case["steps"])]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if kind == "matrix":
        return {"bytes": 8 * p * case["points"] + 48 * case["points"], "flops": _PAIR * lines * case["points"]}
    if kind == "vectors":
        return {"bytes": 24 * p * case["points"] + 24 * case["points"], "flops": _PAIR * lines * case["points"]}
    if kind == "field":
        return {"bytes": 48 * case["points"] + 8 * p, "flops": _PAIR * lines * case["points"]}
    return _step_work(ns, nc, case["rows"], 2 * p ** 3 // 3 if kind == "step" else 4 * p * p)


# --------------------------------------------------------------------------- exact values
def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64)).to(_dev() if torch.cuda.is_available() else "cpu")


def _pairs(pts, r1, r2, tol):
    """(n, L, 3) velocity of unit segments r1 -> r2 at pts (times 4 pi, the reference's scaling)."""
    e = r2 - r1
    ln = e.norm(dim=1)
    d = e / ln.clamp_min(1e-300)[:, None]
    a = pts[:, None, :] - r1[None]
    t1 = (a * d[None]).sum(-1)
    c = torch.linalg.cross(a, d[None].expand_as(a), dim=-1)
    h2 = (c * c).sum(-1)
    ang = torch.atan2(-h2.sqrt() * ln, h2 + t1 * (t1 - ln))
    off = (h2 < tol * tol) | (ln < tol)[None]
    return torch.where(off, torch.zeros_like(ang), ang / h2.clamp_min(1e-300).sqrt())[..., None] * c


def _rows(n_pts, n_seg):
    return max(1, min(n_pts, (1 << 23) // max(1, n_seg)))


def _velocity(pts, r1, r2, gamma, tol):
    out = torch.zeros_like(pts)
    step = 1 << 15
    for l in range(0, r1.shape[0], step):
        n = _rows(pts.shape[0], min(step, r1.shape[0] - l))
        for i in range(0, pts.shape[0], n):
            k = _pairs(pts[i:i + n], r1[l:l + step], r2[l:l + step], tol)
            out[i:i + n] += torch.einsum("nlc,l->nc", k, gamma[l:l + step])
    return out


def _loops(elements):
    return torch.as_tensor(np.asarray(elements, np.int64)).to(_t(0.0).device)


def _ring_vectors(pts, pos, loops, tol):
    k = loops.shape[1]
    out = torch.empty((pts.shape[0], loops.shape[0], 3), dtype=torch.float64, device=pos.device)
    n = _rows(pts.shape[0], loops.shape[0])
    for i in range(0, pts.shape[0], n):
        out[i:i + n] = sum(_pairs(pts[i:i + n], pos[loops[:, q]], pos[loops[:, (q + 1) % k]], tol) for q in range(k))
    return out


def _ring_normals(pts, nrm, pos, loops, tol):
    out = torch.empty((pts.shape[0], loops.shape[0]), dtype=torch.float64, device=pos.device)
    n = _rows(pts.shape[0], loops.shape[0])
    for i in range(0, pts.shape[0], n):
        out[i:i + n] = (_ring_vectors(pts[i:i + n], pos, loops, tol) * nrm[i:i + n, None, :]).sum(-1)
    return out


def _centres_normals(pos, loops):
    p = pos[loops]
    d = p - p.roll(-1, 1)
    n = torch.linalg.cross(d.roll(-1, 1), d, dim=-1).sum(1)
    return p.mean(1), n / n.norm(dim=1, keepdim=True)


def _wake_edges(wpos, wcirc, first):
    """Edges and circulations of the wake rings of rows >= first; wpos (S, 2, R+1, 3), wcirc (S, R)."""
    a, b = wpos[:, 0], wpos[:, 1]
    loop = [a[:, first:-1], b[:, first:-1], b[:, first + 1:], a[:, first + 1:]]
    r1 = torch.stack(loop).reshape(-1, 3)
    r2 = torch.stack(loop[1:] + loop[:1]).reshape(-1, 3)
    return r1, r2, wcirc[:, first:].reshape(-1).repeat(4)


def _one_step(pos, vel, loops, te_rings, te_nodes, u, wpos, wcirc, rows, dt, tol, with_wake):
    """One iteration of the solver loop with the free wake; rows: complete wake rows (>= 1)."""
    cps, nrm = _centres_normals(pos, loops)
    rhs = -(nrm * (u - vel[loops].mean(1))).sum(-1)
    A = _ring_normals(cps, nrm, pos, loops, tol)
    if with_wake:
        S = wpos.shape[0]
        row0 = torch.stack([wpos[:, 0, 0], wpos[:, 1, 0], wpos[:, 1, 1], wpos[:, 0, 1]], 1).reshape(-1, 3)
        A[:, te_rings] -= _ring_normals(cps, nrm, row0, torch.arange(4 * S, device=pos.device).reshape(S, 4), tol)
        if wcirc.shape[1] > 1:
            rhs = rhs + (_velocity(cps, *_wake_edges(wpos, wcirc, 1), tol) * nrm).sum(-1)
    gamma = torch.linalg.solve(A, rhs)
    k = loops.shape[1]
    r1, r2 = (torch.cat([pos[loops[:, (q + o) % k]] for q in range(k)]) for o in (0, 1))
    old = wpos[:, :, :rows]
    v = u + _velocity(old.reshape(-1, 3), r1, r2, gamma.repeat(k), tol).reshape(old.shape)
    new = torch.empty_like(wpos)
    new[:, :, 0] = pos[te_nodes]
    new[:, :, 1:rows + 1] = old + v * dt
    new[:, :, rows + 1:] = new[:, :, rows:rows + 1]
    circ = torch.cat([gamma[te_rings][:, None], wcirc[:, :-1]], 1)
    return gamma, new, circ


def _te(ns, nc, device):
    """Rings at the trailing edge and the nodes of its shed lines (from node s + 1 to node s)."""
    s = torch.arange(ns, device=device)
    return s * nc + nc - 1, torch.stack([(s + 1) * (nc + 1) + nc, s * (nc + 1) + nc], 1)


def _bf16(x):
    return x.to(torch.bfloat16).double()


def _network(case, seed):
    """Gradient, loss and prediction of the BF16 network (rounded weights, inputs and activations)
    with every sum in FP64."""
    x, t, q, base = (_t(a) for a in _train_data(case, seed))
    p = _bf16(_t(init_params(seed)))
    w1, b1, w2, b2, w3 = p[:1536].reshape(128, 12), p[1536:1664], p[1664:18048].reshape(128, 128), p[18048:18176], p[18176:18304]
    x, q = _bf16(x), _bf16(q)

    def forward(v):
        h1 = _bf16(torch.relu(v @ w1.T + b1))
        h2 = _bf16(torch.relu(h1 @ w2.T + b2))
        return h1, h2, h2 @ w3 + p[18304]

    h1, h2, y = forward(x)
    dy = 2.0 * (y - t) / t.numel()
    d2 = torch.outer(dy, w3) * (h2 > 0)
    d1 = (d2 @ w2) * (h1 > 0)
    grad = [d1.T @ x, d1.sum(0), d2.T @ h1, d2.sum(0), h2.T @ dy, dy.sum()]
    return {"grad": torch.cat([g.reshape(-1) for g in grad]), "loss": ((y - t) ** 2).mean().reshape(1),
            "prediction": base + 0.5 * forward(q)[2]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _network(case, seed)
    if kind == "run":
        c = _flat_run(case, seed)
        pos, loops, u = _t(c.positions), _loops(c.elements), _t(c.freestream)
        rings, nodes = _te(case["ns"], case["nc"], pos.device)
        wpos = pos[nodes][:, :, None, :].repeat(1, 1, c.line_rows + 1, 1)
        wcirc = torch.zeros((rings.numel(), c.line_rows), dtype=torch.float64, device=pos.device)
        found, t = [], -c.dt
        for i in range(c.nt):
            rows, dt, t = min(i + 1, c.line_rows), i * c.dt - t, i * c.dt
            g, wpos, wcirc = _one_step(pos, torch.zeros_like(pos), loops, rings, nodes, u, wpos, wcirc, rows, dt, c.tol,
                                       i > 0)
            found.append(g)
        return {"circulations": torch.stack(found), "wake": wpos, "shed": wcirc}
    if kind in ("matrix", "vectors", "field"):
        c, p = _static_wing(case, seed)
        pos, loops = _t(p), _loops(c.elements)
        if kind == "matrix":
            pick = torch.as_tensor(_cp_choice(case, seed)).to(pos.device)
            cps, nrm = _centres_normals(pos, loops)
            return _ring_normals(cps[pick], nrm[pick], pos, loops, c.tol)
        pts = _t(_probe_points(case, seed))
        if kind == "vectors":
            return _ring_vectors(pts, pos, loops, c.tol)
        r1, r2 = (torch.cat([pos[loops[:, (q + o) % 4]] for q in range(4)]) for o in (0, 1))
        return _velocity(pts, r1, r2, _t(_circulation(case, seed)).repeat(4), c.tol)
    if kind in ("step", "mixed"):
        c, t0, wpos, wcirc = _moving_wing(case, seed)
        pos, loops = _t(c.positions_at(t0)), _loops(c.elements)
        rings, nodes = _te(case["ns"], case["nc"], pos.device)
        g, w, s = _one_step(pos, _t(c.velocities_at(t0)), loops, rings, nodes, _t(c.freestream), _t(wpos), _t(wcirc),
                            c.line_rows, c.dt, c.tol, True)
        return {"gamma": g, "wake": w, "shed": s}
    if kind == "closed":
        c = _sphere(case, seed)
        pos, loops = _t(c.positions), _loops(c.elements)
        cps, nrm = _centres_normals(pos, loops)
        n = loops.shape[0]
        K = torch.zeros((n + 1, n + 1), dtype=torch.float64, device=pos.device)
        K[:n, :n] = _ring_normals(cps, nrm, pos, loops, c.tol)
        K[:n, n] = K[n, :n] = 1.0
        b = torch.cat([-(nrm * _t(c.freestream)).sum(-1), torch.zeros(1, dtype=torch.float64, device=pos.device)])
        g = torch.linalg.solve(K, b)[:n]
        return {"gamma": g - g.mean()}
    found = []
    cases = _batch_cases(case, seed)
    for c, (wpos, wcirc) in zip(cases, _batch_wakes(cases, seed)):
        pos, loops = _t(c.positions), _loops(c.elements)
        ns = len(c.te_node_pairs)
        rings, nodes = _te(ns, len(c.elements) // ns, pos.device)
        found.append(_one_step(pos, torch.zeros_like(pos), loops, rings, nodes, _t(c.freestream), _t(wpos), _t(wcirc),
                               c.line_rows, c.dt, c.tol, True))
    return {"gamma": torch.cat([g for g, _, _ in found]), "wake": torch.cat([w.reshape(-1, 3) for _, w, _ in found]),
            "shed": torch.cat([s.reshape(-1) for _, _, s in found])}
