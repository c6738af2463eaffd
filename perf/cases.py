"""Performance cases of the flow solver: what a user's program has it do.

A user has a mesh and a configuration, lays a solver out once (``UfvmSolver``,
``UfvmBatch``), gives it a flow field, advances it a number of time steps and takes the
field back (with the per-step records where the run is monitored); or evaluates one
residual (``ufvm_solver``) or a batch of face fluxes (``roe_flux``) on host arrays.

``prepare`` lays the solver out and makes the starting field: the free stream (or the
manufactured field) under smooth waves of a few percent whose amplitudes, wave vectors
and phases come from the seed.  ``run`` sets that field and the time, advances, and
returns the field: each pass does the same work.

``exact`` computes the same flow in plain torch, in 64 bits: the second-order
finite-volume scheme (least-squares gradients, min/max limiter, Roe or Rusanov flux,
viscous flux, boundary states, Runge-Kutta steps at the lagged CFL time step).
"""
import functools
import json
import math

import numpy as np
import torch

import ebbcfd_gb300 as E
from ebbcfd_gb300 import meshgen

GAMMA = 1.4
STAGES = {"Euler": 1, "RK2": 2, "RK2_TVD": 2, "RK4": 4}


# ---- the cases ---------------------------------------------------------------------

def listed():
    return [
        # the 32 x 32 manufactured-solution run of a convergence study: the smallest call,
        # one launch after the other
        {"name": "mms_quads_fp64", "kind": "mms", "size": 32, "precision": "fp64", "flux": "roeFlux",
         "integrator": "RK2_TVD", "steps": 40, "records": True},
        # non-conforming polygons (pentagons and a hexagon) in the double-float form
        {"name": "mms_polygons_df", "kind": "polygons", "size": 48, "precision": "df", "flux": "roeFlux",
         "integrator": "RK2", "steps": 40, "records": True},
        # a small viscous solve as the request server is given it, monitored every step
        {"name": "cylinder_split", "kind": "cylinder", "size": 6001, "precision": "split", "flux": "roeFlux",
         "integrator": "RK2_TVD", "steps": 100, "records": True},
        # the middle of the range in the reference's own precision, monitored
        {"name": "cylinder_fp64", "kind": "cylinder", "size": 20000, "precision": "fp64", "flux": "roeFlux",
         "integrator": "RK2_TVD", "steps": 10, "records": True},
        # one residual evaluation on a host state: an outer solver's call of the operator
        {"name": "residual_fp64", "kind": "residual", "size": 90000, "precision": "fp64", "flux": "roeFlux",
         "integrator": "RK4", "steps": 1, "records": False},
        # the supersonic wedge (triangles, inviscid)
        {"name": "wedge_fp64", "kind": "wedge", "size": 200000, "precision": "fp64", "flux": "rusanovFlux",
         "integrator": "RK2", "steps": 20, "records": False},
        {"name": "wedge_split", "kind": "wedge", "size": 500000, "precision": "split", "flux": "rusanovFlux",
         "integrator": "RK2", "steps": 200, "records": False},
        # the Navier-Stokes flat plate (quads under triangles, viscous, four stages) in each
        # precision form: beyond the L2 cache in all three
        {"name": "plate_fp64", "kind": "plate", "size": 400000, "precision": "fp64", "flux": "roeFlux",
         "integrator": "RK4", "steps": 12, "records": False},
        {"name": "plate_df", "kind": "plate", "size": 500000, "precision": "df", "flux": "roeFlux",
         "integrator": "RK4", "steps": 40, "records": False},
        {"name": "plate_split", "kind": "plate", "size": 1000000, "precision": "split", "flux": "roeFlux",
         "integrator": "RK4", "steps": 100, "records": False},
        # many uneven meshes advanced together: a parameter sweep of bump channels
        {"name": "batch_split", "kind": "batch", "size": 20000, "precision": "split", "flux": "roeFlux",
         "integrator": "RK2_TVD", "steps": 100, "records": False, "instances": 40},
        # the flux operator alone on host arrays
        {"name": "faces_roe", "kind": "faces", "size": 150001, "precision": "fp64", "flux": "roeFlux",
         "integrator": "Euler", "steps": 1, "records": False},
    ]


def draw(rng):
    kind = rng.choice(["mms", "polygons", "cylinder", "residual", "wedge", "plate", "batch", "faces"])
    lo, hi = {"mms": (16, 256), "polygons": (12, 96), "cylinder": (2000, 120000), "residual": (2000, 120000),
              "wedge": (3000, 250000), "plate": (8000, 400000), "batch": (2000, 20000), "faces": (37, 300000)}[kind]
    size = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind == "polygons":
        size += size % 2
    c = {"kind": kind, "size": size, "records": rng.random() < 0.5,
         "precision": rng.choice(["fp64", "split", "df"]), "flux": rng.choice(["roeFlux", "rusanovFlux"]),
         "integrator": rng.choice(["RK2", "RK2_TVD", "RK4", "Euler"])}
    if kind == "wedge":
        c["flux"], c["integrator"] = "rusanovFlux", rng.choice(["RK2", "RK4"])
    if kind == "batch":
        c.update(records=False, instances=rng.randint(2, 24), integrator=rng.choice(["RK2", "RK2_TVD"]))
    if kind in ("residual", "faces"):
        c.update(records=False, steps=1)
    else:
        c["steps"] = max(3, min(200, int(rng.uniform(1.0e6, 4.0e6) / _cells(c) / STAGES[c["integrator"]])))
    if kind == "faces":
        c["precision"] = "fp64"
    return c


def _cells(case):
    """About how many cells the case's meshes have together."""
    n = case["size"]
    if case["kind"] == "mms":
        return n * n
    if case["kind"] == "polygons":
        return n * n * 13 // 4
    return n * case.get("instances", 1)


# ---- meshes and configurations -----------------------------------------------------

def _instances(case):
    """(kind, size, seed, bump height, Mach) of each instance of a batch: cell counts spread
    over a factor of 30."""
    rng = np.random.default_rng(11)
    out = []
    for k in range(case["instances"]):
        n = int(case["size"] * math.exp(rng.uniform(math.log(0.1), math.log(3.0))))
        out.append(("bump", max(500, n), k, float(rng.uniform(0.02, 0.1)), float(rng.uniform(0.3, 0.8))))
    return out


@functools.lru_cache(maxsize=256)
def _mesh(kind, size, seed=0, h=0.05):
    if kind == "mms":
        return meshgen.uniform_quads(size)
    if kind == "polygons":
        return meshgen.hanging_quads(size)
    if kind == "cylinder":
        return meshgen.cylinder(size, seed=seed)
    if kind == "wedge":
        return meshgen.wedge(size, seed=seed)
    if kind == "bump":
        return meshgen.bump_channel(size, h=h, seed=seed)
    # the wall layer stays below a fifth of the cells on coarse plates
    return meshgen.flat_plate(size, layer_top=None if size > 100000 else 0.01)


@functools.lru_cache(maxsize=256)
def _host_mesh(*key):
    return _mesh(*key).to_solver_mesh()


def _config(case, mach=None, dt=None):
    kind, visc = case["kind"], False
    c = {"mesh": "mesh.msh", "dt": 1e-6, "tEnd": 1e9, "flux": case["flux"], "saveIter": -1, "plotIter": -1,
         "integrator": case["integrator"], "limited": True}
    bc = lambda tag, typ, q: {"tag": tag, "type": typ, "q": q}  # noqa: E731
    if kind in ("mms", "polygons"):
        q = [0.5, 0, 1, 1]
        c.update(CFL=0.3 if case["integrator"] == "Euler" else 0.5, forceBoundary="Freestream",
                 boudaryConditions=[bc("Freestream", "dirichlet", q)])
    elif kind == "cylinder":
        q = [0.2, 0, 1, 1]
        visc = True
        c.update(CFL=0.3, forceBoundary="Cylinder",
                 boudaryConditions=[bc(t, "fullState", q) for t in ("Inflow", "Outflow", "Top", "Bottom")] +
                 [bc("Cylinder", "viscidWall", q)],
                 physicalConfig={"Pr": 0.72, "R": 1.0, "gamma": 1.4, "Re": 100.0, "L": 1.0})
    elif kind == "wedge":
        q = [2.5, 0, 1, 1]
        c.update(CFL=0.4, forceBoundary="Ramp",
                 boudaryConditions=[bc(t, "fullState", q) for t in ("Inflow", "Top", "Outflow")] +
                 [bc("Symmetry", "symmetry", q), bc("Ramp", "inviscidWall", q)])
    elif kind == "batch":
        q = [mach, 0, 1, 1]
        c.update(dt=dt, dynamicDt=False, forceBoundary="Wall",
                 boudaryConditions=[bc("Inflow", "fullState", q), bc("Outflow", "fullState", q),
                                    bc("Wall", "inviscidWall", q)])
    else:  # plate, residual
        q = [0.3, 0, 1, 1]
        visc = True
        c.update(CFL=0.3 if case["integrator"] == "Euler" else 0.8, forceBoundary="Wall", cflAdjust=False,
                 boudaryConditions=[bc("Inflow", "fullState", q), bc("Top", "fullState", q),
                                    bc("Outflow", "constP", [1.0 / (GAMMA * 0.09)]), bc("Symmetry", "symmetry", q),
                                    bc("Wall", "viscidWall", q)],
                 physicalConfig={"Pr": 0.72, "R": 1.0, "gamma": 1.4, "Re": 1e5, "L": 1.0})
    c.update(initialConditions=q, viscosity=visc)
    return c


def _mesh_kind(case):
    return "plate" if case["kind"] == "residual" else case["kind"]


def _solves(case):
    """[(mesh key, configuration)] of the case's solves (one, or a batch's instances)."""
    if case["kind"] != "batch":
        return [((_mesh_kind(case), case["size"]), _config(case))]
    out = []
    for kind, n, seed, h, mach in _instances(case):
        spacing = math.sqrt(6.0 / n)
        out.append(((kind, n, seed, h), _config(case, mach, dt=0.08 * spacing / (1.0 + 1.0 / mach))))
    return out


def _field(case, cfg, xy, seed):
    """The starting field at the cell centroids: primitive values under smooth waves."""
    rng = np.random.default_rng(seed)
    w = np.zeros((4, len(xy)))
    for k in range(4):
        for _ in range(3):
            kx, ky, ph, a = rng.uniform(-9, 9), rng.uniform(-9, 9), rng.uniform(0, 2 * math.pi), rng.uniform(0.2, 1)
            w[k] += a * np.sin(kx * xy[:, 0] + ky * xy[:, 1] + ph)
    if case["kind"] in ("mms", "polygons"):
        r, u, v, p = _sine(torch.from_numpy(np.ascontiguousarray(xy)))
        r, u, v, p = (t.numpy() for t in (r, u, v, p))
        eps = 2e-3
    else:
        m = cfg["initialConditions"][0]
        r, u, v, p = np.ones(len(xy)), np.ones(len(xy)), np.full(len(xy), 0.05), np.full(len(xy), 1.0 / (GAMMA * m * m))
        eps = 1e-2
    r, p = r * (1 + eps * w[0]), p * (1 + 0.5 * eps * w[3])
    u, v = u + eps * w[1], v + eps * w[2]
    return np.stack([r, r * u, r * v, p / (GAMMA - 1) + 0.5 * r * (u * u + v * v)], axis=1)


def _faces(case, seed):
    """Left and right states of neighbouring cells and unit normals."""
    rng = np.random.default_rng(seed)
    n = case["size"]
    ang = rng.uniform(0, 2 * math.pi, n)
    states = []
    base = np.stack([rng.uniform(0.5, 2, n), rng.normal(0.5, 0.5, n), rng.normal(0, 0.5, n), rng.uniform(0.5, 3, n)])
    for _ in range(2):
        r, u, v, p = base * (1 + 0.05 * rng.standard_normal((4, n)))
        states.append(np.stack([r, r * u, r * v, p / (GAMMA - 1) + 0.5 * r * (u * u + v * v)], axis=1))
    return states[0], states[1], np.stack([np.cos(ang), np.sin(ang)], axis=1)


# ---- the framework's pass ----------------------------------------------------------

def prepare(case, seed):
    if case["kind"] == "faces":
        return {"case": case, "faces": _faces(case, seed)}
    solves = _solves(case)
    meshes = [_host_mesh(*key) for key, _ in solves]
    cfgs = []
    for _, c in solves:
        cfg = E.load_config(json.dumps(c))
        cfg.mms = 2 if case["kind"] in ("mms", "polygons") else 0
        cfgs.append(cfg)
    q = np.concatenate([_field(case, c, m.centroids(), seed * 1000 + k)
                        for k, (m, (_, c)) in enumerate(zip(meshes, solves))])
    if case["kind"] == "batch":
        sol = E.UfvmBatch(meshes, cfgs, case["precision"])
    else:
        sol = E.UfvmSolver(meshes[0], cfgs[0], case["precision"])
    return {"case": case, "solver": sol, "q": q, "dt": solves[0][1]["dt"]}


def run(state):
    case = state["case"]
    if case["kind"] == "faces":
        flux = E.roe_flux if case["flux"] == "roeFlux" else E.rusanov_flux
        F, s = flux(*state["faces"])
        return {"flux": F, "speed": s}
    sol = state["solver"]
    if case["kind"] == "residual":
        R, dt, rmax = sol.ufvm_solver(state["q"])
        return {"residual": R, "dt": dt, "rmax": rmax}
    sol.set_state(state["q"])
    if case["kind"] != "batch":
        sol.set_time(0.0, state["dt"])
    rec = sol.run(case["steps"], records=case["records"])
    out = {"state": sol.state}
    if case["records"]:
        out["records"] = rec
    return out


def work(case):
    """Each stage reads the field and the mesh (neighbour and face indices, gradient
    weights, neighbour and face offsets per cell side; normal and length per face) and
    writes the field once; the operations are those of one face's flux and one cell's
    gradient, limiter and sums."""
    r = 4 if case["precision"] == "split" else 8
    if case["kind"] == "faces":
        return {"bytes": case["size"] * 15 * 8, "flops": case["size"] * 230}
    cells = _cells(case)
    sides = cells * {"mms": 4.0, "polygons": 4.0, "plate": 3.35, "residual": 3.35}.get(case["kind"], 3.0)
    visc = case["kind"] in ("plate", "residual", "cylinder")
    stages = case["steps"] * STAGES[case["integrator"]] if case["kind"] != "residual" else 1
    face = (230 if case["flux"] == "roeFlux" else 130) + (150 if visc else 0)
    return {"bytes": stages * (cells * 8 * r + sides * (8 + 6 * r) + sides / 2 * 3 * r) + cells * 64,
            "flops": stages * (sides / 2 * face + sides * 60 + cells * 40)}


# ---- the same flow in plain torch, in 64 bits --------------------------------------

def exact(case, seed):
    if case["kind"] == "faces":
        qL, qR, n = (torch.from_numpy(a) for a in _faces(case, seed))
        f = _roe if case["flux"] == "roeFlux" else _rusanov
        F, s = f(qL, qR, n)
        return {"flux": F.numpy(), "speed": s.numpy()}
    states, out = [], {}
    for k, (key, cfg) in enumerate(_solves(case)):
        flow = _Flow(_mesh(*key), cfg, mms=case["kind"] in ("mms", "polygons"))
        q = flow.tensor(_field(case, cfg, flow.centroid[:flow.C].cpu().numpy(), seed * 1000 + k))
        if case["kind"] == "residual":
            R, dt, rmax = flow.residual(q)
            return {"residual": R.cpu().numpy(), "dt": float(dt), "rmax": float(rmax)}
        q, rec = flow.advance(q, case["steps"], case["records"])
        states.append(q.cpu().numpy())
        if case["records"]:
            out["records"] = rec
    return {"state": np.concatenate(states), **out}


def _sine(xy):
    """Density, velocity and pressure of the sine manufactured solution."""
    x, y = 2 * math.pi * xy[:, 0], 2 * math.pi * xy[:, 1]
    return (1 + 0.1 * torch.sin(x) * torch.cos(y), 0.5 + 0.05 * torch.cos(x) * torch.sin(y),
            0.3 + 0.05 * torch.sin(x + 1), 1 / GAMMA + 0.1 * torch.cos(y))


def _conserved(w):
    r, u, v, p = w
    return torch.stack([r, r * u, r * v, p / (GAMMA - 1) + 0.5 * r * (u * u + v * v)], 1)


def _sine_source(xy):
    """div F of the sine solution, by differentiating its fluxes."""
    xy = xy.clone().requires_grad_(True)
    w = _sine(xy)
    q = _conserved(w)
    S = []
    for k in range(4):
        s = torch.zeros_like(w[0])
        for d in range(2):
            f = (q[:, k] + (w[3] if k == 3 else 0)) * w[1 + d] + (w[3] if k == 1 + d else 0)
            s = s + torch.autograd.grad(f.sum(), xy, retain_graph=True)[0][:, d]
        S.append(s.detach())
    return torch.stack(S, 1)


def _pressure(q):
    return (GAMMA - 1) * (q[:, 3] - 0.5 * (q[:, 1] ** 2 + q[:, 2] ** 2) / q[:, 0])


def _convective(q, p, n):
    un = (q[:, 1] * n[:, 0] + q[:, 2] * n[:, 1]) / q[:, 0]
    return torch.stack([q[:, 0] * un, q[:, 1] * un + p * n[:, 0], q[:, 2] * un + p * n[:, 1], (q[:, 3] + p) * un], 1)


def _speeds(u, a):
    eps = 0.01 * a
    lam = torch.stack([(u + a).abs(), (u - a).abs(), u.abs()], 1)
    e = eps[:, None]
    return torch.where(lam < e, (e * e + lam * lam) / (2 * e), lam)


def _roe(qL, qR, n):
    pL, pR = _pressure(qL), _pressure(qR)
    w = torch.sqrt(qR[:, 0] / qL[:, 0])
    mean = lambda a, b: (w * b + a) / (1 + w)  # noqa: E731
    u0, u1 = mean(qL[:, 1] / qL[:, 0], qR[:, 1] / qR[:, 0]), mean(qL[:, 2] / qL[:, 0], qR[:, 2] / qR[:, 0])
    h = mean((qL[:, 3] + pL) / qL[:, 0], (qR[:, 3] + pR) / qR[:, 0])
    u, k = u0 * n[:, 0] + u1 * n[:, 1], 0.5 * (u0 * u0 + u1 * u1)
    a = torch.sqrt((GAMMA - 1) * (h - k))
    d = qR - qL
    lam = _speeds(u, a)
    l1, l2, l3 = lam.unbind(1)
    s1, s2 = 0.5 * (l1 + l2), 0.5 * (l1 - l2)
    G1 = (GAMMA - 1) * (k * d[:, 0] - (u0 * d[:, 1] + u1 * d[:, 2]) + d[:, 3])
    G2 = -u * d[:, 0] + (d[:, 1] * n[:, 0] + d[:, 2] * n[:, 1])
    C1 = G1 / (a * a) * (s1 - l3) + G2 / a * s2
    C2 = G1 / a * s2 + (s1 - l3) * G2
    D = l3[:, None] * d + C1[:, None] * torch.stack([torch.ones_like(u), u0, u1, h], 1) + \
        C2[:, None] * torch.stack([torch.zeros_like(u), n[:, 0], n[:, 1], u], 1)
    return 0.5 * (_convective(qL, pL, n) + _convective(qR, pR, n)) - 0.5 * D, lam.max(1).values


def _rusanov(qL, qR, n):
    pL, pR = _pressure(qL), _pressure(qR)
    sL, sR = torch.sqrt(qL[:, 0]), torch.sqrt(qR[:, 0])
    mean = lambda a, b: (sL * a + sR * b) / (sL + sR)  # noqa: E731
    u0, u1 = mean(qL[:, 1] / qL[:, 0], qR[:, 1] / qR[:, 0]), mean(qL[:, 2] / qL[:, 0], qR[:, 2] / qR[:, 0])
    a = torch.sqrt(GAMMA * mean(pL, pR) / (sL * sR))
    s = _speeds(u0 * n[:, 0] + u1 * n[:, 1], a).max(1).values
    return 0.5 * (_convective(qL, pL, n) + _convective(qR, pR, n)) - 0.5 * s[:, None] * (qR - qL), s


def _viscous(q, g, n, mu, pr):
    """Viscous flux from the face state and the gradients g[:, variable, direction]."""
    r = q[:, 0]
    u, v, e = q[:, 1] / r, q[:, 2] / r, q[:, 3] / r
    du, dv = (g[:, 1] - u[:, None] * g[:, 0]) / r[:, None], (g[:, 2] - v[:, None] * g[:, 0]) / r[:, None]
    de = (g[:, 3] - e[:, None] * g[:, 0]) / r[:, None]
    dT = de - u[:, None] * du - v[:, None] * dv  # internal energy
    div = du[:, 0] + dv[:, 1]
    txx, tyy, txy = mu * (2 * du[:, 0] - 2 / 3 * div), mu * (2 * dv[:, 1] - 2 / 3 * div), mu * (du[:, 1] + dv[:, 0])
    k = GAMMA / pr * mu
    fx = u * txx + v * txy + k * dT[:, 0]
    fy = u * txy + v * tyy + k * dT[:, 1]
    # the scheme's own viscous matrices take d(rho v)/dx for d(rho u)/dx in the y-momentum's
    # normal stress (not in its work)
    tyy = tyy + 2 / 3 * mu * (g[:, 1, 0] - g[:, 2, 0]) / r
    return torch.stack([torch.zeros_like(r), txx * n[:, 0] + txy * n[:, 1], txy * n[:, 0] + tyy * n[:, 1],
                        fx * n[:, 0] + fy * n[:, 1]], 1)


class _Flow:
    """One mesh and configuration: topology, geometry and the scheme, vectorised over cells
    and faces."""

    def __init__(self, mesh, cfg, mms):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.cfg, self.mms = cfg, mms
        blocks = [np.asarray(b, dtype=np.int64) - 1 for b in (mesh.elements if isinstance(mesh.elements, list)
                                                               else [mesh.elements])]
        K = max(b.shape[1] for b in blocks)
        C = self.C = sum(len(b) for b in blocks)
        node = np.zeros((C, K, 2), dtype=np.int64)  # the two nodes of each cell side
        mask = np.zeros((C, K), dtype=bool)
        at = 0
        for b in blocks:
            m = b.shape[1]
            node[at:at + len(b), :m, 0], node[at:at + len(b), :m, 1] = b, np.roll(b, -1, axis=1)
            mask[at:at + len(b), :m] = True
            at += len(b)
        xy = np.asarray(mesh.nodes, dtype=np.float64)[:, :2]
        cell, side = np.nonzero(mask)
        a, b = node[cell, side, 0], node[cell, side, 1]
        key = np.minimum(a, b) * len(xy) + np.maximum(a, b)
        uniq, first, face = np.unique(key, return_index=True, return_inverse=True)
        face = face.reshape(-1)
        F = len(uniq)
        own = cell[first]
        other = np.full(F, -1, dtype=np.int64)
        second = np.ones(len(cell), dtype=bool)
        second[first] = False
        other[face[second]] = cell[second]
        # boundary groups by node pair
        bn = np.asarray(mesh.b_nodes, dtype=np.int64)
        group = np.searchsorted(np.asarray(list(mesh.b_group_start) + [len(bn)]), np.arange(len(bn)), side="right") - 1
        bkey = np.minimum(bn[:, 0], bn[:, 1]) * len(xy) + np.maximum(bn[:, 0], bn[:, 1])
        bface = np.searchsorted(uniq, bkey)
        fgroup = np.full(F, -1, dtype=np.int64)
        fgroup[bface] = group
        bnd = np.nonzero(fgroup >= 0)[0]
        other[bnd] = C + np.arange(len(bnd))
        pa, pb = xy[a[first]], xy[b[first]]  # face ends, in the owner's orientation
        t = pb - pa
        length = np.hypot(t[:, 0], t[:, 1])
        # cell areas and centroids
        x0, x1 = xy[node[:, :, 0]], xy[node[:, :, 1]]
        o = x0[:, :1]  # about the first node
        p0, p1 = (x0 - o) * mask[:, :, None], (x1 - o) * mask[:, :, None]
        det = p0[:, :, 0] * p1[:, :, 1] - p1[:, :, 0] * p0[:, :, 1]
        area = 0.5 * det.sum(1)
        cen = o[:, 0] + ((p0 + p1) * det[:, :, None]).sum(1) / (6 * area[:, None])
        nb_ = np.stack([t[:, 1], -t[:, 0]], 1) / length[:, None]
        # ghost centroids: the owner's, reflected in the boundary face, by the face's slope
        # as the scheme has it (a face that is vertical but for rounding puts its ghost
        # somewhere else)
        ba, co = pa[bnd], cen[own[bnd]]
        flat = t[bnd, 0] != 0
        m = np.where(flat, -t[bnd, 1], 0) / np.where(flat, -t[bnd, 0], 1)
        c = ba[:, 1] - m * ba[:, 0]
        d = (co[:, 0] + (co[:, 1] - c) * m) / (1.0 + m * m)
        ghost = np.where(flat[:, None], np.stack([2.0 * d - co[:, 0], 2.0 * d * m - co[:, 1] + 2.0 * c], 1),
                         np.stack([2.0 * ba[:, 0] - co[:, 0], co[:, 1]], 1))
        T = self.tensor
        self.centroid = T(np.concatenate([cen, ghost]))
        self.area, self.n, self.len, self.mid = T(area), T(nb_), T(length), T(0.5 * (pa + pb))
        self.own, self.other, self.bnd = T(own), T(other), T(bnd)
        self.mask = T(mask)
        nbr, fce, sign = np.zeros((C, K), np.int64), np.zeros((C, K), np.int64), np.zeros((C, K))
        nbr[cell, side] = np.where(second, own[face], other[face])
        fce[cell, side] = face
        sign[cell, side] = np.where(second, -1.0, 1.0)
        self.nbr, self.face, self.sign = T(nbr), T(fce), T(sign)
        self.perim = (self.len[self.face] * self.mask).sum(1)
        self.cell_d = 2 * self.area / self.perim
        self.off = (self.centroid[self.nbr] - self.centroid[:C, None]) * self.mask[:, :, None]
        A = torch.einsum("ckr,cks->crs", self.off, self.off)
        self.weights = torch.einsum("crs,cks->ckr", torch.linalg.inv(A), self.off)
        g = fgroup[bnd]
        kinds = {b["tag"]: b for b in cfg["boudaryConditions"]}
        self.bcs = [(kinds[tag], T(np.nonzero(g == i)[0])) for i, tag in enumerate(mesh.tags)]
        self.force = T(bnd[g == list(mesh.tags).index(cfg["forceBoundary"])])
        self.flux = _roe if cfg["flux"] == "roeFlux" else _rusanov
        self.mu = 1.0 / cfg["physicalConfig"]["Re"] if cfg["viscosity"] else 0.0
        if mms:
            self.q_ghost, self.q_mid = (_conserved(_sine(x)) for x in (self.centroid[C:], self.mid[self.bnd]))
            self.source = _sine_source(self.centroid[:C])

    def tensor(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def _stream(self, q):
        m, aoa, _, r = q
        one = torch.ones(1, dtype=torch.float64, device=self.dev)
        return _conserved((r * one, math.cos(math.radians(aoa)) * one, math.sin(math.radians(aoa)) * one,
                           r / (GAMMA * m * m) * one))

    @staticmethod
    def _mirror(q, n):
        mom = q[:, 1:3] - 2 * (q[:, 1:3] * n).sum(1, keepdim=True) * n
        return torch.cat([q[:, :1], mom, q[:, 3:]], 1)

    def ghosts(self, q):
        """Ghost states and the right-hand states of the boundary faces that need only them."""
        out = torch.zeros(len(self.bnd), 4, dtype=torch.float64, device=self.dev)
        for bc, b in self.bcs:
            if not len(b):
                continue
            qi, n = q[self.own[self.bnd[b]]], self.n[self.bnd[b]]
            typ = bc["type"]
            if typ == "dirichlet":
                out[b] = self.q_ghost[b]
            elif typ in ("inviscidWall", "symmetry"):
                out[b] = self._mirror(qi, n)
            elif typ == "viscidWall":
                out[b] = qi * self.tensor(np.array([1.0, -1, -1, 1]))
            elif typ == "constP":
                r, u, v, p = qi[:, 0], qi[:, 1] / qi[:, 0], qi[:, 2] / qi[:, 0], _pressure(qi)
                pb = bc["q"][0]
                J = u + 2 * torch.sqrt(GAMMA * p / r) / (GAMMA - 1)
                rb = (pb * r ** GAMMA / p) ** (1 / GAMMA)
                ub = J - 2 * torch.sqrt(GAMMA * pb / rb) / (GAMMA - 1)
                jump = ((ub * n[:, 0] + v * n[:, 1]) - (u * n[:, 0] + v * n[:, 1]))[:, None] * n
                out[b] = torch.stack([rb, rb * (u + jump[:, 0]), rb * (v + jump[:, 1]),
                                      pb / (GAMMA - 1) + 0.5 * rb * (ub * ub + v * v)], 1)
            else:
                out[b] = qi
        return out

    def residual(self, q, limit=True):
        """(R, CFL time step, largest |sum of face fluxes|)."""
        C, bnd = self.C, self.bnd
        ghost = self.ghosts(q)
        qa = torch.cat([q, ghost])
        qn = torch.where(self.mask[:, :, None], qa[self.nbr], q[:, None])
        grad = torch.einsum("ckv,ckr->cvr", qn - q[:, None], self.weights)
        lim = torch.ones_like(q)
        if limit:
            lo, hi = torch.minimum(q, qn.amin(1)), torch.maximum(q, qn.amax(1))
            for k in range(self.off.shape[1]):
                d = torch.einsum("cvr,cr->cv", grad, self.off[:, k])
                e = q + d
                bound = torch.where(e < lo, lo, hi)
                s = torch.where((e < lo) | (e > hi), (bound - q) / d, torch.ones_like(d))
                lim = torch.where(self.mask[:, k:k + 1], torch.minimum(lim, s), lim)
        lg = lim[:, :, None] * grad
        rebuild = lambda c: q[c] + torch.einsum("fvr,fr->fv", lg[c], self.mid_of(c) - self.centroid[c])  # noqa: E731
        faces = torch.arange(len(self.len), device=self.dev)
        self.mid_of = lambda c: self.mid[faces]
        qL = rebuild(self.own)
        inner = torch.nonzero(self.other < C).reshape(-1)
        faces = inner
        qR = torch.empty_like(qL)
        qR[inner] = rebuild(self.other[inner])
        qR[bnd] = qL[bnd]
        cv = self.cfg["viscosity"]
        F, s = torch.empty_like(qL), torch.empty_like(self.len)
        F[inner], s[inner] = self.flux(qL[inner], qR[inner], self.n[inner])
        if cv:
            g = 0.5 * (grad[self.own[inner]] + grad[self.other[inner]])
            F[inner] -= _viscous(0.5 * (qL[inner] + qR[inner]), g, self.n[inner], self.mu, self.cfg["physicalConfig"]["Pr"])
        for bc, b in self.bcs:
            f = bnd[b]
            if not len(f):
                continue
            n, l, typ, g = self.n[f], qL[f], bc["type"], grad[self.own[f]]
            if typ in ("dirichlet", "fullState"):
                r = self.q_mid[b] if typ == "dirichlet" else self._stream(bc["q"]).expand(len(f), 4)
                F[f], s[f] = self.flux(l, r, n)
                if cv:
                    F[f] -= _viscous(0.5 * (l + r), 0.5 * g, n, self.mu, self.cfg["physicalConfig"]["Pr"])
            elif typ == "inviscidWall":
                vel = l[:, 1:3] / l[:, :1]
                t = vel - (vel * n).sum(1, keepdim=True) * n
                p = (GAMMA - 1) * (l[:, 3] - 0.5 * l[:, 0] * (t * t).sum(1))
                F[f], s[f] = _wall(p, n), torch.sqrt(GAMMA * p / l[:, 0])
            elif typ == "viscidWall":
                p = (GAMMA - 1) * l[:, 3]
                qw = l * self.tensor(np.array([1.0, 0, 0, 1]))
                g = g.clone()
                g[:, 3] = (l[:, 3] / l[:, 0])[:, None] * g[:, 0]
                F[f] = _wall(p, n) - _viscous(qw, g, n, self.mu, self.cfg["physicalConfig"]["Pr"])
                s[f] = torch.sqrt(GAMMA * p / l[:, 0])
            elif typ == "constP":
                x = ghost[b]
                p = _pressure(x)
                F[f], s[f] = _convective(x, p, n), torch.sqrt(GAMMA * p / x[:, 0])
            else:  # symmetry
                r = self._mirror(l, n)
                F[f], s[f] = self.flux(l, r, n)
                if cv:
                    nn = n[:, :, None] * n[:, None, :]
                    eye = torch.eye(2, dtype=torch.float64, device=self.dev)
                    t1 = g.clone()
                    t1[:, 1:3] = torch.einsum("frs,fsc->frc", eye - nn, g[:, 1:3])
                    gb = torch.einsum("frk,fkc->frc", g, nn) + torch.einsum("frk,fkc->frc", t1, eye - 2 * nn)
                    F[f] -= _viscous(0.5 * (l + r), gb, n, self.mu, self.cfg["physicalConfig"]["Pr"])
        F, s = F * self.len[:, None], s * self.len
        self.forces = F[self.force, 1:3].sum(0)
        total = (F[self.face] * self.sign[:, :, None]).sum(1)
        ave = (s[self.face] * self.mask).sum(1) / self.perim
        dt = (self.cfg.get("CFL", 0.5) * self.cell_d / ave).min()
        R = -total / self.area[:, None]
        if self.mms:
            R = R + self.source
        return R, dt, total.abs().max()

    def advance(self, q, steps, records):
        kind, t, dt = self.cfg["integrator"], 0.0, self.cfg["dt"]
        rec = []
        for _ in range(steps):
            q0, rmax = q, 0.0
            k1, new, m1 = self.residual(q)
            if kind == "Euler":
                q, top = q0 + dt * k1, [m1]
            elif kind == "RK2":
                k2, new, m2 = self.residual(q0 + dt * k1)
                q, top = q0 + 0.5 * dt * (k1 + k2), [m1, m2]
            elif kind == "RK2_TVD":
                fe = q0 + dt * k1
                k2, new, m2 = self.residual(fe, limit=False)
                q, top = 0.5 * (q0 + fe + dt * k2), [m1, m2]
            else:
                k2, _, m2 = self.residual(q0 + 0.5 * dt * k1)
                k3, _, m3 = self.residual(q0 + 0.5 * dt * k2)
                k4, new, m4 = self.residual(q0 + dt * k3)
                q, top = q0 + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4), [m1, m2, m3, m4]
            if self.cfg.get("dynamicDt", True):
                dt = float(new)
            if records:
                rmax = max(float(m) for m in top)
                res = torch.sqrt(self.C * ((q - q0) ** 2).sum(0)) / q.sum(0)
                fx, fy = (float(v) for v in self.forces)
                a = math.radians(self.cfg["initialConditions"][1])
                rec.append([t, math.cos(a) * fx - math.sin(a) * fy, math.sin(a) * fx + math.cos(a) * fy,
                            *(float(v) for v in res), rmax, dt, self.cfg.get("CFL", 0.5)])
            t += dt
        return q, np.array(rec)


def _wall(p, n):
    z = torch.zeros_like(p)
    return torch.stack([z, p * n[:, 0], p * n[:, 1], z], 1)
