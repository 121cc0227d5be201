"""The workloads whose speed this repository is judged by, as a user's program calls them.

A case is a dict of plain values; ``prepare`` makes its inputs from a seed, ``run``
is one pass through the public entry points of ``sqbem``, ``work`` counts what the
pass cannot do without and ``exact`` solves the same boundary-element problem in
64-bit torch, independently of the library.

Kinds of case:

  velocity    velocity_at: the representation formula at points inside a duct
  unbounded   one squirmer in the unbounded fluid, through the handles
  swimmer     Tube + SwimmerSolver + solve_free + solve_prescribed, through the handles
  duct        DuctFlow: factor once, one solve per pressure drop, a velocity profile
  batch       kinematics_batch with tractions: the (a/R, beta) rows of a sweep
  adjoint     adjoint_batch: U, Omega and their derivatives by the sphere's position
  ensemble    trajectory_ensemble: time steps of swimmers that share a tube
  field       ensemble_field: the velocity on a 3-D grid around swimmers

Sizes are those of the five benchmark workloads (sqbem/workloads.py), of the
library's defaults (trajectories: n_theta = 30) and of the tests.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "squirmer-bem-3dtube_gb300"))
import sqbem  # noqa: E402

PRECISION = {"fp64": sqbem.FP64, "mixed": sqbem.MIXED}


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the 60 profile points of the duct program: the smallest call, all latency
        dict(name="profile_60pts", kind="velocity", n_theta=24, n_z=24, n_r=6, points=60, precision="fp64"),
        # a sphere in the unbounded fluid, as the tests and a first user run it
        dict(name="unbounded_l1", kind="unbounded", level=1, precision="fp64"),
        # an odd, ragged tube at the level the trajectories use
        dict(name="swimmer_fp64_odd", kind="swimmer", a_over_R=0.37, L_over_R=3.1, n_theta=17, n_r=3, level=2,
             precision="fp64"),
        # the kinematics workload in both precisions: 1280 sphere panels, n_theta = 24
        dict(name="swimmer_fp64_l3", kind="swimmer", a_over_R=0.3, L_over_R=4.0, n_theta=24, n_r=4, level=3,
             precision="fp64"),
        dict(name="swimmer_mixed_l3", kind="swimmer", a_over_R=0.3, L_over_R=4.0, n_theta=24, n_r=4, level=3,
             precision="mixed"),
        # the duct workload: 1680 panels, four pressure drops, a profile
        dict(name="duct_fp64", kind="duct", n_theta=24, n_z=24, n_r=6, precision="fp64"),
        # rows of the sweep in FP64, and the whole sweep in mixed precision
        dict(name="sweep4_fp64", kind="batch", n=4, lam_lo=0.1, lam_hi=0.6, n_theta=24, L_over_R=4.0, level=0,
             precision="fp64"),
        dict(name="sweep128_mixed", kind="batch", n=128, lam_lo=0.1, lam_hi=0.6, n_theta=24, L_over_R=4.0, level=0,
             precision="mixed"),
        # sensitivities of the adjoint workload (backward direction)
        dict(name="adjoint2", kind="adjoint", n=2, lam_lo=0.2, lam_hi=0.5, n_theta=24, L_over_R=4.0, level=2),
        # one step of a single FP64 trajectory with the library's default tube
        dict(name="trajectory_fp64", kind="ensemble", n=1, steps=1, a_over_R=0.3, n_theta=30, level=2,
             precision="fp64"),
        # one RK4 step of the 256-swimmer ensemble
        dict(name="ensemble256_mixed", kind="ensemble", n=256, steps=1, a_over_R=0.3, n_theta=24, level=2,
             precision="mixed"),
        # the ensemble's field output for a few swimmers
        dict(name="field4_mixed", kind="field", n=4, nx=25, nz=41, a_over_R=0.3, n_theta=24, level=2,
             precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["velocity", "unbounded", "swimmer", "swimmer", "swimmer", "duct", "batch", "batch", "adjoint",
                       "ensemble", "field"])
    prec = rng.choice(["fp64", "mixed"])
    lam = round(rng.uniform(0.2, 0.55), 3)
    if kind == "velocity":
        return dict(kind=kind, n_theta=rng.randint(7, 30), n_z=rng.randint(5, 28), n_r=rng.randint(2, 6),
                    points=_log(rng, 10, 20000), precision=prec)
    if kind == "unbounded":
        return dict(kind=kind, level=rng.choice([1, 2, 3]), precision=prec, radius=round(rng.uniform(0.5, 2), 3))
    if kind == "swimmer":
        return dict(kind=kind, a_over_R=lam, L_over_R=round(rng.uniform(2.5, 4.0), 2), n_theta=rng.randint(9, 24),
                    n_r=rng.randint(2, 4), level=rng.choice([1, 2, 2, 3]), precision=prec)
    if kind == "duct":
        return dict(kind=kind, n_theta=rng.randint(9, 24), n_z=rng.randint(6, 24), n_r=rng.randint(2, 6),
                    precision="fp64")
    if kind == "batch":
        n = rng.randint(1, 3) if prec == "fp64" else _log(rng, 1, 96)
        return dict(kind=kind, n=n, lam_lo=0.15, lam_hi=0.55, n_theta=rng.randint(10, 24),
                    L_over_R=round(rng.uniform(3.0, 4.0), 2), level=rng.choice([0, 2]), precision=prec)
    if kind == "adjoint":
        return dict(kind=kind, n=rng.randint(1, 2), lam_lo=0.2, lam_hi=0.5, n_theta=rng.randint(9, 24),
                    L_over_R=round(rng.uniform(2.5, 4.0), 2), level=rng.choice([1, 2]))
    if kind == "ensemble":
        n = 1 if prec == "fp64" else _log(rng, 1, 200)
        return dict(kind=kind, n=n, steps=1, a_over_R=lam, n_theta=rng.randint(10, 30), level=rng.choice([1, 2]),
                    precision=prec)
    return dict(kind=kind, n=rng.randint(1, 4), nx=rng.randint(9, 25), nz=rng.randint(11, 41), a_over_R=lam,
                n_theta=rng.randint(10, 24), level=rng.choice([1, 2]), precision="mixed")


# ---------------------------------------------------------------- inputs
def _unit(v):
    return v / np.linalg.norm(v)


def _instances(case, seed):
    """Instances of a sweep or an adjoint batch, drawn like sqbem/workloads.py draws them.  The confinements and
    levels are the case's own, so that every seed gives arrays of the same shapes; offsets and directions vary."""
    rng, sizes = np.random.default_rng([seed, 11]), np.random.default_rng(case["n"])
    out = []
    for k in range(case["n"]):
        lam = sizes.uniform(case["lam_lo"], case["lam_hi"])
        beta = rng.uniform(0.0, 0.8 * (1.0 - lam)) if case["kind"] == "batch" else rng.uniform(0.0, 0.5)
        level = case["level"] or 2 + k % 2
        out.append(dict(a_over_R=float(lam), beta=float(beta), L_over_R=case["L_over_R"],
                        e=tuple(map(float, _unit(rng.normal(size=3)))), n_theta=case["n_theta"], n_r=4,
                        sphere_level=level, towed=0))
    return out


def _swimmer_input(case, seed):
    rng = np.random.default_rng([seed, 12])
    R = 1.0 / case["a_over_R"] if "a_over_R" in case else 0.0
    b = float(rng.uniform(0.05, 0.6) * (R - 1.0)) if R else 0.0
    return dict(R=R, c=np.array([b, 0.0, 0.0]), e=_unit(rng.normal(size=3)), U=rng.normal(size=3),
                Om=rng.normal(size=3))


def _swarm(case, seed):
    rng = np.random.default_rng([seed, 13])
    n, R = case["n"], 1.0 / case["a_over_R"]
    y = np.zeros((n, 6))
    y[:, 0] = rng.uniform(0.0, 0.6, n) * (R - 1.0)
    e = rng.normal(size=(n, 3))
    y[:, 3:] = e / np.linalg.norm(e, axis=1)[:, None]
    return y, rng.uniform(-5.0, 5.0, n)


def _traj_params(case):
    return sqbem.TrajParams(a_over_R=case["a_over_R"], n_theta=case["n_theta"], sphere_level=case["level"], dt=0.05)


def _duct_points(case):
    r = np.linspace(0.0, 0.95, 20)
    return np.concatenate([np.stack([r * math.cos(p), r * math.sin(p), np.full(20, 2.0)], 1)
                           for p in (0.0, math.pi / 5, math.pi / 2)])


def _velocity_input(case, seed):
    """A duct's panels with smooth boundary data and points inside it."""
    rng = np.random.default_rng([seed, 14])
    P = 2 * case["n_theta"] * case["n_z"] + 2 * case["n_theta"] * (2 * case["n_r"] - 1)
    n = case["points"]
    r, t, z = 0.95 * np.sqrt(rng.uniform(size=n)), rng.uniform(0, 2 * math.pi, n), rng.uniform(0.05, 3.95, n)
    pts = np.stack([r * np.cos(t), r * np.sin(t), z], 1)
    return rng.normal(size=(P, 3)), rng.normal(size=(P, 3)), pts


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case, precision=PRECISION[case.get("precision", "fp64")])
    if kind == "velocity":
        s["u"], s["f"], s["points"] = _velocity_input(case, seed)
        s["mesh"] = sqbem.tube_mesh(1.0, sqbem.uniform_z(0.0, 4.0, case["n_z"]), case["n_theta"], case["n_r"])
    elif kind == "unbounded" or kind == "swimmer":
        s.update(_swimmer_input(case, seed))
        s["sphere"] = sqbem.icosphere(case.get("radius", 1.0), case["level"], s["c"])
    elif kind == "duct":
        s["drops"] = [float(x) for x in np.random.default_rng([seed, 15]).uniform(0.5, 4.0, 4)]
        s["points"] = _duct_points(case)
    elif kind == "batch" or kind == "adjoint":
        s["instances"] = _instances(case, seed)
    elif kind == "ensemble":
        s["y0"], s["alpha"] = _swarm(case, seed)
        s["params"] = _traj_params(case)
    elif kind == "field":
        s["y0"], s["alpha"] = _swarm(case, seed)
        s["params"] = _traj_params(case)
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    kind, prec, case = s["kind"], s["precision"], s["case"]
    if kind == "velocity":
        return sqbem.velocity_at(s["mesh"], s["u"], s["f"], 1.0, s["points"], prec)
    if kind == "unbounded" or kind == "swimmer":
        tube = None
        if kind == "swimmer":
            tube = sqbem.Tube(s["R"], case["L_over_R"] * s["R"], 1.0, case["n_theta"], case["n_r"], 1.0, prec)
        solver = sqbem.SwimmerSolver(tube, s["sphere"], s["c"], 1.0, prec)
        free = solver.solve_free([solver.slip(s["e"], 1.0, 0.0), solver.slip(s["e"], 0.0, 1.0)])
        towed = solver.solve_prescribed(s["U"], s["Om"])
        solver.close()
        out = dict(motion=np.stack([np.concatenate([m.U, m.Om]) for m in free]),
                   f_sphere=np.stack([m.f_sphere for m in free + [towed]]))
        if tube:
            out["f_tube"] = np.stack([m.f_tube for m in free + [towed]])
            tube.close()
        return out
    if kind == "duct":
        duct = sqbem.DuctFlow(1.0, 4.0, case["n_theta"], case["n_z"], case["n_r"], 1.0, prec)
        sols = [duct.solve(dp, 0.0) for dp in s["drops"]]
        v = duct.velocity(sols[0], s["points"])
        duct.close()
        return dict(Q=np.array([x.Q for x in sols]), u=np.stack([x.u for x in sols]),
                    f=np.stack([x.f for x in sols]), profile=v)
    if kind == "batch":
        res, _, fs, ft = sqbem.kinematics_batch(s["instances"], prec, tractions=True)
        return dict(motion=res[:, :12], panels=res[:, 13:15].astype(np.int64),
                    f_sphere=np.concatenate([f.ravel() for f in fs]), f_tube=np.concatenate([f.ravel() for f in ft]))
    if kind == "adjoint":
        d, _ = sqbem.adjoint_batch(s["instances"])
        return d
    if kind == "ensemble":
        states, U, Om, status, _ = sqbem.trajectory_ensemble(s["y0"], s["alpha"], s["params"], case["steps"], 1, prec)
        return dict(states=states, motion=np.concatenate([U, Om], axis=2), status=status)
    u, _ = sqbem.ensemble_field(s["y0"], s["alpha"], s["params"], case["nx"], case["nx"], case["nz"], 7.0, prec)
    return u


# ---------------------------------------------------------------- what a pass cannot do without
PAIR = 7 * 64.0  # the 7-point rule, 64 operations a node


def _tube_panels(a_over_R, L_over_R, n_theta, n_r):
    R = 1.0 / a_over_R
    h = 2 * math.pi * R / n_theta
    nz = len(_graded_z(L_over_R * R, 0.6 * h, 1.4 * h, 1.0 + 0.5 * R)) - 1
    return 2 * n_theta * nz + 2 * n_theta * (2 * n_r - 1)


def _solve_work(nt, ns, with_tube=True):
    """Assembly of the blocks, LU of the tube and of the sphere's Schur complement, its product."""
    t, s = 3.0 * nt, 3.0 * ns
    tube = PAIR * nt * nt + 2.0 / 3.0 * t ** 3 if with_tube else 0.0
    return tube + PAIR * (2.0 * nt * ns + ns * ns) + 2.0 * t * t * s + 2.0 * s * s * t + 2.0 / 3.0 * s ** 3


def work(case):
    """Bytes: host inputs and outputs once.  Operations: pair integrals and the dense solves."""
    kind = case["kind"]
    if kind == "velocity":
        P = 2 * case["n_theta"] * case["n_z"] + 2 * case["n_theta"] * (2 * case["n_r"] - 1)
        return dict(bytes=8.0 * (9 + 6) * P + 48.0 * case["points"], flops=PAIR * P * case["points"])
    if kind == "duct":
        P = 2 * case["n_theta"] * case["n_z"] + 2 * case["n_theta"] * (2 * case["n_r"] - 1)
        n = 3.0 * P
        return dict(bytes=8.0 * (9 * P + 4 * 2 * n), flops=PAIR * P * P + 2.0 / 3.0 * n ** 3 + 4 * 2 * n * n)
    if kind == "unbounded":
        ns = 20 * 4 ** case["level"]
        return dict(bytes=8.0 * ns * (9 + 2 * 3 + 3 * 3), flops=_solve_work(0, ns))
    if kind == "swimmer":
        nt = _tube_panels(case["a_over_R"], case["L_over_R"], case["n_theta"], case["n_r"])
        ns = 20 * 4 ** case["level"]
        return dict(bytes=8.0 * (ns * (9 + 6 + 9) + nt * 9), flops=_solve_work(nt, ns))
    if kind in ("batch", "adjoint"):
        nt = _tube_panels(0.5 * (case["lam_lo"] + case["lam_hi"]), case["L_over_R"], case["n_theta"], 4)
        levels = [case["level"]] if case["level"] else [2, 3]
        one = [(20 * 4 ** lv) for lv in levels]
        flops = case["n"] * sum(_solve_work(nt, ns) for ns in one) / len(one)
        back = 48.0 if kind == "adjoint" else 16.0 + 6.0 * (nt + sum(one) / len(one))
        return dict(bytes=8.0 * case["n"] * (8 + back), flops=flops)
    nt = _tube_panels(case["a_over_R"], 4.0, case["n_theta"], 4)
    ns = 20 * 4 ** case["level"]
    if kind == "ensemble":
        evals = 4.0 * case["n"] * case["steps"]
        return dict(bytes=8.0 * case["n"] * (7 + 6 * (case["steps"] + 1) + 6 * case["steps"]),
                    flops=evals * _solve_work(nt, ns, False))
    pts = case["nx"] * case["nx"] * case["nz"]
    return dict(bytes=8.0 * case["n"] * (7 + 3 * pts),
                flops=case["n"] * (_solve_work(nt, ns, False) + 0.74 * PAIR * pts * (nt + ns)))


# ---------------------------------------------------------------- the same problems in 64-bit torch
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _graded_z(L, dzmin, dzmax, core):
    half, pos, dz = L / 2, [0.0], dzmin
    while pos[-1] < half - 1e-12:
        if pos[-1] >= core:
            dz = min(dz * 1.25, dzmax)
        pos.append(min(pos[-1] + dz, half))
    if len(pos) > 2 and half - pos[-2] < 0.3 * dz:
        del pos[-2]
    return [-p for p in reversed(pos)] + pos[1:]


def _oriented(nodes, tris, direction):
    """Triangles flipped so that their normal points along direction(centroid)."""
    V = nodes[tris]
    n = np.cross(V[:, 1] - V[:, 0], V[:, 2] - V[:, 0])
    flip = np.einsum("pc,pc->p", n, direction(V.mean(axis=1))) < 0
    V[flip] = V[flip][:, [0, 2, 1]]
    return V


def _tube_vertices(R, z, nth, nr):
    """Panels (P, 3, 3) of the closed tube, and a mask of its inlet (1) and outlet (2) panels."""
    al = 2 * math.pi / nth
    Rp = R * math.sqrt(al / math.sin(al))
    nz = len(z) - 1
    ang = [(math.cos(i * al), math.sin(i * al)) for i in range(nth)]
    nodes = np.array([(Rp * c, Rp * s, zz) for c, s in ang for zz in z])
    node = lambda i, k: (i % nth) * (nz + 1) + k  # noqa: E731
    tris = []
    for i in range(nth):
        for k in range(nz):
            a, b, c, d = node(i, k), node(i + 1, k), node(i + 1, k + 1), node(i, k + 1)
            tris += [(a, b, c), (a, c, d)]
    parts = [_oriented(nodes, np.array(tris), lambda x: x * np.array([1.0, 1.0, 0.0]))]
    for z0, sign in ((z[0], -1.0), (z[-1], 1.0)):
        cap = [(0.0, 0.0, z0)] + [(Rp * k / nr * c, Rp * k / nr * s, z0) for k in range(1, nr + 1) for c, s in ang]
        cn = lambda ring, i: 1 + ring * nth + i % nth  # noqa: E731
        tris = [(0, cn(0, i), cn(0, i + 1)) for i in range(nth)]
        for k in range(nr - 1):
            for i in range(nth):
                a, b, c, d = cn(k, i), cn(k, i + 1), cn(k + 1, i + 1), cn(k + 1, i)
                tris += [(a, d, c), (a, c, b)]
        parts.append(_oriented(np.array(cap), np.array(tris),
                               lambda x, s=sign: np.broadcast_to(np.array([0.0, 0.0, s]), x.shape)))
    tag = np.concatenate([np.full(len(p), k) for k, p in enumerate(parts)])
    return np.concatenate(parts), tag


def _swimmer_tube_vertices(R, L, nth, nr):
    h = 2 * math.pi * R / nth
    return _tube_vertices(R, _graded_z(L, 0.6 * h, 1.4 * h, 1.0 + 0.5 * R), nth, nr)[0]


def _icosphere_vertices(level, center):
    g = (1 + math.sqrt(5.0)) / 2
    one = lambda x: x * (1.0 / math.sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]))  # noqa: E731
    v = [one(np.array(x, float)) for x in
         [(-1, g, 0), (1, g, 0), (-1, -g, 0), (1, -g, 0), (0, -1, g), (0, 1, g), (0, -1, -g), (0, 1, -g), (g, 0, -1),
          (g, 0, 1), (-g, 0, -1), (-g, 0, 1)]]
    F = [(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2), (10, 7, 6),
         (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11), (6, 2, 10),
         (8, 6, 7), (9, 8, 1)]
    for _ in range(level):
        mid, nxt = {}, []

        def half(i, j):
            key = (min(i, j), max(i, j))
            if key not in mid:
                mid[key] = len(v)
                v.append(one(v[i] + v[j]))
            return mid[key]

        for a, b, c in F:
            ab, bc, ca = half(a, b), half(b, c), half(c, a)
            nxt += [(a, ab, ca), (b, bc, ab), (c, ca, bc), (ab, bc, ca)]
        F = nxt
    nodes, F = np.array(v), np.array(F)
    W = nodes[F]
    vol = abs(sum(float(a @ b) for a, b in zip(W[:, 0], np.cross(W[:, 1], W[:, 2])))) / 6
    nodes = np.asarray(center)[None, :] + float(np.cbrt(4 * math.pi / 3 / vol)) * nodes
    return _oriented(nodes, F, lambda x: np.asarray(center)[None, :] - x)


def _rules():
    """Barycentric points and weights of the 7-point rule on 1, 4, 16 and 64 sub-triangles."""
    a1, b1, w1 = 0.059715871789770, 0.470142064105115, 0.132394152788506
    a2, b2, w2 = 0.797426985353087, 0.101286507323456, 0.125939180544827
    L = [(1 / 3, 1 / 3, 1 / 3)]
    for a, b in ((a1, b1), (a2, b2)):
        L += [(a, b, b), (b, a, b), (b, b, a)]
    L, W = np.array(L), np.array([0.225] + [w1] * 3 + [w2] * 3)
    tris, out = [np.eye(3)], []
    for _ in range(4):
        out.append((np.concatenate([L @ t for t in tris]), np.concatenate([W / len(tris)] * len(tris))))
        nxt = []
        for p, q, r in tris:
            pq, qr, rp = (p + q) / 2, (q + r) / 2, (r + p) / 2
            nxt += [np.array([p, pq, rp]), np.array([pq, q, qr]), np.array([rp, qr, r]), np.array([pq, qr, rp])]
        tris = nxt
    return out


class _Panels:
    """Vertices, normals, centroids and areas of panels, on the device."""

    def __init__(self, V):
        self.V = torch.as_tensor(np.ascontiguousarray(V), dtype=torch.float64, device=_dev()).reshape(-1, 3, 3)
        c = torch.cross(self.V[:, 1] - self.V[:, 0], self.V[:, 2] - self.V[:, 0], dim=1)
        nn = torch.sqrt((c * c).sum(1))
        self.n, self.area, self.h = c / nn[:, None], 0.5 * nn, torch.sqrt(nn)
        self.c = (self.V[:, 0] + self.V[:, 1] + self.V[:, 2]) / 3.0
        self.P = self.V.shape[0]


def _nodes_sum(r, w, m):
    """Sums over the last-but-one axis (nodes) of w G(r) and w T(r).m; r (..., q, 3), w (..., q), m (..., 3)."""
    r2 = (r * r).sum(-1)
    ir = 1.0 / torch.sqrt(r2)
    ir3 = ir ** 3
    S = r.mT @ ((w * ir3)[..., None] * r)
    S = S + (w * ir).sum(-1)[..., None, None] * torch.eye(3, dtype=r.dtype, device=r.device)
    d = -6.0 * w * (r * m[..., None, :]).sum(-1) * ir3 * ir ** 2
    return S, r.mT @ (d[..., None] * r)


def _block(x0, src, same=False, shift=None):
    """Single- and double-layer integrals SL, DL (nT, nS, 3, 3).  With `shift` (3 values) the separation
    source - target is moved by i * shift * 1e-30, so the imaginary parts / 1e-30 are the derivatives."""
    dev = x0.device
    rules = [(torch.as_tensor(a, device=dev), torch.as_tensor(b, device=dev)) for a, b in _rules()]
    dt = torch.float64 if shift is None else torch.complex128
    mv = None if shift is None else 1e-30j * torch.as_tensor(shift, dtype=torch.complex128, device=dev)
    nT, nS = x0.shape[0], src.P
    SL = torch.zeros((nT, nS, 3, 3), dtype=dt, device=dev)
    DL = torch.zeros_like(SL)
    step = max(1, 200_000 // max(nS, 1))
    for i0 in range(0, nT, step):
        x = x0[i0:i0 + step]
        d = src.c[None] - x[:, None]
        dist = torch.sqrt(d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2]) / src.h[None]
        level = (dist < 3.0).int() + (dist < 1.5).int() + (dist < 0.75).int()
        own = torch.zeros_like(level, dtype=torch.bool)
        if same:
            k = torch.arange(x.shape[0], device=dev)
            own[k, i0 + k] = True
        for lv, (lam, w) in enumerate(rules):
            for part in ((level == lv) & ~own).nonzero().split(max(1, 1_500_000 // len(w))):
                if not len(part):
                    continue
                i, p = part[:, 0], part[:, 1]
                r = torch.einsum("qk,nkc->nqc", lam, src.V[p]) - x[i][:, None]
                r = r if mv is None else r + mv
                ww = (w[None] * src.area[p][:, None]).to(dt)
                SL[i0 + i, p], DL[i0 + i, p] = _nodes_sum(r, ww, src.n[p].to(dt))
    if same:
        gx, gw = np.polynomial.legendre.leggauss(10)
        gx, gw = torch.as_tensor(0.5 * (gx + 1), device=dev), torch.as_tensor(0.5 * gw, device=dev)
        u, v = [t.reshape(-1) for t in torch.meshgrid(gx, gx, indexing="ij")]
        w = (gw[:, None] * gw[None, :]).reshape(-1)
        k = torch.arange(nT, device=dev)
        SL[k, k], DL[k, k] = 0, 0
        for e in range(3):
            e1, e2 = src.V[:, e] - x0, src.V[:, (e + 1) % 3] - x0
            J = torch.linalg.norm(torch.cross(e1, e2, dim=1), dim=1)
            r = u[None, :, None] * ((1 - v)[None, :, None] * e1[:, None] + v[None, :, None] * e2[:, None])
            SL[k, k] += _nodes_sum(r, (w * u)[None] * J[:, None], src.n)[0]
    return SL, DL


def _flat(B):
    return B.permute(0, 2, 1, 3).reshape(3 * B.shape[0], 3 * B.shape[1])


def _deflate(A, p):
    A += (1.0 / (8 * math.pi * torch.sqrt(p.area.sum()))) * torch.outer(p.n.reshape(-1),
                                                                        (p.n * p.area[:, None]).reshape(-1))


class _Exact:
    """The full system [T B A_uBt K; D E A_uBs K; 0 F 0] of a squirmer in a tube (or in the unbounded fluid)."""

    def __init__(self, tube, sphere, c):
        k8 = 8 * math.pi
        self.t, self.s, self.nt, self.ns = tube, sphere, 3 * tube.P if tube else 0, 3 * sphere.P
        nt, ns, dev = self.nt, self.ns, sphere.V.device
        r = sphere.c - torch.as_tensor(c, device=dev)[None]
        self.r = r
        K = torch.zeros((ns, 6), dtype=torch.float64, device=dev)
        F = torch.zeros((6, ns), dtype=torch.float64, device=dev)
        for a in range(3):
            b, g = (a + 1) % 3, (a + 2) % 3
            K[a::3, a] = 1
            K[g::3, 3 + a] = r[:, b]   # (Omega x r): Omega along a turns r_b into g ...
            K[b::3, 3 + a] = -r[:, g]  # ... and r_g into -b
            F[a, a::3] = sphere.area
            F[3 + a, g::3] = sphere.area * r[:, b]
            F[3 + a, b::3] = -sphere.area * r[:, g]
        E, AuBs = [_flat(x) for x in _block(sphere.c, sphere, True)]
        E, AuBs = E / k8, AuBs / -k8
        diag = -AuBs.reshape(ns, -1, 3).sum(1)  # (ns, 3): minus the row sums over the panels
        _deflate(E, sphere)
        A = torch.zeros((nt + ns + 6, nt + ns + 6), dtype=torch.float64, device=dev)
        if tube:
            T = _flat(_block(tube.c, tube, True)[0]) / k8
            _deflate(T, tube)
            B, AuBt = [_flat(x) for x in _block(tube.c, sphere)]
            D, Dd = [_flat(x) for x in _block(sphere.c, tube)]
            self.AuBt = AuBt / -k8
            diag = diag + (Dd / k8).reshape(ns, -1, 3).sum(1)
            A[:nt, :nt], A[:nt, nt:nt + ns], A[nt:nt + ns, :nt] = T, B / k8, D / k8
            A[:nt, nt + ns:] = self.AuBt @ K
        else:
            self.AuBt = torch.zeros((0, ns), dtype=torch.float64, device=dev)
            diag = diag - torch.eye(3, dtype=torch.float64, device=dev).repeat(sphere.P, 1)
        for p in range(3):
            for q in range(3):
                AuBs[torch.arange(p, ns, 3), torch.arange(q, ns, 3)] += diag[p::3, q]
        A[nt:nt + ns, nt:nt + ns], A[nt:nt + ns, nt + ns:], A[nt + ns:, nt:nt + ns] = E, AuBs @ K, F
        self.A, self.AuBs, self.K = A, AuBs, K
        self.lu = torch.linalg.lu_factor(A)

    def slip(self, e, B1, B2):
        rh = self.r / torch.linalg.norm(self.r, dim=1)[:, None]
        e = torch.as_tensor(np.asarray(e, float), device=rh.device)
        ct = rh @ e
        return (B1 + B2 * ct)[:, None] * (ct[:, None] * rh - e)

    def free(self, slips):
        u = torch.stack([x.reshape(-1) for x in slips], 1)
        b = torch.zeros((self.nt + self.ns + 6, u.shape[1]), dtype=u.dtype, device=u.device)
        b[:self.nt], b[self.nt:self.nt + self.ns] = -self.AuBt @ u, -self.AuBs @ u
        x = torch.linalg.lu_solve(*self.lu, b)
        return x + torch.linalg.lu_solve(*self.lu, b - self.A @ x)

    def prescribed(self, U, Om):
        w = torch.as_tensor(np.concatenate([U, Om]), device=self.A.device)
        m = self.nt + self.ns
        return torch.cat([torch.linalg.solve(self.A[:m, :m], -(self.A[:m, m:] @ w)), w])

    def split(self, x):
        """(U, Omega) rows, f_sphere, f_tube of the solution columns x."""
        n = self.nt + self.ns
        k = x.shape[1]
        return (x[n:].T.cpu().numpy().copy(), x[self.nt:n].T.reshape(k, -1, 3).cpu().numpy().copy(),
                x[:self.nt].T.reshape(k, -1, 3).cpu().numpy().copy())

    def position_derivatives(self, slips, x):
        """d(U, Omega)/dc_j for the solutions x: (nrhs, 6, 3)."""
        nt, ns, k8 = self.nt, self.ns, 8 * math.pi
        u = torch.stack([s.reshape(-1) for s in slips], 1)
        w = u + self.K @ x[nt + ns:]  # velocity of the sphere's surface
        out = []
        for j in range(3):
            step = [1.0 if a == j else 0.0 for a in range(3)]
            dB, dAt = [_flat(t.imag / 1e-30) for t in _block(self.t.c, self.s, shift=step)]
            dD, dDd = [_flat(t.imag / 1e-30) for t in _block(self.s.c, self.t, shift=[-a for a in step])]
            dg = (dDd / k8).reshape(ns, -1, 3).sum(1).reshape(-1, 3, 3)
            db = torch.zeros_like(x)
            db[:nt] = -(dB / k8 @ x[nt:nt + ns] + dAt / -k8 @ w)
            db[nt:nt + ns] = -(dD / k8 @ x[:nt] + torch.einsum("pab,pbk->pak", dg, w.reshape(-1, 3, w.shape[1]))
                               .reshape(ns, -1))
            out.append(torch.linalg.lu_solve(*self.lu, db)[nt + ns:].T)
        return torch.stack(out, 2).cpu().numpy()


def _exact_of(a_over_R, L_over_R, n_theta, n_r, level, c):
    R = 1.0 / a_over_R
    tube = _Panels(_swimmer_tube_vertices(R, L_over_R * R, n_theta, n_r))
    return _Exact(tube, _Panels(_icosphere_vertices(level, c)), c)


def _exact_velocity(src, u, f, pts):
    x = torch.as_tensor(pts, device=_dev())
    u, f = (torch.as_tensor(t, device=_dev()) for t in (u, f))
    out = []
    for part in x.split(max(1, 3_000_000 // src.P)):
        SL, DL = _block(part, src)
        out.append((torch.einsum("ipab,pb->ia", SL, f) - torch.einsum("ipab,pb->ia", DL, u)) / (8 * math.pi))
    return torch.cat(out).cpu().numpy()


def _exact_duct(case, seed):
    V, tag = _tube_vertices(1.0, [4.0 * k / case["n_z"] for k in range(case["n_z"] + 1)], case["n_theta"], case["n_r"])
    p, k8 = _Panels(V), 8 * math.pi
    S, D = [_flat(x) / k8 for x in _block(p.c, p, True)]
    cap = np.nonzero(tag)[0]
    zc = torch.as_tensor(3 * cap + 2, device=S.device)
    M, Fk = S.clone(), S[:, zc].clone()
    M[:, zc] = -D[:, zc]
    rows = D.reshape(3 * p.P, -1, 3).sum(1)
    for a in range(3):
        M[torch.as_tensor(3 * cap + a, device=S.device), zc] += rows[3 * cap + a, 2]
    lu = torch.linalg.lu_factor(M)
    Q, us, fs = [], [], []
    drops = [float(x) for x in np.random.default_rng([seed, 15]).uniform(0.5, 4.0, 4)]
    for dp in drops:
        fk = torch.as_tensor(np.where(tag[cap] == 1, dp, -0.0), device=S.device)
        b = -(Fk @ fk)[:, None]
        x = torch.linalg.lu_solve(*lu, b)
        x = (x + torch.linalg.lu_solve(*lu, b - M @ x))[:, 0].reshape(-1, 3)
        u, f = torch.zeros_like(x), x.clone()
        u[cap, 2], f[cap, 2] = x[cap, 2], fk
        out = np.nonzero(tag == 2)[0]
        Q.append(float((u[out, 2] * p.area[out]).sum()))
        us.append(u.cpu().numpy())
        fs.append(f.cpu().numpy())
    return dict(Q=np.array(Q), u=np.stack(us), f=np.stack(fs), profile=_exact_velocity(p, us[0], fs[0],
                                                                                       _duct_points(case)))


def _exact_motion(case, y, alpha):
    """d/dt of the state (x, y, z, e) of one swimmer, and its (U, Omega)."""
    e = _unit(y[3:])
    c = np.array([y[0], y[1], 0.0])
    E = _exact_of(case["a_over_R"], 4.0, case["n_theta"], 4, case["level"], c)
    w, _, _ = E.split(E.free([E.slip(e, 1.0, 0.0), E.slip(e, 0.0, 1.0)]))
    w = w[0] + alpha * w[1]
    return np.concatenate([w[:3], np.cross(w[3:], e)]), w


def exact(case, seed):
    kind = case["kind"]
    if kind == "velocity":
        u, f, pts = _velocity_input(case, seed)
        V, _ = _tube_vertices(1.0, [4.0 * k / case["n_z"] for k in range(case["n_z"] + 1)], case["n_theta"],
                              case["n_r"])
        return _exact_velocity(_Panels(V), u, f, pts)
    if kind in ("unbounded", "swimmer"):
        s = _swimmer_input(case, seed)
        E = (_Exact(None, _Panels(case.get("radius", 1.0) * _icosphere_vertices(case["level"], s["c"])), s["c"])
             if kind == "unbounded" else _exact_of(case["a_over_R"], case["L_over_R"], case["n_theta"], case["n_r"],
                                                  case["level"], s["c"]))
        w, fs, ft = E.split(E.free([E.slip(s["e"], 1.0, 0.0), E.slip(s["e"], 0.0, 1.0)]))
        _, ps, pt = E.split(E.prescribed(s["U"], s["Om"])[:, None])
        out = dict(motion=w, f_sphere=np.concatenate([fs, ps]))
        if kind == "swimmer":
            out["f_tube"] = np.concatenate([ft, pt])
        return out
    if kind == "duct":
        return _exact_duct(case, seed)
    if kind == "batch" and case["n"] <= 8 or kind == "adjoint":
        ws, fs, ft, dw, panels = [], [], [], [], []
        for q in _instances(case, seed):
            c = np.array([q["beta"] * (1.0 / q["a_over_R"] - 1.0), 0.0, 0.0])
            E = _exact_of(q["a_over_R"], q["L_over_R"], q["n_theta"], q["n_r"], q["sphere_level"], c)
            slips = [E.slip(q["e"], 1.0, 0.0), E.slip(q["e"], 0.0, 1.0)]
            x = E.free(slips)
            w, s, t = E.split(x)
            ws.append(w)
            fs.append(s.ravel())
            ft.append(t.ravel())
            panels.append([E.nt // 3, E.ns // 3])
            if kind == "adjoint":
                dw.append(E.position_derivatives(slips, x))
        w = np.stack(ws)
        if kind == "adjoint":
            dw = np.stack(dw)
            return dict(U=w[:, :, :3], Om=w[:, :, 3:], dU_dc=dw[:, :, :3], dOm_dc=dw[:, :, 3:])
        return dict(motion=w.reshape(-1, 12), panels=np.array(panels), f_sphere=np.concatenate(fs),
                    f_tube=np.concatenate(ft))
    if kind == "ensemble" and case["n"] <= 4:
        y0, alpha = _swarm(case, seed)
        states, motion, dt = [], [], 0.05
        for y, al in zip(y0, alpha):
            k1, w = _exact_motion(case, y, al)
            k2, _ = _exact_motion(case, y + dt / 2 * k1, al)
            k3, _ = _exact_motion(case, y + dt / 2 * k2, al)
            k4, _ = _exact_motion(case, y + dt * k3, al)
            z = y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
            z[3:] = _unit(z[3:])
            states.append([y, z])
            motion.append([w])
        return dict(states=np.array(states), motion=np.array(motion), status=None)
    if kind == "field":
        y0, alpha = _swarm(case, seed)
        R, nx, nz = 1.0 / case["a_over_R"], case["nx"], case["nz"]
        lim = 0.97 * R
        ax = -lim + 2 * lim * np.arange(nx) / (nx - 1)
        az = -7.0 + 14.0 * np.arange(nz) / (nz - 1)
        X = np.stack(np.meshgrid(ax, ax, az, indexing="ij"), -1)
        out = []
        for y, al in zip(y0, alpha):
            c, e = np.array([y[0], y[1], 0.0]), _unit(y[3:])
            E = _exact_of(case["a_over_R"], 4.0, case["n_theta"], 4, case["level"], c)
            slips = [E.slip(e, 1.0, 0.0), E.slip(e, 0.0, 1.0)]
            x = E.free(slips)
            x = x[:, 0] + al * x[:, 1]
            u = torch.zeros((E.t.P + E.s.P, 3), dtype=torch.float64, device=x.device)
            u[E.t.P:] = (E.K @ x[E.nt + E.ns:]).reshape(-1, 3) + slips[0] + al * slips[1]
            both = _Panels(torch.cat([E.t.V, E.s.V]).cpu().numpy())
            D = X - c
            ok = ((X[..., 0] * X[..., 0] + X[..., 1] * X[..., 1] <= lim * lim)
                  & ~(np.sqrt(D[..., 0] * D[..., 0] + D[..., 1] * D[..., 1] + D[..., 2] * D[..., 2]) < 1.03))
            v = np.full(X.shape, np.nan)
            v[ok] = _exact_velocity(both, u, x[:E.nt + E.ns].reshape(-1, 3), X[ok])
            out.append(v)
        return np.stack(out)
    return None
