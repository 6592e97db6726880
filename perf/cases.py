"""Workloads of the narrow phase and the time step, for timing.

A case names a kind of call, a scene and its size.  Scenes are the ones of
this repository's configurations (cube lattices, icosphere piles, the torus
chain, hull piles, slab stacks), in contact states drawn from the seed, so
that the calls meet what a running simulation gives them: near contacts,
resting contacts and bodies about to collide.

``prepare`` makes the scene's context and the device poses a program holds,
``run`` makes one call (or the few calls that belong together) through the
``rigc`` package, ``exact`` restates the results that have a closed form in
plain 64-bit torch: contacts found by brute force, derivatives by automatic
differentiation, projections by torch's eigensolver.

Lists whose length depends on the state (candidates, constraints, Hessian
blocks) come back in arrays that the state keeps, sized for the scene, with
the call's values at the front and their number beside them.
"""
import dataclasses
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "rigid-ipc_gb300"))
from rigc import Context, Scene, meshes  # noqa: E402
from rigc import scene as S  # noqa: E402
from rigc.adjoint import DifferentiableSimulation, qdot_from_omega  # noqa: E402

GRAVITY = (0.0, -9.81, 0.0)


def listed():
    return [
        # the query calls of a small scene: world vertices, inertial energy
        # with derivatives, minimum distance and intersection check, as every
        # step of a run makes them; launches and latency
        {"name": "queries, 27 cubes", "kind": "queries", "scene": "cubes", "n": 3},
        # one Newton iteration's narrow phase of a small resting scene
        {"name": "narrow phase, 27 cubes", "kind": "narrow_phase", "scene": "cubes", "n": 3},
        # the same through host buffers (a program that keeps its poses on
        # the host), an ordinary pile of an odd size
        {"name": "host narrow phase, 131 spheres", "kind": "host_pass", "scene": "spheres", "n": 131},
        # one Newton iteration's narrow phase of the large plain scene
        {"name": "narrow phase, 1000 spheres", "kind": "narrow_phase", "scene": "spheres", "n": 1000},
        # edge-edge contacts of interlocked links
        {"name": "narrow phase, 200-link chain", "kind": "narrow_phase", "scene": "chain", "n": 200},
        # many independent scenes in one context
        {"name": "batched narrow phase, 48 piles", "kind": "narrow_phase", "scene": "hulls", "n": 48},
        # candidate lists for a program's own narrow phase
        {"name": "candidates, 417 spheres", "kind": "candidates", "scene": "spheres", "n": 417},
        # face-to-face resting contact, the constraint set and its barrier terms
        {"name": "barrier, 32 slabs", "kind": "barrier", "scene": "slabs", "n": 4},
        # lagged friction of resting contact
        {"name": "friction, 18 slabs", "kind": "friction", "scene": "slabs", "n": 3},
        # the piecewise-linear trajectory (the scene format's default), every
        # candidate's own time of impact
        {"name": "linear CCD, 150 spheres", "kind": "linear_ccd", "scene": "spheres", "n": 150},
        # whole time steps in contact
        {"name": "time steps, 27 cubes", "kind": "step", "scene": "cubes", "n": 3},
        # a differentiated rollout, forward and backward
        {"name": "adjoint, 27 cubes", "kind": "adjoint", "scene": "cubes", "n": 3},
    ]


# kind -> (scene, smallest and largest size, spread over the logarithm)
RANGES = {
    "queries": [("cubes", 2, 6, False), ("spheres", 10, 1000, True)],
    "narrow_phase": [("cubes", 2, 6, False), ("spheres", 10, 1000, True), ("chain", 8, 200, True),
                     ("hulls", 4, 48, True)],
    "host_pass": [("cubes", 2, 6, False), ("spheres", 10, 400, True)],
    "candidates": [("spheres", 10, 1000, True), ("hulls", 4, 48, True)],
    "barrier": [("slabs", 1, 4, False), ("cubes", 2, 6, False)],
    "friction": [("slabs", 1, 3, False), ("cubes", 2, 6, False)],
    "linear_ccd": [("spheres", 10, 150, True), ("cubes", 2, 4, False)],
    "step": [("cubes", 2, 4, False)],
    "adjoint": [("cubes", 3, 4, False)],
}


def draw(rng):
    kind = rng.choice(sorted(RANGES))
    scene, lo, hi, log = rng.choice(RANGES[kind])
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) if log else rng.randint(lo, hi)
    # a draw says its own seed of shapes and offsets, so that small integer
    # ranges still give different scenes
    return {"kind": kind, "scene": scene, "n": n, "variant": rng.randrange(1 << 20)}


# --------------------------------------------------------------------------
# scenes

@functools.lru_cache(maxsize=None)
def _template(name, k=0):
    if name == "cube":
        V, F = meshes.cube()
    elif name == "sphere":
        V, F = meshes.icosphere(3, 1.0)
    elif name == "torus":
        V, F = meshes.torus(1.0, 0.25, 48, 24)
    elif name == "slab":
        V, F = meshes.tessellated_box((1.0, 0.2, 1.0), (32, 4, 32))
    else:  # a convex hull of 32 points of the unit sphere
        P = np.random.default_rng(1000 + k).normal(size=(32, 3))
        V, F = meshes.convex_hull(P / np.linalg.norm(P, axis=1, keepdims=True))
    return S.make_body(V, F)


def _body(t, scale=1.0, position=(0, 0, 0), theta=None, velocity=None):
    """A copy of a template body, scaled, at a pose and velocity."""
    pose = np.concatenate([position, t.pose[3:] if theta is None else theta])
    vel = np.zeros(6) if velocity is None else np.asarray(velocity, np.float64)
    return dataclasses.replace(
        t, vertices=t.vertices * scale, pose=pose, velocity=vel, group_id=-1,
        mass=t.mass * scale ** 3, moment_of_inertia=t.moment_of_inertia * scale ** 5,
        is_dof_fixed=t.is_dof_fixed.copy(), r_max=t.r_max * scale,
        average_edge_length=t.average_edge_length * scale,
        Qdot=S.rotvec_to_matrix(pose[3:]) @ S.hat(vel[3:]))


def _plane(size):
    V, F = meshes.plane(size)
    return S.make_body(V, F, is_dof_fixed=True, body_type="static")


def _scene(bodies, dt=0.01, dhat=1e-3, mu=0.0):
    S.assign_group_ids(bodies)
    return Scene(bodies=bodies, timestep=dt, dhat=dhat, gravity=GRAVITY, friction=mu)


def _rotvec(rng):
    axis = rng.normal(size=3)
    return axis / np.linalg.norm(axis) * math.pi * rng.uniform() ** (1 / 3)


def _pile(rng, r, gap=2e-4, tries=64):
    """Centres of spheres of radii r heaped on the floor of a bin: each is
    put `gap` away from the floor or from an earlier one, at the lowest of
    `tries` free places."""
    n = len(r)
    half = 0.5 * math.sqrt(np.pi * np.sum(r ** 2) / 0.6 / max(1.0, n ** (1 / 3)))
    half = max(half, 1.01 * r.max())
    P = np.zeros((n, 3))
    for i in range(n):
        k = tries // 4 if i else tries
        C = np.empty((tries, 3))
        C[:k, 0], C[:k, 2] = rng.uniform(-half + r[i], half - r[i], (2, k))
        C[:k, 1] = r[i] + gap
        if i:
            q = rng.integers(0, i, tries - k)
            d = rng.normal(size=(tries - k, 3))
            d /= np.linalg.norm(d, axis=1, keepdims=True)
            C[k:] = P[q] + d * (r[q] + r[i] + gap)[:, None]
        bad = (np.abs(C[:, 0]) > half - r[i] + 1e-12) | (np.abs(C[:, 2]) > half - r[i] + 1e-12)
        bad |= C[:, 1] < r[i] + gap
        if i:
            D = np.linalg.norm(C[:, None] - P[None, :i], axis=2)
            bad |= (D < r[:i] + r[i] + 0.999 * gap).any(1)
        if bad.all():  # on top of everything
            C[0] = (0.0, (P[:i, 1] + r[:i]).max() + r[i] + gap, 0.0)
            bad[0] = False
        P[i] = C[np.argmin(np.where(bad, np.inf, C[:, 1]))]
    return P


def _velocities(rng, n, sigma, omega):
    return np.concatenate([rng.normal(0, sigma, (n, 3)), rng.normal(0, omega, (n, 3))], 1)


def _cubes(rng, n, speed):
    """n^3 unit cubes in resting stacks, a fraction of dhat apart, tilted by
    what a landing leaves, moving at what is left of their speed."""
    t = _template("cube")
    bodies = []
    vel = _velocities(rng, n ** 3, speed, 0.5 * speed)
    for i in range(n):
        for k in range(n):
            y = 0.0
            yaw = rng.uniform(-0.15, 0.15)
            for _ in range(n):
                tilt = rng.uniform(-1e-4, 1e-4, 2)
                theta = np.array([tilt[0], yaw + rng.uniform(-0.05, 0.05), tilt[1]])
                R = S.rotvec_to_matrix(theta)
                h = (t.vertices @ R.T)[:, 1]
                y += rng.uniform(2e-4, 7e-4) - h.min()
                x = [(i - (n - 1) / 2) * 1.45, y, (k - (n - 1) / 2) * 1.45]
                bodies.append(_body(t, 1.0, x, theta, vel[len(bodies)]))
                y += h.max()
    bodies.append(_plane(4.0 * n + 8.0))
    return _scene(bodies)


def _spheres(rng, n):
    r = rng.uniform(0.3, 0.6, n)
    P = _pile(rng, r)
    vel = _velocities(rng, n, 1.0, 2.0)
    t = _template("sphere")
    bodies = [_body(t, r[i], P[i], _rotvec(rng), vel[i]) for i in range(n)]
    bodies.append(_plane(2.5 * np.abs(P[:, [0, 2]]).max() + 4.0))
    return _scene(bodies)


def _chain(rng, n):
    """Interlocked tori, odd ones turned by 90 degrees, the first one fixed;
    neighbours in contact (within dhat = 1e-4) and moving."""
    t = _template("torus")
    vel = _velocities(rng, n, 0.3, 0.2)
    bodies = []
    for i in range(n):
        b = _body(t, 1.0, [1.49993 * i + rng.uniform(-1e-5, 1e-5), *rng.uniform(-2e-5, 2e-5, 2)],
                  S.matrix_to_rotvec(S.euler_xyz_deg_to_matrix([90.0 if i % 2 else 0.0, 0, 0])
                                     @ S.rotvec_to_matrix(t.pose[3:])), vel[i])
        if i == 0:
            b.type, b.velocity = S.BODY_STATIC, np.zeros(6)
            b.is_dof_fixed[:] = True
        bodies.append(b)
    return _scene(bodies, dt=0.005, dhat=1e-4)


def _hulls(rng, n, variant):
    """n scenes of uneven sizes, each a pile of hulls on its own plane."""
    scenes = []
    for m in _hull_counts(n, variant):
        r = rng.uniform(0.5, 2.0, m)
        P = _pile(rng, r, tries=32)
        vel = _velocities(rng, m, 1.0, 0.0)
        bodies = [_body(_template("hull", int(rng.integers(24))), r[i], P[i], _rotvec(rng), vel[i])
                  for i in range(m)]
        bodies.append(_plane(2.5 * np.abs(P[:, [0, 2]]).max() + 10.0))
        scenes.append(_scene(bodies))
    return S.concat_scenes(scenes)


def _hull_counts(n, variant):
    u = np.random.default_rng([n, variant]).uniform(math.log(8), math.log(100), n)
    return np.rint(np.exp(u)).astype(int)


def _slabs(rng, n):
    """n x n columns of two tessellated slabs resting face to face."""
    t = _template("slab")
    bodies = []
    for i in range(n):
        for k in range(n):
            y = 0.0
            for _ in range(2):
                theta = np.array([*rng.uniform(-3e-5, 3e-5, 1), rng.uniform(-0.06, 0.06),
                                  *rng.uniform(-3e-5, 3e-5, 1)])
                R = S.rotvec_to_matrix(theta) @ S.rotvec_to_matrix(t.pose[3:])
                h = (t.vertices @ R.T)[:, 1]
                y += 3e-4 - h.min()
                off = rng.uniform(-0.02, 0.02, 2)
                bodies.append(_body(t, 1.0, [(i - (n - 1) / 2) * 1.25 + off[0], y,
                                             (k - (n - 1) / 2) * 1.25 + off[1]],
                                    S.matrix_to_rotvec(R), _velocities(rng, 1, 0.02, 0.0)[0]))
                y += h.max()
    bodies.append(_plane(1.25 * n + 2.0))
    return _scene(bodies, mu=0.5)


def _make(case, seed):
    rng = np.random.default_rng([int(seed), case["n"], int(case.get("variant", 0))])
    sob = None
    if case["scene"] == "hulls":
        sc, sob = _hulls(rng, case["n"], int(case.get("variant", 0)))
    elif case["scene"] == "cubes":
        sc = _cubes(rng, case["n"], 0.01 if case["kind"] == "adjoint" else 0.1)
    else:
        sc = {"spheres": _spheres, "chain": _chain, "slabs": _slabs}[case["scene"]](rng, case["n"])
    return sc, sob, rng


# --------------------------------------------------------------------------
# the calls

# per body: continuous candidates, discrete ones, constraints, Hessian blocks
ROOM = {"cubes": (400, 400, 300, 60), "spheres": (1600, 500, 60, 60), "chain": (1200, 600, 100, 20),
        "hulls": (200, 100, 60, 40), "slabs": (0, 0, 16000, 20)}


def _room(case, nb):
    """Arrays for the outputs whose length depends on the state."""
    cont, disc, cons, blocks = (k * nb + 4096 for k in ROOM[case["scene"]])
    kind, full = case["kind"], lambda shape, dtype: np.full(shape, -1, dtype)
    out = {}
    if kind == "candidates":
        out = {k: full((m, 2), np.int32) for k, m in (("ee", cont), ("fv", cont), ("ee_discrete", disc),
                                                      ("fv_discrete", disc))}
    if kind == "linear_ccd":
        out = {"per_candidate": full(cont, np.float64)}
    if kind in ("narrow_phase", "barrier", "friction"):
        out = {"type": full(cons, np.int32), "verts": full((cons, 4), np.int32),
               "weight": full(cons, np.float64)}
    if kind in ("narrow_phase", "barrier", "friction", "host_pass"):
        out.update(col=full(blocks, np.int32), val=np.zeros((blocks, 6, 6)))
    return out


def _put(room, name, a):
    room[name][:len(a)] = a
    return room[name]


def prepare(case, seed):
    sc, sob, rng = _make(case, seed)
    x0 = sc.poses()
    st = {"kind": case["kind"], "scene": sc, "x0": x0, "room": _room(case, sc.num_bodies)}
    if case["kind"] == "adjoint":
        nb = sc.num_bodies
        dev = dict(dtype=torch.float64, device="cuda")
        st["sim"] = DifferentiableSimulation(sc, sc.timestep, GRAVITY, sc.dhat,
                                             max_newton_iterations=200)
        st["poses"] = torch.as_tensor(x0.reshape(nb, 6), **dev)
        st["velocities"] = torch.as_tensor(sc.velocities().reshape(nb, 6), **dev)
        return st
    ctx = Context(sc, scene_of_body=sob)
    st["ctx"] = ctx
    st["x1"] = sc.predictor_poses(x0)
    st["x0d"], st["x1d"] = ctx.device(x0), ctx.device(st["x1"])
    if case["kind"] == "queries":
        st["bodies"] = ctx.body_state()
    if case["kind"] == "friction":
        # poses during the step: a slide of up to a few times the static bound
        d = np.zeros((sc.num_bodies, 6))
        dyn = np.array([b.type == S.BODY_DYNAMIC for b in sc.bodies])
        d[dyn, 0], d[dyn, 2] = rng.normal(0, 2e-5, (2, dyn.sum()))
        d[dyn, 4] = rng.normal(0, 2e-5, dyn.sum())
        st["x"] = x0 + d.reshape(-1)
        st["xd"] = ctx.device(st["x"])
    return st


FRICTION_MU, FRICTION_KAPPA, FRICTION_EPSVH = 0.5, 1e6, 1e-5


def run(st):
    kind, sc, room = st["kind"], st["scene"], st["room"]
    if kind == "adjoint":
        sim = st["sim"]
        p = st["poses"].detach().requires_grad_()
        v = st["velocities"].detach().requires_grad_()
        P, V, Q = sim(p, v, qdot_from_omega(p, v[:, 3:]), 2)
        # each body's distance to a point, as a trajectory loss weighs it
        loss = ((P[:, :3] - torch.tensor([3.0, 0.0, 0.5], dtype=P.dtype, device=P.device)) ** 2).sum()
        gp, gv = torch.autograd.grad(loss, (p, v))
        return {"loss": loss.detach(), "poses": P.detach(), "d_poses": gp, "d_velocities": gv}
    ctx = st["ctx"]
    if kind == "queries":
        e, g, H = ctx.body_energy(st["x1d"], st["bodies"])
        return {"vertices": ctx.world_vertices(st["x0d"]), "energy": e, "grad": g, "hess": H,
                "min_distance": ctx.compute_min_distance(st["x0d"], sc.dhat),
                "intersections": ctx.detect_intersections(st["x0d"])}
    if kind == "candidates":
        ee, fv = ctx.detect_collision_candidates_rigid(st["x0d"], st["x1d"], True, 0.0)
        ee_d, fv_d = ctx.detect_collision_candidates_rigid(st["x0d"], None, False, sc.dhat / 2)
        lists = {"ee": ee, "fv": fv, "ee_discrete": ee_d, "fv_discrete": fv_d}
        return {"counts": [len(a) for a in lists.values()], **{k: _put(room, k, a) for k, a in lists.items()}}
    if kind == "linear_ccd":
        ctx.count_collision_candidates_rigid(st["x0d"], st["x1d"], True, 0.0)
        toi, per, _ = ctx.earliest_toi_piecewise_linear(st["x0d"], st["x1d"], per_candidate=True)
        return {"toi": toi, "count": len(per), "per_candidate": _put(room, "per_candidate", per)}
    if kind == "host_pass":
        toi, e, g, (rp, col, val), _ = ctx.narrow_phase_host(st["x0"], st["x1"], sc.dhat)
        return {"toi": toi, "energy": e, "grad": g, "row_ptr": rp, "col": _put(room, "col", col),
                "val": _put(room, "val", val)}
    if kind == "step":
        ctx.sim_init(sc.timestep, GRAVITY, sc.dhat, poses=st["x0"])
        ctx.sim_step(2)
        P, V, Q, kappa = ctx.sim_state()
        return {"poses": P, "velocities": V, "Qdot": Q, "stiffness": kappa}
    out = {}
    if kind == "narrow_phase":
        out["toi"] = ctx.compute_earliest_toi(st["x0d"], st["x1d"])
        if ctx.num_scenes > 1:
            out["scene_tois"] = ctx.scene_tois()
    cs = ctx.construct_constraint_set(st["x0d"], sc.dhat)
    out["counts"] = list(cs["counts"])
    out["constraints"] = {k: _put(room, k, cs[k]) for k in ("type", "verts", "weight")}
    if kind == "friction":
        ctx.friction_setup(st["x0d"], sc.dhat, FRICTION_KAPPA, FRICTION_MU)
        e, g, H = ctx.compute_friction_term(st["xd"], FRICTION_EPSVH)
    else:
        e, g, H = ctx.compute_barrier_term(st["x0d"], sc.dhat)
    out.update({"energy": e, "grad": g, "row_ptr": H[0], "col": _put(room, "col", H[1]),
                "val": _put(room, "val", H[2])})
    return out


def work(case):
    """Bytes: rest vertices, connectivity and poses read once, and the
    outputs that grow with the scene written once; operations: per candidate,
    contact or solve, a plain evaluation of the path's formulas, with the
    candidates and contacts per body that these scenes have."""
    per_cubes, per_scene = case["n"] ** 3, case["n"]
    nb, nv, ne, nf = {
        "cubes": (per_cubes, 8, 18, 12), "spheres": (per_scene, 642, 1920, 1280),
        "chain": (per_scene, 1152, 3456, 2304), "hulls": (36 * per_scene, 32, 90, 60),
        "slabs": (2 * per_scene ** 2, 2562, 7680, 5120)}[case["scene"]]
    candidates = nb * {"cubes": 30, "spheres": 600, "chain": 160, "hulls": 250, "slabs": 30000}[case["scene"]]
    contacts = nb * {"cubes": 12, "spheres": 2, "chain": 1, "hulls": 2, "slabs": 5000}[case["scene"]]
    mesh = nb * (24 * nv + 8 * ne + 24 * nf + 96)
    ccd = {"bytes": mesh + 8 * candidates, "flops": 3000.0 * candidates}
    terms = {"bytes": mesh + 1456 * contacts, "flops": 20000.0 * contacts}
    kind = case["kind"]
    if kind == "queries":
        return {"bytes": nb * (48 * nv + 8 * ne + 24 * nf + 600), "flops": nb * (60.0 * nv + 2000.0)}
    if kind == "candidates":
        return {"bytes": 2 * mesh + 12 * candidates, "flops": nb * 100.0 * nv}
    if kind in ("barrier", "friction"):
        return terms
    if kind == "linear_ccd":
        return {"bytes": ccd["bytes"] + 8 * candidates, "flops": 20000.0 * candidates}
    both = {k: ccd[k] + terms[k] for k in ccd}
    if kind == "step":  # some ten Newton iterations and their dense solves
        return {"bytes": 10 * both["bytes"], "flops": 10 * (both["flops"] + (6 * nb) ** 3 / 3.0)}
    if kind == "adjoint":  # two steps, and the same again backwards
        return {"bytes": 40 * both["bytes"], "flops": 40 * (both["flops"] + (6 * nb) ** 3 / 3.0)}
    return both


# --------------------------------------------------------------------------
# plain 64-bit restatement

def _rotation(th):
    """R(theta) = I + sinc|t| [t] + sinc(|t|/2)^2 / 2 [t]^2, smooth in theta."""
    s = (th * th).sum()
    small = s < 1e-2
    q = torch.sqrt(torch.where(small, torch.ones_like(s), s))
    a_s, b_s = torch.zeros_like(s), torch.zeros_like(s)
    for k in range(8, -1, -1):
        a_s = a_s * s + (-1) ** k / math.factorial(2 * k + 1)
        b_s = b_s * s + (-1) ** k / math.factorial(2 * k + 2)
    a = torch.where(small, a_s, torch.sin(q) / q)
    b = torch.where(small, b_s, 2 * (torch.sin(q / 2) / q) ** 2)
    z = torch.zeros_like(s)
    K = torch.stack([z, -th[2], th[1], th[2], z, -th[0], -th[1], th[0], z]).reshape(3, 3)
    return torch.eye(3, dtype=th.dtype, device=th.device) + a * K + b * (K @ K)


def _world(x, body, rest):
    R = torch.func.vmap(_rotation)(x[:, 3:])
    return (R[body] @ rest[:, :, None])[:, :, 0] + x[body, :3]


def _overlaps(lo_a, hi_a, lo_b, hi_b, chunk=4096):
    out = []
    for s in range(0, len(lo_a), chunk):
        m = ((lo_a[s:s + chunk, None] <= hi_b[None]) & (lo_b[None] <= hi_a[s:s + chunk, None])).all(2)
        i, j = m.nonzero(as_tuple=True)
        out.append(torch.stack([i + s, j], 1))
    return torch.cat(out)


def _close_pairs(sc, V, sob, dhat):
    """(edge, edge) and (face, vertex) pairs of different bodies whose boxes
    come within dhat, by brute force over bodies whose boxes do."""
    dev = V.device
    E = torch.as_tensor(sc.edges, dtype=torch.long, device=dev)
    F = torch.as_tensor(sc.faces, dtype=torch.long, device=dev)
    box = {}
    for key, ids in (("v", torch.arange(len(V), device=dev)[:, None]), ("e", E), ("f", F)):
        P = V[ids]
        box[key] = (P.amin(1) - dhat, P.amax(1) + dhat)
    starts = {"v": sc.body_vertex_start, "e": sc.body_edge_start, "f": sc.body_face_start}
    nb = sc.num_bodies
    vs = sc.body_vertex_start
    Vh = V.cpu().numpy()
    lo = np.stack([Vh[vs[b]:vs[b + 1]].min(0) for b in range(nb)]) - dhat
    hi = np.stack([Vh[vs[b]:vs[b + 1]].max(0) for b in range(nb)]) + dhat
    near = np.triu(((lo[:, None] <= hi[None]) & (lo[None] <= hi[:, None])).all(2), 1)
    if sob is not None:
        near &= sob[:, None] == sob[None]
    near &= sc.group_ids[:, None] != sc.group_ids[None]
    ee, fv = [], []

    def part(key, b, blo, bhi):
        a, z = int(starts[key][b]), int(starts[key][b + 1])
        l, h = box[key][0][a:z], box[key][1][a:z]
        k = ((l <= bhi) & (blo <= h)).all(1).nonzero()[:, 0]
        return k + a, l[k], h[k]

    for a, b in np.argwhere(near):
        blo = torch.as_tensor(np.maximum(lo[a], lo[b]) - dhat, device=dev)
        bhi = torch.as_tensor(np.minimum(hi[a], hi[b]) + dhat, device=dev)
        P = {(k, i): part(k, i, blo, bhi) for k in "vef" for i in (a, b)}
        for ka, ia, kb, ib, out in (("e", a, "e", b, ee), ("f", a, "v", b, fv), ("f", b, "v", a, fv)):
            p, q = P[ka, ia], P[kb, ib]
            if len(p[0]) and len(q[0]):
                m = _overlaps(p[1], p[2], q[1], q[2])
                out.append(torch.stack([p[0][m[:, 0]], q[0][m[:, 1]]], 1))
    none = torch.zeros((0, 2), dtype=torch.long, device=dev)
    return E, F, torch.cat(ee + [none]), torch.cat(fv + [none])


def _d_pp(p, q):
    return ((p - q) ** 2).sum(-1)


def _d_pl(p, a, b):
    c = torch.linalg.cross(a - p, b - p)
    return (c * c).sum(-1) / ((b - a) ** 2).sum(-1)


def _d_ll(a0, a1, b0, b1):
    n = torch.linalg.cross(a1 - a0, b1 - b0)
    return ((b0 - a0) * n).sum(-1) ** 2 / (n * n).sum(-1)


def _inside(p, a, b):
    t = ((p - a) * (b - a)).sum(-1) / ((b - a) ** 2).sum(-1)
    return (t > 0) & (t < 1)


# closest features of the pair's four vertices (0-3): a point and a point, a
# point and an edge's line, or both primitives whole
PP_EE, PL_EE = [(0, 2), (0, 3), (1, 2), (1, 3)], [(2, 0, 1), (3, 0, 1), (0, 2, 3), (1, 2, 3)]
PP_FV, PL_FV = [(0, 1), (0, 2), (0, 3)], [(0, 1, 2), (0, 2, 3), (0, 3, 1)]


def _features(X, pp, pl, whole, feasible):
    d = [_d_pp(X[:, i], X[:, j]) for i, j in pp]
    for i, j, k in pl:
        d.append(torch.where(_inside(X[:, i], X[:, j], X[:, k]), _d_pl(X[:, i], X[:, j], X[:, k]), math.inf))
    d.append(torch.where(feasible, whole, math.inf))
    v, f = torch.stack(d).min(0)
    return v, f


def _contacts(sc, V, sob, dhat):
    """Groups of active contacts: (kind, feature, vertex ids n x 4): the
    closest features of every edge-edge and face-vertex pair within dhat;
    nearly parallel edges are the kind "mollified"."""
    E, F, ee, fv = _close_pairs(sc, V, sob, dhat)
    groups = []
    ids = torch.cat([E[ee[:, 0]], E[ee[:, 1]]], 1)
    X = V[ids]
    a, b, w = X[:, 1] - X[:, 0], X[:, 3] - X[:, 2], X[:, 0] - X[:, 2]
    aa, ab, bb, aw, bw = (a * a).sum(1), (a * b).sum(1), (b * b).sum(1), (a * w).sum(1), (b * w).sum(1)
    det = aa * bb - ab * ab
    s, t = (ab * bw - bb * aw) / det, (aa * bw - ab * aw) / det
    d, f = _features(X, PP_EE, PL_EE, _d_ll(X[:, 0], X[:, 1], X[:, 2], X[:, 3]),
                     (s > 0) & (s < 1) & (t > 0) & (t < 1))
    n = torch.linalg.cross(a, b)
    eps = 1e-3 * aa * bb
    moll = (n * n).sum(1) < eps
    act = d < dhat * dhat
    for k in range(9):
        m = act & (f == k)
        groups.append(("mollified", k, ids[m & moll], eps[m & moll]))
        groups.append(("ee", k, ids[m & ~moll], None))
    ids = torch.cat([fv[:, 1:], F[fv[:, 0]]], 1)
    X = V[ids]
    p, q, r = X[:, 0] - X[:, 1], X[:, 2] - X[:, 1], X[:, 3] - X[:, 1]
    n = torch.linalg.cross(q, r)
    nn = (n * n).sum(1)
    u = (torch.linalg.cross(p, r) * n).sum(1) / nn
    v = (torch.linalg.cross(q, p) * n).sum(1) / nn
    d, f = _features(X, PP_FV, PL_FV, (p * n).sum(1) ** 2 / nn, (u > 0) & (v > 0) & (u + v < 1))
    act = d < dhat * dhat
    for k in range(7):
        groups.append(("fv", k, ids[act & (f == k)], None))
    return [g for g in groups if len(g[2])]


def _distance(X, kind, k):
    pp, pl = (PP_FV, PL_FV) if kind == "fv" else (PP_EE, PL_EE)
    if k < len(pp):
        return _d_pp(X[pp[k][0]], X[pp[k][1]])
    if k < len(pp) + len(pl):
        i, j, l = pl[k - len(pp)]
        return _d_pl(X[i], X[j], X[l])
    if kind == "fv":
        n = torch.linalg.cross(X[2] - X[1], X[3] - X[1])
        return ((X[0] - X[1]) * n).sum() ** 2 / (n * n).sum()
    return _d_ll(X[0], X[1], X[2], X[3])


def _positions(q, rest, side):
    """The four vertices from the two bodies' poses q (12)."""
    R = torch.stack([_rotation(q[3:6]), _rotation(q[9:12])])
    p = torch.stack([q[:3], q[6:9]])
    return (R[side] @ rest[:, :, None])[:, :, 0] + p[side]


def _barrier(d, dhat):
    s = dhat * dhat
    return -(d - s) ** 2 * torch.log(d / s)


def _slide(kind, k, X):
    """Weights of the closest points (4) and tangent plane's normal (3)."""
    one = torch.ones(())
    g = torch.zeros(4, dtype=X.dtype, device=X.device)
    pp, pl = (PP_FV, PL_FV) if kind == "fv" else (PP_EE, PL_EE)
    if kind != "mollified" and k < len(pp):
        i, j = pp[k]
        hot = lambda m: torch.nn.functional.one_hot(torch.tensor(m, device=X.device), 4)  # noqa: E731
        return g + hot(i) - hot(j), X[i] - X[j]
    if kind != "mollified" and k < len(pp) + len(pl):
        i, j, l = pl[k - len(pp)]
        e, w = X[l] - X[j], X[i] - X[j]
        t = (e * w).sum() / (e * e).sum()
        val = {i: one.to(X), j: t - 1, l: -t}
        return torch.stack([val.get(m, g[0]) for m in range(4)]), w - t * e
    if kind == "fv":
        q, r, w = X[2] - X[1], X[3] - X[1], X[0] - X[1]
        n = torch.linalg.cross(q, r)
        u = (torch.linalg.cross(w, r) * n).sum() / (n * n).sum()
        v = (torch.linalg.cross(q, w) * n).sum() / (n * n).sum()
        return torch.stack([one.to(X), u + v - 1, -u, -v]), n
    a, b, w = X[1] - X[0], X[3] - X[2], X[2] - X[0]
    n = torch.linalg.cross(a, b)
    al = (torch.linalg.cross(w, b) * n).sum() / (n * n).sum()
    be = (torch.linalg.cross(w, a) * n).sum() / (n * n).sum()
    return torch.stack([1 - al, al, be - 1, -be]), n


def _terms(sc, sob, x, dhat, x_fric=None):
    """Energy, gradient and block-sparse projected Hessian of the barrier at
    x, or of the friction lagged at x (evaluated at x_fric)."""
    dev = torch.device("cuda")
    nb = sc.num_bodies
    xt = torch.as_tensor(np.asarray(x).reshape(nb, 6), device=dev)
    rest = torch.as_tensor(sc.rest_vertices, device=dev)
    body = torch.as_tensor(np.repeat(np.arange(nb), np.diff(sc.body_vertex_start)), device=dev)
    V0 = _world(xt, body, rest)
    xe = xt if x_fric is None else torch.as_tensor(np.asarray(x_fric).reshape(nb, 6), device=dev)
    grad = torch.zeros((nb, 6), dtype=torch.float64, device=dev)
    energy = torch.zeros((), dtype=torch.float64, device=dev)
    keys, blocks = [], []
    for kind, k, ids, eps in _contacts(sc, V0, sob, dhat):
        # the pair's bodies: of the vertex and of the face, or of the edges
        pair = body[ids[:, [0, 1 if kind == "fv" else 2]]]
        side = torch.tensor([0, 1, 1, 1] if kind == "fv" else [0, 0, 1, 1], device=dev)

        def f(q, v, e, x0):
            X = _positions(q, v, side)
            if x_fric is not None:
                d = _distance(x0, kind, k)
                s = dhat * dhat
                lam = -FRICTION_KAPPA * (s - d) * (2 * torch.log(d / s) - s / d + 1) * 2 * torch.sqrt(d)
                g, n = _slide(kind, k, x0)
                u = g @ (X - x0)
                u = u - (u @ n) / (n @ n) * n
                y2 = (u * u).sum()
                y = torch.sqrt(torch.clamp(y2, min=1e-60))
                h = FRICTION_EPSVH
                f0 = torch.where(y >= h, y, -y ** 3 / (3 * h * h) + y2 / h + h / 3)
                return FRICTION_MU * lam * f0
            b = _barrier(_distance(X, kind, k), dhat)
            if kind == "mollified":
                n = torch.linalg.cross(X[1] - X[0], X[3] - X[2])
                r = (n * n).sum() / e
                b = b * (2 - r) * r
            return b

        for s in range(0, len(ids), 16384):
            i, pr = ids[s:s + 16384], pair[s:s + 16384]
            q = xe[pr].reshape(-1, 12)
            e = eps[s:s + 16384] if eps is not None else torch.ones(len(i), dtype=torch.float64, device=dev)
            args = (q, rest[i], e, V0[i])
            energy = energy + torch.func.vmap(f)(*args).sum()
            g = torch.func.vmap(torch.func.grad(f))(*args)
            H = torch.func.vmap(torch.func.jacfwd(torch.func.grad(f)))(*args)
            w, Q = torch.linalg.eigh(0.5 * (H + H.mT))
            H = Q @ (w.clamp(min=0)[:, :, None] * Q.mT)
            grad.index_add_(0, pr.reshape(-1), g.reshape(-1, 6))
            keys.append((pr[:, :, None] * nb + pr[:, None, :]).reshape(-1))
            blocks.append(H.reshape(-1, 2, 6, 2, 6).transpose(2, 3).reshape(-1, 6, 6))
    if not keys:
        return 0.0, grad.reshape(-1).cpu().numpy(), np.zeros(nb + 1, np.int32), np.zeros(0, np.int32), np.zeros((0, 6, 6))
    key, at = torch.unique(torch.cat(keys), return_inverse=True)
    val = torch.zeros((len(key), 6, 6), dtype=torch.float64, device=dev)
    val.index_add_(0, at, torch.cat(blocks))
    rows = torch.bincount(key // nb, minlength=nb).cumsum(0).cpu().numpy()
    return (float(energy), grad.reshape(-1).cpu().numpy(),
            np.concatenate([[0], rows]).astype(np.int32),
            (key % nb).cpu().numpy().astype(np.int32), val.cpu().numpy())


def _body_energy(sc, x):
    """Inertial energy of every body, its gradient and Hessian."""
    dev = torch.device("cuda")
    nb, h = sc.num_bodies, sc.timestep
    t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
    x0, v0 = t(sc.poses()).reshape(nb, 6), t(sc.velocities()).reshape(nb, 6)
    Qd = t(np.stack([b.Qdot for b in sc.bodies]))
    I = t(sc.moment)
    J = 0.5 * I.sum(1, keepdim=True) - I
    grav = torch.tensor(GRAVITY, dtype=torch.float64, device=dev)

    def f(q, x0, v0, Qd, m, J):
        hat = x0[:3] + h * (v0[:3] + h * grav)
        T = _rotation(x0[3:]) + h * Qd
        Q = _rotation(q[3:])
        return 0.5 * m * (q[:3] @ q[:3]) - m * (q[:3] @ hat) + (J * (0.5 * Q * Q - Q * T)).sum()

    args = (t(x).reshape(nb, 6), x0, v0, Qd, t(sc.mass), J)
    on = t([float(b.type == S.BODY_DYNAMIC) for b in sc.bodies])
    e = (torch.func.vmap(f)(*args) * on).sum()
    g = torch.func.vmap(torch.func.grad(f))(*args) * on[:, None]
    H = torch.func.vmap(torch.func.jacfwd(torch.func.grad(f)))(*args) * on[:, None, None]
    return float(e), g.reshape(-1).cpu().numpy(), H.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("candidates", "linear_ccd", "step", "adjoint"):
        return None  # whole numbers, conservative bounds, iterated solves
    sc, sob, _ = _make(case, seed)
    if kind == "queries":
        st = prepare(case, seed)
        body = torch.as_tensor(np.repeat(np.arange(sc.num_bodies), np.diff(sc.body_vertex_start)), device="cuda")
        V = _world(torch.as_tensor(st["x0"].reshape(-1, 6), device="cuda"), body,
                   torch.as_tensor(sc.rest_vertices, device="cuda"))
        e, g, H = _body_energy(sc, st["x1"])
        return {"vertices": V, "energy": e, "grad": g, "hess": H, "min_distance": None,
                "intersections": None}
    x_fric = prepare(case, seed)["x"] if kind == "friction" else None
    e, g, rp, col, val = _terms(sc, sob, sc.poses(), sc.dhat, x_fric)
    out = {"toi": None} if kind in ("narrow_phase", "host_pass") else {}
    if kind == "narrow_phase" and sob is not None:
        out["scene_tois"] = None
    if kind != "host_pass":
        out["counts"] = out["constraints"] = None
    room = _room(case, sc.num_bodies)
    out.update({"energy": e, "grad": g, "row_ptr": rp, "col": _put(room, "col", col),
                "val": _put(room, "val", val)})
    return out
