"""The work that programs built on this framework have it do, as cases to be timed and compared.

A case is one simulation substep (``CollisionPipeline.collide`` + ``SolverVBD.step``), one batched
call, one inference of the warm-start network or one of its training steps, through the public
entry points and with the library's default launch shape.  The scenes are those of
``newton_b200.scenes``; the states put the cloth where a running simulation has it (resting on
its colliders, falling, folded over itself), with the seed deciding the wrinkles, the velocities
and the external forces.  Every pass starts from the state that ``prepare`` made, as a program
does that steps from given states (resets, rollouts from recorded states).

``exact`` restates the substep in 64-bit torch: the stable Neo-Hookean membrane, dihedral bending,
particle-shape contact, cloth self-contact, the residual gate and the learned start.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from newton_b200 import CollisionPipeline, scenes
from newton_b200.learned import IN, N_PARAMS, OFF_B1, OFF_B2, OFF_B3, OFF_W1, OFF_W2, OFF_W3, WarmStartMLP
from newton_b200.solvers import SolverVBD

DT = 1.0 / 600.0
MARGIN = 5.0e-3
GATE_CAP = 40
SELF_RADIUS, SELF_MARGIN = 2.0e-3, 3.0e-3
SELF_SPACING = 4.0 / 1023.0  # vertex spacing of the self-contact cloth (4 m at 1024 vertices)
DEVICE = "cuda:0"


def listed():
    return [
        # the smallest simulation: one 32 x 32 cloth hanging from two corners; launches and host work
        {"name": "hanging_32", "kind": "hanging", "n": 32, "iterations": 10},
        # eight small garments of uneven size, each with its own solver, stepped by one call
        {"name": "batch_8_small", "kind": "batch", "count": 8, "n": 20, "n_max": 48, "iterations": 10},
        # the ordinary simulation: a 256 x 256 cloth on a sphere, the fixed iteration count
        {"name": "drape_256", "kind": "drape", "n": 256, "iterations": 10},
        # the same at an odd size, iterated until the force residual has fallen (device-side loop)
        {"name": "drape_gate_181", "kind": "drape", "n": 181, "gate": 0.9},
        # a pinned, damped curtain (membrane and bending damping) in wind (external forces)
        {"name": "curtain_150", "kind": "curtain", "n": 150, "iterations": 10},
        # the largest batch: 512 uneven worlds (1.9 M vertices) in one model, for learning
        {"name": "worlds_512", "kind": "worlds", "worlds": 512, "iterations": 10},
        # a smaller batch, to the residual gate
        {"name": "worlds_gate_96", "kind": "worlds", "worlds": 96, "gate": 0.1},
        # cloth folded over itself, small: detection, contact forces and truncation per color
        {"name": "self_contact_64", "kind": "self", "n": 64, "iterations": 10},
        # the largest single cloth (1.05 M vertices) with self-contact
        {"name": "self_contact_1024", "kind": "self", "n": 1024, "iterations": 10},
        # the learned warm start as the step mode
        {"name": "learned_drape_256", "kind": "learned", "n": 256, "iterations": 4},
        # inference of the warm-start network on the feature rows of a 1 M vertex model
        {"name": "mlp_forward_1m", "kind": "mlp_forward", "rows": 1048576},
        # one training step of the warm-start network at the default mini-batch
        {"name": "mlp_train_32768", "kind": "mlp_train", "rows": 32768},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["hanging", "batch", "drape", "drape", "curtain", "worlds", "worlds", "self", "learned",
                       "mlp_forward", "mlp_train"])
    if kind == "hanging":
        return {"kind": kind, "n": log_int(8, 96), "iterations": rng.randint(4, 20)}
    if kind == "batch":
        n = rng.randint(8, 32)
        return {"kind": kind, "count": rng.randint(2, 16), "n": n, "n_max": n + rng.randint(1, 32), "iterations": 10}
    if kind in ("drape", "worlds"):
        c = {"kind": kind, "n": log_int(48, 512)} if kind == "drape" else {"kind": kind, "worlds": log_int(4, 500)}
        if rng.random() < 0.4:
            c["gate"] = round(rng.uniform(0.85, 0.95) if kind == "drape" else rng.uniform(0.08, 0.2), 3)
        else:
            c["iterations"] = rng.choice([5, 10, 10, 15] if kind == "drape" else [5, 10])
        return c
    if kind == "curtain":
        return {"kind": kind, "n": log_int(24, 400), "iterations": rng.choice([5, 10, 15])}
    if kind == "self":
        return {"kind": kind, "n": log_int(40, 800), "iterations": rng.choice([5, 10])}
    if kind == "learned":
        return {"kind": kind, "n": log_int(40, 512), "iterations": rng.randint(3, 6)}
    return {"kind": kind, "rows": log_int(128, 1000000) if kind == "mlp_forward" else log_int(1000, 131072)}


# ------------------------------------------------------------------------------------------------
# scenes (built once per program, as a simulation builds its own) and states (from the seed)
# ------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _scene(kind: str, n: int, worlds: int = 0):
    if kind == "hanging":
        return scenes.single_cloth(n=n, side=n / 32.0, pin_top_corners=True, ground=-1.0, height=0.05, vertical=True,
                                   z_noise=0.0, device=DEVICE)
    if kind in ("drape", "learned"):
        return scenes.draped_cloth(n=n, height=0.904, device=DEVICE)
    if kind == "curtain":
        material = dict(tri_ke=5.0e3, tri_ka=5.0e3, tri_kd=1.0e-2, edge_ke=5.0e-2, edge_kd=1.0e-3)
        return scenes.single_cloth(n=n, side=1.5, pin_top_corners=True, ground=None, height=1.6, vertical=True,
                                   material=material, z_noise=0.0, device=DEVICE)
    if kind == "worlds":
        return scenes.batched_worlds(worlds, seed=worlds, device=DEVICE)
    return scenes.cloth_on_boxes(n=n, side=SELF_SPACING * (n - 1), device=DEVICE)


def _models(case):
    if case["kind"] == "batch":
        k = case["count"]
        sizes = [case["n"] + (case["n_max"] - case["n"]) * j // max(k - 1, 1) for j in range(k)]
        by_size = {s: scenes.draped_cloth(n=s, height=0.904, device=DEVICE) for s in set(sizes)}
        return [by_size[s] for s in sizes]
    return [_scene(case["kind"], case.get("n", 0), case.get("worlds", 0))]


def _waves(u, v, size, rng, count=6, phase=0.0):
    """Smooth wrinkles of unit size: plane waves of random direction, a tenth to a half of the cloth long."""
    out = np.zeros_like(u)
    for _ in range(count):
        a, lam, p = rng.uniform(0, 2 * np.pi), size * rng.uniform(0.1, 0.5), rng.uniform(0, 2 * np.pi)
        out += np.sin(2 * np.pi / lam * (u * np.cos(a) + v * np.sin(a)) + p + phase)
    return out / count


def _state(kind, model, q0, seed):
    """Positions, velocities and external forces (float32 numpy) of a running simulation."""
    rng = np.random.default_rng([seed, model.particle_count])
    q = q0.astype(np.float64).copy()
    qd = np.zeros_like(q)
    f = np.zeros_like(q)
    x, y, z = q[:, 0].copy(), q[:, 1].copy(), q[:, 2].copy()
    if kind in ("hanging", "curtain"):
        size = float(np.ptp(x))
        sway = (z.max() - z) / size
        q[:, 1] += 5e-3 * size * _waves(x, z, size, rng) * sway
        qd[:, 1] = 0.4 * _waves(x, z, size, rng) * sway
        qd[:, 2] = -0.1 * sway
        if kind == "curtain":  # wind, of the order of the weight
            f[:, 1] = 9.81 * model.particle_mass * (0.5 + 0.5 * _waves(x, z, size, rng))
    elif kind in ("drape", "learned", "batch"):
        # resting on the sphere (centre z 0.5, radius 0.4) with a small penetration, then a cone
        # whose rim is still falling
        r, top = 0.4 + 5e-3 - 8e-4, 0.25
        s = np.hypot(x, y)
        cap = r * top
        rho = np.where(s < cap, r * np.sin(s / r), r * np.sin(top) + (s - cap) * np.cos(top))
        h = np.where(s < cap, r * np.cos(s / r), r * np.cos(top) - (s - cap) * np.sin(top))
        k = rho / np.maximum(s, 1e-12)
        free = np.clip((s - cap) / 0.3, 0.0, 1.0)
        q[:, 0], q[:, 1] = x * k, y * k
        q[:, 2] = 0.5 + h + 4e-3 * _waves(x, y, 2.0, rng) * free
        qd[:, 2] = -1.0 * np.maximum(s - cap, 0.0) + 0.1 * _waves(x, y, 2.0, rng)
    elif kind == "worlds":
        # every cloth landing on its ground plane
        phase = rng.uniform(0, 2 * np.pi, int(model.particle_world.max()) + 1)[model.particle_world]
        q[:, 2] = 6e-3 + 4e-3 * _waves(x, y, 1.0, rng, phase=phase)
        qd[:, 2] = -0.3 + 0.2 * _waves(x, y, 1.0, rng, phase=phase)
    else:
        # the cloth just landed on the tallest box, its last third folded back over itself 2 to
        # 3.5 mm above: part of the layers inside the contact radius, all near the margin
        size = float(np.ptp(x))
        gap, crease = 2.7e-3, float(x.max()) - size / 3.0
        base = float((model.shape_transform[:, 2] + model.shape_scale[:, 2])[1:].max()) + 1e-3 - 3e-4
        t = np.maximum(x - crease, 0.0)
        bend = 0.5 * np.pi * gap
        a = np.minimum(t, bend) / (0.5 * gap)
        back = np.maximum(t - bend, 0.0)
        q[:, 0] = np.minimum(x, crease) + 0.5 * gap * np.sin(a) - back
        q[:, 2] = base + 0.5 * gap * (1.0 - np.cos(a))
        q[:, 2] += np.clip(back / (8 * gap), 0.0, 1.0) * 8e-4 * _waves(x, y, 0.25, rng)
        q[:, 2] += 2e-4 * _waves(q[:, 0], y, 0.25, rng)
        qd[:, 2] = -0.2 + 0.1 * _waves(x, y, 0.25, rng) - 0.2 * np.clip(back / (8 * gap), 0.0, 1.0)
        qd[:, 0] = 0.05 * _waves(x, y, 0.25, rng)
    moving = ((model.particle_flags & 1) != 0)[:, None]
    return q.astype(np.float32), np.where(moving, qd, 0.0).astype(np.float32), np.where(moving, f, 0.0).astype(np.float32)


def _tensor(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)


def _gate(case):
    return {"tolerance": case["gate"], "max_iterations": GATE_CAP, "check_every": 1, "relative": True, "norm": "mean",
            "residual": "sweep"}


def _network(seed):
    """A warm-start network whose predictions are a few hundredths of an edge, as trained ones' are."""
    mlp = WarmStartMLP(DEVICE, seed=seed)
    mlp.params[OFF_W3:OFF_B3] *= 0.2
    mean, inv = torch.zeros(IN), torch.ones(IN)
    mean[54:58] = torch.tensor([4.0, 4.0, -2.0, -5.0])
    inv[0:6], inv[30:54] = 4.0, 4.0
    mlp.mean.copy_(mean)
    mlp.inv_std.copy_(inv)
    mlp.pack()
    return mlp


def _correction(model, seed):
    """The previous step's solver correction that the learned features read ([V,3], model order)."""
    rng = np.random.default_rng([seed, 7])
    q = model.particle_q.astype(np.float64)
    c = np.stack([_waves(q[:, 0], q[:, 1], 2.0, rng) for _ in range(3)], axis=1)
    return _tensor((3e-4 * c).astype(np.float32))


def _rows(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    X = torch.randn(case["rows"], IN, generator=g, device=DEVICE)
    X[:, IN - 1] = 1.0
    return X, 0.05 * torch.randn(case["rows"], 3, generator=g, device=DEVICE) + 0.02 * X[:, :3]


def prepare(case, seed):
    if case["kind"].startswith("mlp"):
        X, T = _rows(case, seed)
        return {"kind": case["kind"], "mlp": _network(seed), "X": X, "T": T}
    s = {"kind": case["kind"], "solvers": [], "pipes": [], "contacts": [], "in": [], "out": [], "q": []}
    for j, (model, q0) in enumerate(_models(case)):
        kw = dict(particle_enable_self_contact=True, particle_self_contact_radius=SELF_RADIUS,
                  particle_self_contact_margin=SELF_MARGIN) if case["kind"] == "self" else {}
        solver = SolverVBD(model, iterations=case.get("iterations", 10), **kw)
        if "gate" in case:
            solver.set_residual_gate(**_gate(case))
        pipe = CollisionPipeline(model, soft_contact_margin=MARGIN) if model.shape_count else None
        q, qd, f = _state(case["kind"], model, q0, seed + 1000003 * j)
        a, b = model.state(), model.state()
        s["q"].append(_tensor(q))
        a.particle_qd.copy_(_tensor(qd))
        a.particle_f.copy_(_tensor(f))
        for key, v in (("solvers", solver), ("pipes", pipe), ("contacts", pipe.contacts() if pipe else None),
                       ("in", a), ("out", b)):
            s[key].append(v)
    if case["kind"] == "learned":
        s["mlp"] = _network(seed)
        s["correction"] = _correction(model, seed)
        solver.set_warm_start(s["mlp"], case["iterations"])
    return s


def run(state):
    if state["kind"] == "mlp_forward":
        return state["mlp"].forward(state["X"])
    if state["kind"] == "mlp_train":
        mlp = state["mlp"]
        loss = mlp.gradients(state["X"], state["T"])
        mlp.adam(1e-3)
        return {"loss": loss, "grads": mlp.grads, "params": mlp.params}
    for pipe, contacts, a, q in zip(state["pipes"], state["contacts"], state["in"], state["q"]):
        a.particle_q.copy_(q)
        if pipe is not None:
            pipe.collide(a, contacts)
    if state["kind"] == "batch":
        SolverVBD.step_batch(state["solvers"], state["in"], state["out"], state["contacts"], DT)
        return [(b.particle_q, b.particle_qd) for b in state["out"]]
    solver, a, b = state["solvers"][0], state["in"][0], state["out"][0]
    if state["kind"] == "learned":
        solver.set_warm_start_correction(state["correction"])
    solver.step(a, b, None, state["contacts"][0], DT)
    return b.particle_q, b.particle_qd


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far another correct implementation may be off
# ------------------------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "mlp_forward":
        return {"bytes": case["rows"] * 4 * (IN + 3) + 4 * N_PARAMS, "flops": case["rows"] * 2 * 25600}
    if case["kind"] == "mlp_train":
        # forward, the gradients of both operands (none for the inputs), Adam's five arrays
        return {"bytes": case["rows"] * 4 * (IN + 3) + 4 * N_PARAMS * 8, "flops": case["rows"] * 2 * (3 * 25600 - 8192)}
    if case["kind"] == "worlds":
        V = case["worlds"] * (56.0 ** 2 + 23.4 ** 2)  # N x N vertices, N ~ U{16..96}: mean 56, deviation 23.4
    elif case["kind"] == "batch":
        k = case["count"]
        V = float(sum((case["n"] + (case["n_max"] - case["n"]) * j // max(k - 1, 1)) ** 2 for j in range(k)))
    else:
        V = float(case["n"] ** 2)
    T, E = 2.0 * V, 3.0 * V
    iterations = case.get("iterations", 8)
    # each vertex is in six triangles and twelve hinges: about 150 flops a record, twice the plain
    # formulas' count where velocities damp; reads state, model and contacts once, writes the state
    flops = iterations * V * 18 * (300 if case["kind"] == "curtain" else 150)
    nbytes = V * (36 + 24 + 16 + 12) + 44 * T + 32 * E + 8 * (3 * T + 4 * E)
    if case["kind"] == "learned":
        flops += V * 2 * 25600
        nbytes += 12 * V + 4 * N_PARAMS
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # the velocities decide: (x - x_prev) / dt magnifies the last bit of a position 600 times.  Each
    # figure is about four times what 32-bit arithmetic shows against 64 bits (hanging and curtain
    # move slowest, so they show most; the self-contact barrier magnifies it on large cloths); the
    # network runs on 16-bit operands (FP16 inference, BF16 training).
    return {"hanging": {"rel": 6e-4}, "batch": {"rel": 1e-4}, "drape": {"rel": 2e-4}, "curtain": {"rel": 1e-3},
            "worlds": {"rel": 2e-4}, "self": {"rel": 1e-3}, "learned": {"rel": 5e-4}, "mlp_forward": {"rel": 3e-3},
            "mlp_train": {"rel": 1.2e-2}}[case["kind"]]


# ------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------
def _dot(a, b):
    return (a * b).sum(-1)


def _outer(a):
    return a[:, :, None] * a[:, None, :]


def _eye(s):
    return s[:, None, None] * torch.eye(3, dtype=s.dtype, device=s.device)


def _rotate(q, v):
    u, w = q[:3].expand_as(v), q[3]
    return v * (2 * w * w - 1) + torch.linalg.cross(u, v) * (2 * w) + u * (2 * _dot(u, v))[:, None]


class _Exact:
    """One substep of a model in 64 bits, on the model's own arrays."""

    def __init__(self, model, self_contact=False):
        self.m = m = model

        def d(a):
            return torch.as_tensor(np.asarray(a), device=DEVICE).double()

        def i(a):
            return torch.as_tensor(np.asarray(a).astype(np.int64), device=DEVICE)

        self.mass, self.radius = d(m.particle_mass), d(m.particle_radius)
        self.solved = ((i(m.particle_flags) & 1) != 0) & (self.mass != 0)
        self.g = d(np.asarray(m.gravity).reshape(-1, 3)[0])
        self.tri, self.edge = i(m.tri_indices).reshape(-1, 3), i(m.edge_indices).reshape(-1, 4)
        self.D, self.area, self.tmat = d(m.tri_poses), d(m.tri_areas), d(m.tri_materials)
        self.rest, self.length, self.bend = d(m.edge_rest_angle), d(m.edge_rest_length), d(m.edge_bending_properties)
        self.world = i(m.particle_world)
        hinge = (self.edge[:, 0] >= 0) & (self.edge[:, 1] >= 0) & (self.bend[:, 0] > 0)
        color = torch.full((m.particle_count,), -1, dtype=torch.int64, device=DEVICE)
        for c, group in enumerate(m.particle_color_groups):
            color[i(group)] = c
        self.colors = []
        for c in range(len(m.particle_color_groups)):
            mine = (color == c)
            tris = [torch.nonzero(mine[self.tri[:, k]] & self.solved[self.tri[:, k]]).reshape(-1) for k in range(3)]
            hinges = [torch.nonzero(hinge & mine[self.edge[:, k].clamp_min(0)] & self.solved[self.edge[:, k].clamp_min(0)])
                      .reshape(-1) for k in range(4)]
            self.colors.append((torch.nonzero(mine & self.solved).reshape(-1), tris, hinges))
        self.self_contact = self_contact
        if self_contact:
            a, b = self.edge[:, 2], self.edge[:, 3]
            V = m.particle_count
            self.ring = torch.unique(torch.cat([a * V + b, b * V + a, torch.arange(V, device=DEVICE) * (V + 1)]))

    # ---- particle against static shapes ----
    def collide(self, q):
        m, out = self.m, []
        kd_all, ke_all, mu_all = float(m.soft_contact_kd), float(m.soft_contact_ke), float(m.soft_contact_mu)
        for s in range(m.shape_count):
            t = torch.as_tensor(m.shape_transform[s], device=DEVICE).double()
            rot, inv = t[3:], t[3:] * torch.tensor([-1.0, -1.0, -1.0, 1.0], device=DEVICE, dtype=torch.float64)
            x = _rotate(inv, q - t[:3])
            kind, scale = int(m.shape_type[s]), [float(v) for v in m.shape_scale[s]]
            if kind == 3:
                l = x.norm(dim=1)
                dist, n = l - scale[0], x / l[:, None]
            elif kind == 7:
                half = torch.tensor(scale, device=DEVICE, dtype=torch.float64)
                over = x.abs() - half
                outside = (over > 0).any(1)
                away = x - torch.minimum(torch.maximum(x, -half), half)
                dist = torch.where(outside, away.norm(dim=1), over.max(1).values)
                axis = torch.nn.functional.one_hot(over.argmax(1), 3) * torch.where(x < 0, -1.0, 1.0)
                n = torch.where(outside[:, None], away / away.norm(dim=1).clamp_min(1e-300)[:, None], axis.double())
            else:
                dist, n = x[:, 2], torch.zeros_like(x)
                n[:, 2] = 1.0
            near = dist < MARGIN + float(m.shape_margin[s]) + self.radius
            w = int(m.shape_world[s])
            if w >= 0:
                near &= self.world == w
            p = torch.nonzero(near & ((torch.as_tensor(m.particle_flags, device=DEVICE) & 1) != 0)).reshape(-1)
            out.append((p, _rotate(rot, x[p] - n[p] * dist[p, None]) + t[:3], _rotate(rot, n[p]),
                        0.5 * (ke_all + float(m.shape_material_ke[s])), 0.5 * (kd_all + float(m.shape_material_kd[s])),
                        math.sqrt(mu_all * float(m.shape_material_mu[s])), float(m.shape_margin[s])))
        p = torch.cat([o[0] for o in out]) if out else torch.zeros(0, dtype=torch.int64, device=DEVICE)
        self.touched = torch.zeros(m.particle_count, dtype=torch.bool, device=DEVICE)
        self.touched[p] = True
        self.by_color = []
        pos, nrm = (torch.cat([o[k] for o in out]) if out else torch.zeros(0, 3, device=DEVICE).double() for k in (1, 2))
        mat = torch.cat([torch.tensor(o[3:], device=DEVICE, dtype=torch.float64).expand(len(o[0]), 4) for o in out]) \
            if out else torch.zeros(0, 4, device=DEVICE).double()
        for ids, _, _ in self.colors:
            mine = torch.zeros(m.particle_count, dtype=torch.bool, device=DEVICE)
            mine[ids] = True
            k = torch.nonzero(mine[p]).reshape(-1)
            self.by_color.append((p[k], pos[k], nrm[k], mat[k]))

    def shape_contacts(self, c, x, prev, f, H):
        p, pos, n, mat = self.by_color[c]
        pen = -(_dot(n, x[p] - pos) - self.radius[p] - mat[:, 3])
        on = pen > 0
        p, pos, n, mat, pen = p[on], pos[on], n[on], mat[on], pen[on]
        rel = x[p] - prev[p]
        fn, dn = pen * mat[:, 0], _dot(n, rel)
        damp = torch.where(dn < 0, mat[:, 1] / DT, 0.0)
        force = n * (fn - damp * dn)[:, None]
        nn = _outer(n)
        hess = nn * (mat[:, 0] + damp)[:, None, None]
        ut = rel - n * dn[:, None]
        un, eps = ut.norm(dim=1), 1e-2 * DT
        f1 = torch.where(un > eps, 1 / un.clamp_min(1e-300), (-un / eps + 2) / eps)
        sc = torch.where(un > 0, mat[:, 2] * fn * f1, 0.0)
        f.index_add_(0, p, force - sc[:, None] * ut)
        H.index_add_(0, p, hess + _eye(sc) - sc[:, None, None] * nn)

    # ---- membrane and bending ----
    def membrane(self, t, k, x, prev, f, H):
        a, b, c = (self.tri[t, j] for j in range(3))
        D, area, mat = self.D[t], self.area[t], self.tmat[t]
        mu, lam = mat[:, 0], mat[:, 0] + mat[:, 1]
        alpha = 1 + mu / torch.where(lam < 0, -1.0, 1.0) / lam.abs().clamp_min(1e-6)

        def grad(y):
            u, v = y[b] - y[a], y[c] - y[a]
            return u * D[:, 0, 0, None] + v * D[:, 1, 0, None], u * D[:, 0, 1, None] + v * D[:, 1, 1, None]

        F0, F1 = grad(x)
        c00, c11, c01 = _dot(F0, F0), _dot(F1, F1), _dot(F0, F1)
        J = (c00 * c11 - c01 * c01).clamp_min(1e-20).sqrt()
        g0 = (c11[:, None] * F0 - c01[:, None] * F1) / J[:, None]
        g1 = (c00[:, None] * F1 - c01[:, None] * F0) / J[:, None]
        d = (-(D[:, 0] + D[:, 1])) if k == 0 else D[:, k - 1]
        d0, d1 = d[:, 0], d[:, 1]
        s = lam * (J - alpha)
        ff = -((mu[:, None] * F0 + s[:, None] * g0) * d0[:, None] + (mu[:, None] * F1 + s[:, None] * g1) * d1[:, None])
        r = s.clamp_min(0) / J
        dJ, w = g0 * d0[:, None] + g1 * d1[:, None], F1 * d0[:, None] - F0 * d1[:, None]
        h = _eye(mu * (d0 * d0 + d1 * d1) + r * (d0 * d0 * c11 + d1 * d1 * c00 - 2 * d0 * d1 * c01))
        h = h + (lam - r)[:, None, None] * _outer(dJ) - r[:, None, None] * _outer(w)
        if bool((mat[:, 2] > 0).any()):
            P0, P1 = grad(prev)
            kd = mat[:, 2]
            rates = [(c00 - _dot(P0, P0)) / DT, (c01 - _dot(P0, P1)) / DT, (c11 - _dot(P1, P1)) / DT]
            dirs = [2 * d0[:, None] * F0, d0[:, None] * F1 + d1[:, None] * F0, 2 * d1[:, None] * F1]
            for weight, rate, e in zip((1.0, 2.0, 1.0), rates, dirs):
                ff = ff - (weight * kd * rate)[:, None] * e
                h = h + (weight * kd / DT)[:, None, None] * _outer(e)
        v = self.tri[t, k]
        f.index_add_(0, v, ff * area[:, None])
        H.index_add_(0, v, h * area[:, None, None])

    def bending(self, t, k, x, prev, f, H):
        ids = [self.edge[t, j] for j in range(4)]

        def angle(y):
            x0, x1, x2, x3 = (y[j] for j in ids)
            n1, n2, e = torch.linalg.cross(x2 - x0, x3 - x0), torch.linalg.cross(x3 - x1, x2 - x1), x3 - x2
            l = e.norm(dim=1)
            return torch.atan2(_dot(torch.linalg.cross(n1, n2), e) / l, _dot(n1, n2)), n1, n2, e, l, x0, x1, x2, x3

        theta, n1, n2, e, l, x0, x1, x2, x3 = angle(x)
        n1, n2 = n1 / _dot(n1, n1)[:, None], n2 / _dot(n2, n2)[:, None]
        if k == 0:
            g = -l[:, None] * n1
        elif k == 1:
            g = -l[:, None] * n2
        elif k == 2:
            g = (_dot(e, x3 - x0) / l)[:, None] * n1 + (_dot(e, x3 - x1) / l)[:, None] * n2
        else:
            g = -(_dot(e, x2 - x0) / l)[:, None] * n1 - (_dot(e, x2 - x1) / l)[:, None] * n2
        ke = self.bend[t, 0] * self.length[t]
        kd = self.bend[t, 1] * self.length[t]
        mag, stiff = ke * (theta - self.rest[t]), ke
        if bool((kd > 0).any()):
            turn = theta - angle(prev)[0]
            turn = turn - 2 * math.pi * torch.round(turn / (2 * math.pi))
            mag, stiff = mag + kd * turn / DT, stiff + kd / DT
        f.index_add_(0, ids[k], -mag[:, None] * g)
        H.index_add_(0, ids[k], stiff[:, None, None] * _outer(g))

    # ---- one color's forces and Hessian blocks ----
    def forces(self, c, x, prev, y):
        ids, tris, hinges = self.colors[c]
        f = torch.zeros_like(x)
        H = torch.zeros(len(x), 3, 3, dtype=x.dtype, device=x.device)
        for k in range(3):
            self.membrane(tris[k], k, x, prev, f, H)
        for k in range(4):
            self.bending(hinges[k], k, x, prev, f, H)
        if self.m.shape_count:
            self.shape_contacts(c, x, prev, f, H)
        if self.self_contact:
            self.pair_forces(x, prev, f, H)
        m = self.mass[ids] / (DT * DT)
        return ids, f[ids] + m[:, None] * (y[ids] - x[ids]), H[ids] + _eye(m)

    def residual(self, ids, f):
        return (f.norm(dim=1) / (self.mass[ids] * self.g.norm())).clamp_max(1e9).sum()

    def step(self, q, qd, f_ext, iterations, gate=None, start=None):
        prev = q.double()
        solved = self.solved[:, None]
        inv = torch.where(self.mass > 0, 1 / self.mass.clamp_min(1e-300), 0.0)[:, None]
        move = torch.where(solved, (qd.double() + (self.g + f_ext.double() * inv) * DT) * DT, 0.0)
        y = prev + move
        if self.m.shape_count:
            self.collide(prev)
        base, disp = prev, move
        if self.self_contact:
            self.detect(base)
            disp = self.truncate(base, disp)
        x = base + disp
        count = int(self.solved.sum())
        if gate:
            ref = sum(self.residual(*self.forces(c, x, prev, y)[:2]) for c in range(len(self.colors))) / count
        if start is not None:
            x = x + start(self, prev, y)
        done = 0
        while done < (gate["max_iterations"] if gate else iterations):
            if self.self_contact and done == 0:
                base, disp = x, torch.zeros_like(x)
                self.detect(base)
            total = 0.0
            for c in range(len(self.colors)):
                ids, f, H = self.forces(c, x, prev, y)
                total = total + self.residual(ids, f)
                dx = torch.linalg.solve(H, f)
                if self.self_contact:
                    disp = disp.index_add(0, ids, dx)
                    disp = self.truncate(base, disp)
                    x = base + disp
                else:
                    x = x.index_add(0, ids, dx)
            done += 1
            if gate and not float(total / count) > gate["tolerance"] * float(ref):
                break
        return x, (x - prev) / DT

    # ---- self-contact ----
    def near(self, a, b):
        key = a * self.m.particle_count + b
        at = torch.searchsorted(self.ring, key).clamp_max(len(self.ring) - 1)
        return self.ring[at] == key

    def detect(self, x):
        """Vertex-triangle pairs and ordered edge-edge pairs closer than the margin."""
        def boxes(ids):
            p = x[ids]
            return p.amin(1), p.amax(1)

        def overlaps(lo, hi, glo, ghi):
            found = []
            for b in range(0, len(lo), 2048):
                l, h = lo[b:b + 2048, None] - SELF_MARGIN, hi[b:b + 2048, None] + SELF_MARGIN
                hit = torch.ones(l.shape[0], len(glo), dtype=torch.bool, device=x.device)
                for k in range(3):
                    hit &= (glo[None, :, k] <= h[..., k]) & (ghi[None, :, k] >= l[..., k])
                i, j = torch.nonzero(hit, as_tuple=True)
                found.append((i + b, j))
            return torch.cat([i for i, _ in found]), torch.cat([j for _, j in found])

        tlo, thi = boxes(self.tri)
        v, t = overlaps(x, x, tlo, thi)
        keep = ~(self.near(v, self.tri[t, 0]) | self.near(v, self.tri[t, 1]) | self.near(v, self.tri[t, 2]))
        v, t = v[keep], t[keep]
        cp, _ = self.closest_on_triangle(x, v, t)
        keep = (cp - x[v]).norm(dim=1) < SELF_MARGIN
        self.vt = (v[keep], t[keep])
        ends = self.edge[:, 2:]
        lo, hi = boxes(ends)
        e, g = overlaps(lo, hi, lo, hi)
        keep = torch.ones(len(e), dtype=torch.bool, device=x.device)
        for i in range(2):
            for j in range(2):
                keep &= ~self.near(ends[e, i], ends[g, j])
        e, g = e[keep], g[keep]
        s, u = self.closest_on_edges(x, e, g)
        a, b = ends[e], ends[g]
        dist = (torch.lerp(x[a[:, 0]], x[a[:, 1]], s[:, None]) - torch.lerp(x[b[:, 0]], x[b[:, 1]], u[:, None])).norm(dim=1)
        keep = dist < SELF_MARGIN
        self.ee = (e[keep], g[keep])

    def closest_on_triangle(self, x, v, t):
        a, b, c, p = x[self.tri[t, 0]], x[self.tri[t, 1]], x[self.tri[t, 2]], x[v]
        ab, ac = b - a, c - a
        d1, d2, d3, d4 = _dot(ab, p - a), _dot(ac, p - a), _dot(ab, p - b), _dot(ac, p - b)
        d5, d6 = _dot(ab, p - c), _dot(ac, p - c)
        va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
        one, zero = torch.ones_like(d1), torch.zeros_like(d1)
        den = va + vb + vc
        r = torch.stack([1 - vb / den - vc / den, vb / den, vc / den], 1)
        w = (d4 - d3) / ((d4 - d3) + (d5 - d6))
        # the first region that holds decides: corners a, b, c, then edges ab, ac, bc, else the face
        for test, bary in (((va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0), (zero, 1 - w, w)),
                           ((vb <= 0) & (d2 >= 0) & (d6 <= 0), (1 - d2 / (d2 - d6), zero, d2 / (d2 - d6))),
                           ((vc <= 0) & (d1 >= 0) & (d3 <= 0), (1 - d1 / (d1 - d3), d1 / (d1 - d3), zero)),
                           ((d6 >= 0) & (d5 <= d6), (zero, zero, one)),
                           ((d3 >= 0) & (d4 <= d3), (zero, one, zero)),
                           ((d1 <= 0) & (d2 <= 0), (one, zero, zero))):
            r = torch.where(test[:, None], torch.stack(bary, 1), r)
        return r[:, :1] * a + r[:, 1:2] * b + r[:, 2:] * c, r

    def closest_on_edges(self, x, e, g):
        ends = self.edge[:, 2:]
        p1, p2 = x[ends[e, 0]], x[ends[g, 0]]
        d1, d2, r = x[ends[e, 1]] - p1, x[ends[g, 1]] - p2, p1 - p2
        a, ee, f, c, b = _dot(d1, d1), _dot(d2, d2), _dot(d2, r), _dot(d1, r), _dot(d1, d2)
        den = a * ee - b * b
        s = torch.where(den != 0, (b * f - c * ee) / den, 0.0).clamp(0, 1)
        t = (b * s + f) / ee
        s = torch.where(t < 0, (-c / a).clamp(0, 1), torch.where(t > 1, ((b - c) / a).clamp(0, 1), s))
        return s, t.clamp(0, 1)

    def pair_forces(self, x, prev, f, H):
        m = self.m
        ke, kd, mu = float(m.soft_contact_ke), float(m.soft_contact_kd), float(m.soft_contact_mu)

        def add(ids, weights, gain):
            """Participants `ids` with the weights of the difference vector; `gain`: those that get their share."""
            diff = sum(w[:, None] * x[i] for i, w in zip(ids, weights))
            dis = diff.norm(dim=1)
            on = (dis > 0) & (dis < SELF_RADIUS)
            ids, weights, diff, dis = [i[on] for i in ids], [w[on] for w in weights], diff[on], dis[on]
            n = diff / dis[:, None]
            tau, dmin = 0.5 * SELF_RADIUS, 1e-5
            k2 = tau * tau * ke
            near, least = (dis < tau) & (dis > dmin), dis <= dmin
            dE = torch.where(near, -k2 / dis, torch.where(least, k2 * (dis - 2 * dmin) / dmin ** 2, -ke * (SELF_RADIUS - dis)))
            d2E = torch.where(near, k2 / dis ** 2, torch.where(least, torch.full_like(dis, k2 / dmin ** 2), torch.full_like(dis, ke)))
            dx = sum(w[:, None] * (x[i] - prev[i]) for i, w in zip(ids, weights))
            dn = _dot(n, dx)
            ut = dx - n * dn[:, None]
            un, eps = ut.norm(dim=1), 1e-2 * DT
            f1 = torch.where(un > eps, 1 / un.clamp_min(1e-300), (-un / eps + 2) / eps)
            slide = torch.where(un > 0, mu * -dE * f1, 0.0)
            rate = dn / DT
            damp = torch.where(rate < -1e-6, -kd * rate, 0.0)
            dh = torch.where(rate < -1e-6, torch.full_like(rate, kd / DT), 0.0)
            nn = _outer(n)
            h = nn * (d2E + dh)[:, None, None] + (_eye(slide) - slide[:, None, None] * nn)
            for j in gain:
                w = weights[j]
                f.index_add_(0, ids[j], w[:, None] * (n * (-dE)[:, None] - slide[:, None] * ut) + (damp * w)[:, None] * n)
                H.index_add_(0, ids[j], (w * w)[:, None, None] * h)

        v, t = self.vt
        _, bary = self.closest_on_triangle(x, v, t)
        add([v, *(self.tri[t, j] for j in range(3))], [torch.ones_like(bary[:, 0]), *(-bary[:, j] for j in range(3))],
            range(4))
        e, g = self.ee
        ends = self.edge[:, 2:]
        s, u = self.closest_on_edges(x, e, g)
        add([ends[e, 0], ends[e, 1], ends[g, 0], ends[g, 1]], [1 - s, s, -(1 - u), -u], range(2))

    def truncate(self, base, disp):
        """Division planes of all pairs shorten the displacements that would cross them."""
        ratio = torch.ones(len(base), dtype=base.dtype, device=base.device)

        def cut(first, second, n, d, mine, other, far):
            for ids, reach in ((first, mine), (second, other)):
                for i in ids:
                    den, num = _dot(n, disp[i]), -_dot(n, base[i] - d)
                    t = num / torch.where(den == 0, 1.0, den)
                    crosses = (reach != 0) & (den.abs() >= 1e-6) & (t >= -1e-8) & (t <= 1 + far)
                    stop = torch.minimum(t * 0.85, t - 1e-3).clamp(0, 1)
                    stop = torch.where(crosses & (den.abs() >= 1e-5) & (t >= 0), stop, 1.0)
                    ratio.scatter_reduce_(0, i, stop, "amin")

        def plane(cp, diff, first, second):
            n = diff / diff.norm(dim=1).clamp_min(1e-300)[:, None]
            mine = torch.stack([-_dot(n, disp[i]) for i in first], 1).amax(1).clamp_min(0)
            other = torch.stack([_dot(n, disp[i]) for i in second], 1).amax(1).clamp_min(0)
            both = mine + other
            l = torch.where(both == 0, 0.5, (other / torch.where(both == 0, 1.0, both)).clamp(0.05, 0.95))
            return n, cp + l[:, None] * diff, mine, other

        v, t = self.vt
        cp, _ = self.closest_on_triangle(base, v, t)
        corners = [self.tri[t, j] for j in range(3)]
        cut([v], corners, *plane(cp, base[v] - cp, [v], corners), 1e-8)
        e, g = self.ee
        ends = self.edge[:, 2:]
        s, u = self.closest_on_edges(base, e, g)
        a, b = [ends[e, 0], ends[e, 1]], [ends[g, 0], ends[g, 1]]
        c1 = torch.lerp(base[a[0]], base[a[1]], s[:, None])
        c2 = torch.lerp(base[b[0]], base[b[1]], u[:, None])
        cut(a, b, *plane(c2, c1 - c2, a, b), 1e-6)
        disp = disp * ratio[:, None]
        l, most = disp.norm(dim=1), SELF_MARGIN * 0.85 * 0.5
        return disp * torch.where(l > most, most / l.clamp_min(1e-300), 1.0)[:, None]


def _exact_network(params, X):
    p = params.double()
    W1, W2 = p[OFF_W1:OFF_B1].reshape(IN, 128), p[OFF_W2:OFF_B2].reshape(128, 128)
    W3 = p[OFF_W3:OFF_B3].reshape(128, 8)
    silu = torch.nn.functional.silu
    out = []
    for b in range(0, len(X), 1 << 17):
        h = silu(X[b:b + (1 << 17)].double() @ W1 + p[OFF_B1:OFF_W2])
        out.append((silu(h @ W2 + p[OFF_B2:OFF_W3]) @ W3 + p[OFF_B3:])[:, :3])
    return torch.cat(out)


def _exact_start(params, mean, inv_std, correction):
    """The learned start: one-ring features of every vertex, the network, the bounded move."""
    def start(ex, prev, y):
        m = ex.m
        V = m.particle_count
        adj = m.soft_mesh_adjacency
        off, val = np.asarray(adj.v_adj_tris_offsets), np.asarray(adj.v_adj_tris)
        tris = np.asarray(m.tri_indices)
        near = np.full((V, 8), -1, np.int64)
        soft = np.zeros((V, 4))
        for v in range(V):
            t = val[off[v]:off[v + 1]:2]
            ring = dict.fromkeys(int(u) for u in tris[t].reshape(-1) if u != v)
            near[v, :min(len(ring), 8)] = list(ring)[:8]
            soft[v, 3] = np.sqrt(2.0 * m.tri_areas[t].astype(np.float64)).mean()
        soft[:, 0] = np.log10(float(m.tri_materials[0, 0]))
        soft[:, 1] = np.log10(float(m.tri_materials[0, 1]))
        soft[:, 2] = np.log10(float(m.edge_bending_properties[0, 0]))
        near, soft = _tensor(near), _tensor(soft)
        L = soft[:, 3]
        F = torch.zeros(V, IN, dtype=torch.float64, device=DEVICE)
        corr = correction.double()
        F[:, 0:3], F[:, 3:6] = (y - prev) / L[:, None], corr / L[:, None]
        for j in range(8):
            have = (near[:, j] >= 0)[:, None]
            u = near[:, j].clamp_min(0)
            F[:, 6 + 3 * j:9 + 3 * j] = torch.where(have, (prev[u] - prev) / L[:, None], 0.0)
            F[:, 30 + 3 * j:33 + 3 * j] = torch.where(have, corr[u] / L[:, None], 0.0)
        F[:, 54:57], F[:, 57] = soft[:, :3], torch.log10(ex.mass)
        F[:, 58], F[:, 59] = ex.touched.double(), (near >= 0).sum(1) / 8.0
        F[:, 60], F[:, 63] = ex.solved.double(), 1.0
        p = _exact_network(params, (F - mean.double()) * inv_std.double())
        l = p.norm(dim=1)
        return torch.where(ex.solved[:, None], p * (L * torch.where(l > 0.25, 0.25 / l.clamp_min(1e-300), 1.0))[:, None], 0.0)

    return start


def exact(case, seed):
    if case["kind"] == "mlp_forward":
        return _exact_network(_network(seed).params, _rows(case, seed)[0])
    if case["kind"] == "mlp_train":
        X, T = _rows(case, seed)
        p = _network(seed).params.double().requires_grad_(True)
        se = ((_exact_network(p, X) - T.double()) ** 2).sum()
        (g,) = torch.autograd.grad(se / len(X), p)
        lr, b1, b2, eps = 1e-3, 0.9, 0.999, 1e-8
        m1, m2 = (1 - b1) * g, (1 - b2) * g * g
        step = lr * (m1 / (1 - b1)) / ((m2 / (1 - b2)).sqrt() + eps)
        return {"loss": se.detach().reshape(1), "grads": g, "params": p.detach() - step}
    if case["kind"] == "self" and case["n"] > 200:
        return None  # the search over all pairs takes too long
    out = []
    for j, (model, q0) in enumerate(_models(case)):
        q, qd, f = (_tensor(a) for a in _state(case["kind"], model, q0, seed + 1000003 * j))
        start = None
        if case["kind"] == "learned":
            mlp = _network(seed)
            start = _exact_start(mlp.params, mlp.mean, mlp.inv_std, _correction(model, seed))
        ex = _Exact(model, case["kind"] == "self")
        out.append(ex.step(q, qd, f, case.get("iterations", 10), _gate(case) if "gate" in case else None, start))
    return out if case["kind"] == "batch" else out[0]
