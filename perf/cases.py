"""What is timed: the calls a user of the simulator makes, over the sizes they make them at.

A case is a dict of plain values. `listed()` gives the fixed ones, `draw(rng)` one more of the same
ranges; `prepare(case, seed)` builds the cloths and their states (inputs from the seed alone),
`run(state)` makes one pass through the package's public entry points, `work(case)` says what a pass
cannot do without, and `exact(case, seed)` computes the same outputs in plain torch in 64 bits.

Kinds of case:

- simstep   the reference-style single cloth: Cloth, PhysicsCloth, SimStep, states as numpy arrays
- step      ClothBatch.step of a batch, states as CUDA tensors; schedule "launches" (the default),
            "graph" (one CUDA graph a step) or "persistent" (graph + one solve kernel)
- learned   the same with the learned preconditioner, its network evaluated every step
- system    assemble, solve, read the solution, apply the matrix (FillMV and EigenSolver on their own)
- tangent   step_tangent: a step with eight material directions on two copies of a cloth
- adjoint   Adjoint.step_back: one reverse step of a rollout's gradient
- respond   Collider: continuous collision detection, the impact-zone response of one step and its backward
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

ys = importlib.import_module("fine-grained-differentiable-physics-a-yarn-level-model-for-fabrics_gb300")

KEYS = ("LPos", "LPosFix", "LVel", "EPos", "EPosBar", "EVel")
BASE = np.array([1e-3, 1e3, 1e-5])  # density, stretch, bend of the benchmark's yarns
L, R = 1e-3, 1e-4


# ------------------------------------------------------------------ the cases
def listed():
    c = lambda name, kind, **kw: dict(dict(  # noqa: E731
        name=name, kind=kind, cloths=1, side_min=0, side_max=0, width=0, length=0, weave=0, blend=False, pose=0,
        h=1e-3, tol=1e-10, ext=False, wind=True, schedule="launches"), **kw)
    return [
        # the smallest call: the 5 x 5 cloth of the reference's drivers, stepped through its own interface
        # with the solver's default tolerance; launches and host work are all there is
        c("simstep 5x5", "simstep", width=5, length=5, tol=0.0),
        # a parameter-learning cloth (two yarns, twill), one cloth, one solve kernel: latency of one chain
        c("step 17x17 twill", "step", width=17, length=17, weave=1, blend=True, schedule="persistent"),
        # the collision scene's flat cloth at its step size and the default tolerance
        c("step 50x50 flat", "step", width=50, length=50, pose=1, h=5e-4, tol=0.0, wind=False,
          schedule="persistent"),
        # one large hanging cloth: the batch kernels on a grid that does not fill the GPU twice
        c("step 100x100", "step", width=100, length=100, schedule="graph"),
        # a ragged mixed batch, external forces, no schedule chosen: what a first program does
        c("step 24 ragged satin", "step", cloths=24, side_min=7, side_max=41, weave=2, blend=True, ext=True),
        # the headline: 256 hanging cloths, sides 5 to 50, wind
        c("step 256 cloths", "step", cloths=256, side_min=5, side_max=50, schedule="graph"),
        # the solver boundary on its own: FillMV, EigenSolver, products with the matrix; odd sides
        c("system 61x83", "system", width=61, length=83, blend=True),
        # the learned preconditioner's batch
        c("learned 64x40x40", "learned", cloths=64, side_min=40, side_max=40, wind=False, schedule="graph"),
        # forward sensitivities of the eight learned scalars
        c("tangent 17x17 blend", "tangent", width=17, length=17, blend=True, tol=0.0),
        # reverse mode of a training rollout
        c("adjoint 17x17 twill", "adjoint", width=17, length=17, weave=1, blend=True, tol=0.0),
        # reverse mode of the force control of the collision scene's cloth
        c("adjoint 50x50 forces", "adjoint", width=50, length=50, pose=1, h=5e-4, tol=0.0, ext=True, wind=False),
        # one collision step of a 64 x 64 cloth landing on a sphere of 20,480 faces
        c("respond 64x64", "respond", width=64, length=64, levels=5),
    ]


def draw(rng):
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["simstep", "step", "step", "step", "system", "learned", "tangent", "adjoint", "respond"])
    c = dict(kind=kind, cloths=1, side_min=0, side_max=0, width=0, length=0, weave=rng.randrange(3),
             blend=rng.random() < 0.5, pose=rng.randrange(2), h=rng.choice([1e-3, 5e-4]),
             tol=rng.choice([0.0, 1e-10]), ext=kind in ("step", "adjoint") and rng.random() < 0.4,
             wind=rng.random() < 0.6, schedule="launches")
    if kind == "simstep":
        c.update(width=log(3, 30), length=log(3, 30))
    elif kind == "step":
        c["schedule"] = rng.choice(["launches", "graph", "persistent"])
        if c["schedule"] == "persistent":
            c.update(width=log(3, 60), length=log(3, 60))
        elif rng.random() < 0.4:
            c.update(width=log(4, 160), length=log(4, 160))
        else:
            lo = log(3, 30)
            c.update(cloths=log(2, 200), side_min=lo, side_max=rng.randint(lo, 50))
    elif kind == "system":
        c.update(width=log(4, 140), length=log(4, 140))
    elif kind == "learned":
        lo = log(5, 40)
        c.update(cloths=log(1, 64), side_min=lo, side_max=rng.randint(lo, 45), tol=1e-10, schedule="graph")
    elif kind == "tangent":
        c.update(width=log(5, 40), length=log(5, 40))
    elif kind == "adjoint":
        c.update(width=log(4, 36), length=log(4, 36))
    else:
        w = log(16, 90)
        c.update(width=w, length=w, levels=rng.choice([3, 4, 5]), ext=False, wind=False, blend=False, weave=0, pose=1)
    return c


# ------------------------------------------------------------------ the inputs
def _sizes(case):
    """[(width, length)] of the case's cloths (from the case, not the seed: the work is the case's)."""
    if case["cloths"] == 1 and case["width"]:
        return [(case["width"], case["length"])]
    rng = np.random.default_rng([case["cloths"], case["side_min"], case["side_max"]])
    s = rng.integers(case["side_min"], case["side_max"] + 1, size=case["cloths"])
    return [(int(a), int(a)) for a in s]


def _specs(case, rng):
    """Cloth descriptions: materials within +-20 % of the benchmark's, a second yarn 1.5-3 times apart on
    the odd lines of a blend, hanging from two corners (upright) or free (flat)."""
    out = []
    for W, H in _sizes(case):
        scale = 1.5 + 1.5 * rng.random(3)

        def lines(n):
            x = BASE * (1.0 + 0.2 * (2.0 * rng.random((n, 3)) - 1.0))
            if case["blend"]:
                x[1::2] *= scale
            return x

        wind = (0.0, float(math.sqrt(2.0 * rng.random()) * rng.choice([-1.0, 1.0])), 0.0) if case["wind"] else (0.0,) * 3
        out.append(dict(width=W, length=H, warp=lines(H), weft=lines(W), height=0.05, L=L, R=R, pose=case["pose"],
                        weave=case["weave"], kc=1.0, kf=1000.0, df=1000.0, mu=0.3 * (1 + 0.2 * (2 * rng.random() - 1)),
                        S=1e-4 * (1 + 0.2 * (2 * rng.random() - 1)), handle_stiffness=1e4, G=(0.0, 0.0, 9.8),
                        wind_vel=wind, wind_density=1.0 if case["wind"] else 0.0,
                        wind_drag=0.5 if case["wind"] else 0.0,
                        handles=[(0, 0), (W - 1, 0)] if case["pose"] == 0 else []))
    return out


def _state(case, specs, rng):
    """States of cloths in motion: the rest pose bent by two waves of a few crossings' length, stretched by
    a few percent crossing to crossing, slid by a few thousandths of the spacing."""
    parts = {k: [] for k in KEYS}
    for s in specs:
        W, H = s["width"], s["length"]
        v, u = np.meshgrid(np.arange(H), np.arange(W), indexing="ij")
        u, v = u.reshape(-1).astype(float), v.reshape(-1).astype(float)
        n = W * H
        inside = ((u > 0) & (u < W - 1) & (v > 0) & (v < H - 1))[:, None]
        rest = np.stack([u * L, 0 * u, s["height"] - v * L] if s["pose"] == 0 else [u * L, v * L, 0 * u + s["height"]], 1)
        wave = np.zeros((n, 3))
        speed = np.zeros((n, 3))
        for _ in range(2):
            k = 2 * np.pi / rng.uniform(8.0, 20.0, 2)
            f = np.sin(k[0] * u + k[1] * v + rng.uniform(0, 2 * np.pi))[:, None]
            wave += f * rng.uniform(-1, 1, 3) * np.array([0.08, 0.3, 0.08] if s["pose"] == 0 else [0.08, 0.08, 0.3]) * L
            speed += f * rng.uniform(-0.1, 0.1, 3)
        x = rest + wave + 0.02 * L * rng.standard_normal((n, 3))
        fix = x.copy()
        for a, b in s["handles"]:
            fix[a + b * W] = rest[a + b * W]
            x[a + b * W] = rest[a + b * W] + 1e-3 * L * rng.standard_normal(3)
        e = np.stack([u * L, v * L], 1)
        parts["LPos"].append(x)
        parts["LPosFix"].append(fix)
        parts["LVel"].append(speed + 0.01 * rng.standard_normal((n, 3)))
        e = e + inside * 2e-3 * L * rng.standard_normal((n, 2))
        parts["EPos"].append(e)
        parts["EPosBar"].append(e + inside * 2e-4 * L * rng.standard_normal((n, 2)))
        parts["EVel"].append(inside * 2e-5 * rng.standard_normal((n, 2)))
    return {k: np.ascontiguousarray(np.concatenate(p)) for k, p in parts.items()}


def _ext(case, n, rng):
    """External forces of the size of a crossing's weight."""
    return np.ascontiguousarray(np.concatenate([1e-5 * rng.standard_normal((n, 3)), np.zeros((n, 2))], 1)) if case["ext"] else None


def _inputs(case, seed):
    rng = np.random.default_rng([int(seed), 11])
    if case["kind"] == "respond":
        W, H = case["width"], case["length"]
        obs, faces = ys.collide.icosphere(0.03, case["levels"])
        u, v = np.meshgrid(np.arange(W), np.arange(H), indexing="xy")
        xp = np.stack([(u.reshape(-1) - (W - 1) / 2) * L, (v.reshape(-1) - (H - 1) / 2) * L, np.full(W * H, 0.032)], 1)
        x = xp + np.array([0.0, 0.0, -3e-3]) + rng.normal(0.0, 1e-5, xp.shape)
        return dict(x=x, x_prev=xp, v=(x - xp) / 1e-3, obs=obs, faces=faces, gx=rng.standard_normal(x.shape),
                    gv=1e-3 * rng.standard_normal(x.shape))
    specs = _specs(case, rng)
    state = _state(case, specs, rng)
    n = len(state["LPos"])
    d = dict(specs=specs, state=state, ext=_ext(case, n, rng))
    if case["kind"] == "system":
        d["y"] = rng.standard_normal((n, 5))
    if case["kind"] == "tangent":
        t = lambda m, a: a * rng.standard_normal((4, 2 * n, m))  # noqa: E731
        d["tan"] = dict(dlpos=t(3, 1e-2 * L), dlvel=t(3, 1e-2), depos=t(2, 1e-3 * L), deposbar=t(2, 1e-3 * L),
                        devel=t(2, 1e-3))
    if case["kind"] == "adjoint":
        d["grad"] = {k: rng.standard_normal((n, m)) for k, m in (("LPos", 3), ("LVel", 3), ("EPos", 2), ("EVel", 2),
                                                                  ("EPosBar", 2))}
        d["grad"]["LVel"] *= 1e-3
        d["grad"]["EVel"] *= 1e-3
    return d


def _seeds(W, H):
    """Directions of the eight scalars (rho, Y, B of the even and odd lines, S, mu), four a copy."""
    nl = W + H
    odd = np.array([j % 2 for j in range(H)] + [i % 2 for i in range(W)])
    line, cloth = np.zeros((3, 4, 2 * nl)), np.zeros((2, 4, 2))
    for p in range(8):
        c, k = divmod(p, 4)
        if p < 6:
            line[p % 3, k, c * nl:(c + 1) * nl] = odd == p // 3
        else:
            cloth[p - 6, k, c] = 1.0
    return line, cloth


def _cluster(n):
    """A cluster shape of the persistent solve that holds n nodes: up to 256 threads a CTA, then 1024."""
    for threads in (128, 256, 512, 1024):
        for size in (1, 2, 4, 8, 16):
            if threads * size >= n and (size <= 4 or threads >= 256):
                return threads, size
    raise ValueError(n)


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    if kind == "respond":  # host arrays: the collider's interface
        d["collider"] = ys.Collider(case["width"], case["length"], obstacle_faces=d["faces"],
                                    n_obstacle_nodes=len(d["obs"]), thickness=5e-4)
        return dict(d, case=case)
    s = dict(case=case)
    if kind == "simstep":
        p = d["specs"][0]
        yarns = [ys.Yarn(R, *p["warp"][0]), ys.Yarn(R, *p["warp"][1])][: 2 if case["blend"] else 1]
        cloth = ys.Cloth(p["width"], p["length"], p["height"], L, R, yarns, p["kc"], p["kf"], p["df"], p["mu"], p["S"],
                         p["handle_stiffness"], ys.WovenPattern(case["weave"]), ys.InitPose(case["pose"]))
        cloth.set_handles(p["handles"])
        s["phy"] = ys.PhysicsCloth(ys.Environment(cloth, p["G"], ys.Wind(p["wind_vel"], p["wind_density"], p["wind_drag"])))
        s["cloth"], s["state"] = cloth, ys.ClothState(**d["state"])
        return s
    specs = [ys.ClothSpec(**p) for p in d["specs"]] * (2 if kind == "tangent" else 1)
    b = s["batch"] = ys.ClothBatch(specs)
    if kind == "system":
        s.update(state=d["state"], y=d["y"])
    elif kind == "tangent":
        s["state"] = {k: np.concatenate([v, v]) for k, v in d["state"].items()}
        s["tan"] = d["tan"]
        b.tangent_enable(0)
        line, cloth = _seeds(case["width"], case["length"])
        b.tangent_seed(*line, *cloth)
    elif kind == "adjoint":
        s.update(state=d["state"], grad=d["grad"], ext=d["ext"], adjoint=ys.Adjoint(b, "exact"))
    else:
        s["state"] = {k: dev(v) for k, v in d["state"].items()}
        s["ext"] = None if d["ext"] is None else dev(d["ext"])
        s["out"] = {k: torch.empty_like(v) for k, v in s["state"].items()}
        if case["schedule"] != "launches":
            b.use_graphs(True)
        if case["schedule"] == "persistent":
            b.set_pcg_schedule(True, *_cluster(b.total_nodes))
            b.set_producer_threads(64)
        if kind == "learned":
            s["net"] = ys.LearnedPreconditioner.pretrained()
            b.set_preconditioner("learned", s["net"])
        if case["schedule"] != "launches":
            run(s)  # a simulation's first step captures its graph
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind, h, tol = case["kind"], case["h"], case["tol"]
    if kind == "respond":
        c = s["collider"]
        c.set_positions(s["x"], s["x_prev"], s["obs"], s["obs"])
        r = c.respond(v=s["v"], h=1e-3, damp=0.1)
        g = c.respond_backward(s["gx"], s["gv"], impacts=True)
        return dict(x=r["x"], v=r["v"], rounds=r["rounds"], zones=r["zones"], impacts=r["impacts"],
                    grad_x=g["x"], grad_v=g["v"], grad_x_prev=g["x_prev"])
    if kind == "simstep":
        s["cloth"].set_ClothState(s["state"])
        ok = ys.SimStep(s["cloth"], s["phy"], h, tol=tol)
        return dict(s["cloth"].get_ClothState().as_dict(), ok=ok)
    b = s["batch"]
    b.set_state(**s["state"])
    if kind == "system":
        b.assemble(h)
        ok = b.solve(tol=tol).all_ok
        return dict(x=b.solution(), y=b.apply(s["y"]), normals=b.normals(), ok=ok)
    if kind == "tangent":
        b.tangent_set_state(**s["tan"])
        ok = b.step_tangent(h, tol=tol).all_ok
        return dict(state=b.get_state(), tangents=b.tangent_get_state(), ok=ok)
    if kind == "adjoint":
        g, p, e = s["adjoint"].step_back(h, s["grad"], s["ext"], tol=tol, want_ext=case["ext"])
        return dict(state=g, params=p, ext=e)
    ok = b.step(h, s["ext"], tol=tol).all_ok
    return dict(b.get_state(s["out"]), ok=ok)


def work(case):
    """State in and out (15 doubles a node), and about 5,000 operations a node for the element terms plus 320
    for each product of some 15 solver iterations. A reverse or forward derivative of one direction costs
    about as much again; the collision step reads its meshes."""
    n = sum(w * k for w, k in _sizes(case))
    nb, f = 240.0 * n, (5000.0 + 15 * 320.0) * n
    if case["kind"] == "system":
        nb = (120.0 + 4 * 40 + 24) * n
    elif case["kind"] == "tangent":
        nb, f = 2 * nb + 2 * 4 * 192.0 * n, 2 * (1 + 4) * f
    elif case["kind"] == "adjoint":
        nb, f = 2 * nb, 4 * f
    elif case["kind"] == "respond":
        nb, f = 120.0 * n + 48.0 * 10 * 4 ** case["levels"], 5000.0 * n
    return {"bytes": nb, "flops": f}


# ------------------------------------------------------------------ the same in plain torch, 64 bits
PI = 3.1415926535897  # the model's PI


class _Model:
    """One step's system as dense matrices per element: edges (8 unknowns), bend segments (12), shear
    segments (9), and per-node diagonals. Unknown c of node i is 5 i + c: x, y, z, u, v."""

    def __init__(self, specs, device):
        t = lambda a, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=device)  # noqa: E731
        off = line = 0
        node, edge, bend, face, shear = [], [], [], [], []
        for c, s in enumerate(specs):
            W, H = s["width"], s["length"]
            v, u = np.meshgrid(np.arange(H), np.arange(W), indexing="ij")
            u, v = u.reshape(-1), v.reshape(-1)
            inside = (u > 0) & (u < W - 1) & (v > 0) & (v < H - 1)
            if s["weave"] == 0:
                flip = (u + v) % 2 != 0
            elif s["weave"] == 1:
                flip = (u + v % 4) % 4 < 2
            else:
                q = (v - 1) % 4
                flip = (u - 1 + (q // 2) * 3 + (q % 2) * 2) % 4 == 0
            fixed = np.zeros(W * H, bool)
            for a, b in s["handles"]:
                fixed[a + b * W] = True
            i = off + u + v * W
            node.append(np.stack([0 * u + c, u, v, inside, flip & inside, fixed], 1))
            for k, step, pos, n, ln in ((0, 1, u, W, line + v), (1, W, v, H, line + H + u)):
                m = pos < n - 1
                edge.append(np.stack([i, i + step, 0 * i + k, ln], 1)[m])
                m = (pos > 0) & (pos < n - 1)
                bend.append(np.stack([i - step, i, i + step, 0 * i + k, ln], 1)[m])
            m = (u < W - 1) & (v < H - 1)
            tl, tr, bl, br = (x[m] for x in (i, i + 1, i + W, i + W + 1))
            even = ((u + v)[m] % 2 == 0)[:, None]
            face += [np.where(even, np.stack([tl, tr, br], 1), np.stack([tl, tr, bl], 1)),
                     np.where(even, np.stack([tl, br, bl], 1), np.stack([tr, br, bl], 1))]
            for du in (-1, 1):
                for dv in (-1, 1):
                    shear.append(np.stack([i, i + du, i + dv * W], 1)[inside])
            off += W * H
            line += W + H
        cat = lambda x, w: t(np.concatenate(x).reshape(-1, w), torch.int64)  # noqa: E731
        node, self.edge, self.bend, self.face, self.shear = (cat(x, w) for x, w in (
            (node, 6), (edge, 4), (bend, 5), (face, 3), (shear, 3)))
        self.n, self.cloth, self.u, self.v = off, node[:, 0], node[:, 1], node[:, 2]
        self.inside, self.flip, self.fixed = (node[:, k].bool() for k in (3, 4, 5))
        self.inner = self.inside.nonzero()[:, 0]
        W = t([s["width"] for s in specs], torch.int64)
        self.cross = torch.stack([self.inner + o for o in (0, -1, 1)] + [self.inner - W[self.cloth[self.inner]],
                                                                         self.inner + W[self.cloth[self.inner]]], 1)
        self.G, self.wind = t([s["G"] for s in specs]), t([s["wind_vel"] for s in specs])
        one = lambda k: t([s[k] for s in specs])  # noqa: E731
        self.kc, self.kf, self.df, self.kh, self.rho_air, self.drag, self.L, self.R = (one(k) for k in (
            "kc", "kf", "df", "handle_stiffness", "wind_density", "wind_drag", "L", "R"))
        lines = np.concatenate([np.concatenate([s["warp"], s["weft"]]) for s in specs])
        area = np.concatenate([np.full(s["width"] + s["length"], PI * s["R"] ** 2) for s in specs])
        self.par = dict(rho=t(lines[:, 0]), Y=t(lines[:, 1]), B=t(lines[:, 2]), S=one("S"), mu=one("mu"))
        self.area = t(area)
        self.uv0 = torch.stack([self.u, self.v], 1) * self.L[self.cloth, None]

    def normals(self, x):
        p = x[self.cross]
        r = p - p.mean(1, keepdim=True)
        n = torch.cat([torch.linalg.eigh(m)[1][:, :, 0] for m in torch.split(r.transpose(1, 2) @ r, 16384)])
        c = torch.linalg.cross(p[:, 2] - p[:, 1], p[:, 4] - p[:, 3])
        n = n * torch.where(((c * n).sum(1) < 0) != self.flip[self.inner], -1.0, 1.0).to(n)[:, None]
        return torch.zeros_like(x).index_copy(0, self.inner, n)

    def edges(self, st, par, h):
        i0, i1, k, ln = self.edge.T
        x0, x1, a0, a1 = st["LPos"][i0], st["LPos"][i1], st["LVel"][i0], st["LVel"][i1]
        pick = lambda a, i: torch.where(k == 0, a[i, 0], a[i, 1])  # noqa: E731
        du = pick(st["EPos"], i1) - pick(st["EPos"], i0)
        e = [pick(st["EVel"], i0), pick(st["EVel"], i1)]
        rho, ks, c = par["rho"][ln], (par["Y"] * self.area)[ln], self.cloth[i0]
        ins = [self.inside[i0].to(x0), self.inside[i1].to(x0)]
        both = ins[0] * ins[1]
        col = lambda s: s[:, None]  # noqa: E731
        dot = lambda a, b: (a * b).sum(1)  # noqa: E731
        dx = x1 - x0
        w, l = dx / col(du), dx.norm(dim=1)
        d, nw, ww = dx / col(l), w.norm(dim=1), dot(w, w)
        F = [torch.zeros_like(x0), torch.zeros_like(du), torch.zeros_like(x0), torch.zeros_like(du)]
        eye = torch.eye(3, dtype=x0.dtype, device=x0.device)
        mats = {}

        def add(X, a, b, iso, xe, ex, ee, full=None):
            """block (a, b) of matrix X: iso I (+ full), column xe, row ex, corner ee; the Eulerian parts
            where the crossings are interior"""
            m = ins[a] if a == b else both
            blk = iso[:, None, None] * eye + (0 if full is None else full)
            top = torch.cat([blk, (col(m) * xe)[:, :, None]], 2)
            low = torch.cat([(col(m) * ex)[:, None, :], (m * ee)[:, None, None]], 2)
            v = torch.cat([top, low], 1)
            mats[X, a, b] = mats[X, a, b] + v if (X, a, b) in mats else v

        q = rho * du / 6
        g = self.G[c]
        zero = torch.zeros_like(du)
        f = col(ks * (nw - 1)) * d
        P = eye - d[:, :, None] * d[:, None, :]
        rl = torch.relu(torch.where(self.flip[i0] != self.flip[i1], 4.0, 2.0).to(du) * self.R[c] - du)
        crowd = self.kc[c] * self.L[c] * rl
        gx = dot(g, x0 + x1)
        F[0] = F[0] - 0.5 * col(rho * du) * g + f
        F[2] = F[2] - 0.5 * col(rho * du) * g - f
        strain = 0.5 * ks * (nw * nw - 1)
        F[1] = F[1] + 0.5 * rho * gx - strain + crowd
        F[3] = F[3] - 0.5 * rho * gx + strain - crowd
        xe_s = col(ks * nw / du) * d
        for a in range(2):
            for b in range(2):
                s, two = (1.0, 2.0) if a == b else (-1.0, 1.0)
                add("M", a, b, two * q, -two * col(q) * w, -two * col(q) * w, two * q * ww)
                gs = 0.5 * col(rho) * g  # rows x_a, column e_b: +g for e0, -g for e1 (and rows e_a alike)
                add("K", a, b, zero, gs if b == 0 else -gs, gs if a == 0 else -gs, zero)
                add("K", a, b, -s * ks / du, s * xe_s, s * xe_s, -s * ks * nw * nw / du, s * (ks / l)[:, None, None] * P)
                add("K", a, b, zero, 0 * gs, 0 * gs, -crowd)
        # kinetic energy: m0 = 2 v0 + v1, m1 = v0 + 2 v1
        ma, me = [2 * a0 + a1, a0 + 2 * a1], [2 * e[0] + e[1], e[0] + 2 * e[1]]
        Saa = dot(a0, ma[0]) + dot(a1, ma[1])
        Sae = a0 * col(me[0]) + a1 * col(me[1])
        Sea = ma[0] * col(e[0]) + ma[1] * col(e[1])
        See = e[0] * me[0] + e[1] * me[1]
        r6, i1_, i2 = rho / 6, 1 / du, 1 / (du * du)
        Qx = col(i1_) * (Sae + Sea) - 2 * col(i2 * See) * dx
        QM = Saa - dot(w, Sae) - dot(w, Sea) + ww * See
        Qu = -i1_ * (dot(w, Sae) + dot(w, Sea)) + 2 * i1_ * ww * See
        Tx, Tu = 0.5 * col(r6 * du) * Qx, 0.5 * (-r6 * QM + r6 * du * Qu)
        F = [F[0] + Tx, F[1] + Tu, F[2] - Tx, F[3] - Tu]
        Qxu = col(i2) * (Sea - Sae) - 4 * col(i2 * See) * w
        Txu = 0.5 * (-col(r6) * Qx + col(r6 * du) * Qxu)
        Tux = 0.5 * (-col(r6) * Qx - col(r6 * du) * Qxu)
        Quu = -2 * i2 * (dot(w, Sae) + dot(w, Sea)) + 6 * i2 * ww * See
        Tuu = 0.5 * (-2 * r6 * Qu + r6 * du * Quu)
        dud = e[1] - e[0]
        wd = ((a1 - a0) * col(du) - dx * col(dud)) * col(i2)
        wwd = 2 * dot(w, wd)
        BM = [ma[b] - w * col(me[b]) for b in range(2)]
        BMe = [-dot(w, ma[b]) + ww * me[b] for b in range(2)]
        rx = [col(r6 * dud) * BM[b] - col(r6 * du * me[b]) * wd for b in range(2)]
        re = [r6 * dud * BMe[b] + r6 * du * (-dot(wd, ma[b]) + wwd * me[b]) for b in range(2)]
        F = [F[0] - rx[0], F[1] - re[0], F[2] - rx[1], F[3] - re[1]]
        for a in range(2):
            for b in range(2):
                s = 1.0 if a == b else -1.0
                add("K", a, b, s * r6 * i2 * See, s * Txu, s * Tux, s * Tuu)
                s = 1.0 if a == 0 else -1.0
                add("D", a, b, s * q * i1_ * me[b], s * col(q) * (col(i1_) * ma[b] - 2 * col(i2 * me[b]) * dx),
                    s * (-col(r6) * (ma[b] - w * col(me[b])) - col(q * i1_ * me[b]) * w),
                    s * (-r6 * (-dot(w, ma[b]) + ww * me[b]) + q * (-i1_ * dot(w, ma[b]) + 2 * i1_ * ww * me[b])))
        for tt, sw in ((0, -1.0), (1, 1.0)):
            wx, wdx = sw * i1_, -sw * dud * i2
            wu = sw * w * col(i1_)
            wdu = -sw * ((a1 - a0) * col(i2) - 4 * dx * col(dud * i2 * i1_))
            wwu, wwdu = 2 * sw * i1_ * ww, 2 * dot(wu, wd) + 2 * dot(wdu, w)
            wdv = -sw * w * col(i1_)
            wwv, cm = 2 * dot(w, wdv), sw * r6
            for b in range(2):
                ex = col(r6 * dud) * (-col(wx) * ma[b] + 2 * sw * dx * col(i2 * me[b])) + col(r6 * du) * (
                    -col(wdx) * ma[b] + 2 * (col(wx) * wd + w * col(wdx)) * col(me[b]))
                xe = col(r6 * dud * me[b]) * wu - col(r6) * rx[b] - col(r6 * du * me[b]) * wdu
                ee = r6 * dud * (dot(wu, ma[b]) + wwu * me[b]) - r6 * re[b] + r6 * du * (-dot(wdu, ma[b]) + wwdu * me[b])
                add("K", b, tt, -r6 * (dud * wx + du * wdx) * me[b], xe, ex, ee)
                fb = 2.0 if b == tt else 1.0
                ex = col(q) * (-col(wx) * ma[b] + 2 * w * col(wx * me[b])) - fb * (col(r6 * dud) * w + col(q) * wd)
                xe = col(cm) * BM[b] - col(q * me[b]) * wdv - fb * (col(r6 * dud) * w + col(q) * wd)
                ee = cm * BMe[b] + q * (-dot(wdv, ma[b]) + wwv * me[b]) + fb * (r6 * dud * ww + q * wwd)
                add("D", b, tt, q * wx * me[b] - r6 * dud * fb, -xe, -ex, -ee)
        full = lambda X: torch.cat([torch.cat([mats[X, a, b] for b in range(2)], 2) for a in range(2)], 1)  # noqa: E731
        M, K, D = full("M"), full("K"), full("D")
        V = torch.cat([a0, col(ins[0] * e[0]), a1, col(ins[1] * e[1])], 1)
        Fv = torch.cat([F[0], col(ins[0] * F[1]), F[2], col(ins[1] * F[3])], 1)
        A = M - h * h * K - h * D
        b = h * Fv + ((M - h * D.transpose(1, 2)) @ V[:, :, None])[:, :, 0]
        sg = torch.where(k == 0, 1.0, -1.0).to(du)[:, None]
        dof = torch.cat([5 * i0[:, None] + torch.arange(3, device=i0.device), (5 * i0 + 3 + k)[:, None],
                         5 * i1[:, None] + torch.arange(3, device=i0.device), (5 * i1 + 3 + k)[:, None]], 1)
        node = torch.cat([i0, i1])
        slot = torch.cat([2 * i0 + k, 2 * i1 + k])
        own = lambda X: torch.cat([X[:, 3, 3], X[:, 7, 7]])  # noqa: E731
        fric = dict(FE=(slot, torch.cat([Fv[:, 3], Fv[:, 7]])), KEE=(slot, own(K)), DEE=(slot, own(D)),
                    CL=(node, torch.cat([sg * f, -sg * f])),
                    CLE=(slot, torch.cat([sg * col(ins[0]) * xe_s, sg * col(ins[1]) * xe_s])))
        return dof, A, b, fric

    @staticmethod
    def bend_terms(x2, x0, x1, du, kb):
        col = lambda s: s[:, None]  # noqa: E731
        a1, a2 = x1 - x0, x2 - x0
        l1, l2 = a1.norm(dim=1), a2.norm(dim=1)
        d1, d2 = a1 / col(l1), a2 / col(l2)
        eye = torch.eye(3, dtype=x0.dtype, device=x0.device)
        out = lambda a, b: a[:, :, None] * b[:, None, :]  # noqa: E731
        P1, P2 = eye - out(d1, d1), eye - out(d2, d2)
        c = -(d1 * d2).sum(1)
        c = torch.clamp(c, -1.0, 1.0)
        th, s = torch.acos(c), torch.sqrt((1 - c) * (1 + c))
        on = s != 0
        s = torch.where(on, s, torch.ones_like(s))
        kb = torch.where(on, kb, torch.zeros_like(kb))
        a, b = (P1 @ d2[:, :, None])[:, :, 0], (P2 @ d1[:, :, None])[:, :, 0]
        m = lambda z: z[:, None, None]  # noqa: E731
        F1, F2 = col(-2 * kb * th / (l1 * du * s)) * a, col(-2 * kb * th / (l2 * du * s)) * b
        cs2 = c / (s * s)
        diag = lambda k, v, d, P: m(k) * (m(th) * (out(v, d) + m(cs2) * out(v, v) + m(c) * P + out(d, v))  # noqa: E731
                                          - m(1 / s) * out(v, v))
        L11 = diag(2 * kb / (l1 * l1 * du * s), a, d1, P1)
        L22 = diag(2 * kb / (l2 * l2 * du * s), b, d2, P2)
        k12 = -2 * kb / (l1 * l2 * du * s)
        mix = lambda v, d, P, Q: m(k12) * ((m(th) * (P - m(cs2) * out(v, d)) + m(1 / s) * out(v, d)) @ Q)  # noqa: E731
        return F1, F2, L11, mix(a, d1, P1, P2), mix(b, d2, P2, P1), L22, -F1 / col(du), -F2 / col(du), th

    def bends(self, st, par, h, nrm):
        n2, n0, n1, k, ln = self.bend.T
        kb, c = (par["B"] * self.area)[ln], self.cloth[n0]
        x = st["LPos"]
        pick = lambda a, i: torch.where(k == 0, a[i, 0], a[i, 1])  # noqa: E731
        du = pick(st["EPos"], n1) - pick(st["EPos"], n2)
        F1, F2, L11, L12, L21, L22, g1, g2, th = self.bend_terms(x[n2], x[n0], x[n1], du, kb)
        ee, fu = -2 * kb * th * th / du ** 3, -kb * th / du ** 2
        ins = {i: self.inside[n].to(x) for i, n in ((2, n2), (0, n0), (1, n1))}
        at = {2: 0, 0: 4, 1: 8}
        L01, L02, L20, L10 = -(L11 + L21), -(L12 + L22), -(L21 + L22), -(L11 + L12)
        blocks = [[None] * 3 for _ in range(3)]
        for (i, j), B in {(2, 2): L22, (1, 1): L11, (0, 0): -(L10 + L20), (0, 1): L01, (0, 2): L02, (2, 0): L20,
                          (1, 0): L10, (2, 1): L21, (1, 2): L12}.items():
            blocks[at[i] // 4][at[j] // 4] = torch.nn.functional.pad(B.transpose(1, 2), (0, 1, 0, 1))
        K = torch.cat([torch.cat(r, 2) for r in blocks], 1)

        def put(i, j, row, column, value):
            E = torch.zeros(12, 12, dtype=x.dtype, device=x.device)
            out = 0
            for r in range(3):
                E.zero_()
                if column:
                    E[at[i] + r, at[j] + 3] = 1.0
                if row:
                    E[at[j] + 3, at[i] + r] = 1.0
                out = out + value[:, r, None, None] * E.clone()
            return out
        q = g1 + g2
        w2, w1 = ins[2][:, None], ins[1][:, None]
        K = K + put(2, 2, True, True, -w2 * g2) + put(1, 1, True, True, w1 * g1)
        m02, m01 = (ins[0] * ins[2])[:, None], (ins[0] * ins[1])[:, None]
        K = K + put(0, 2, False, True, m02 * q) + put(0, 1, False, True, -m01 * q)
        # row e of the middle crossing and the columns x of n2; row e of n1 and the columns x of the middle
        K = K + put(2, 0, True, False, m02 * q) + put(0, 1, True, False, -m01 * q)
        D = torch.zeros(12, 12, dtype=x.dtype, device=x.device)
        D[3, 3] = 1.0
        E = torch.zeros_like(D)
        E[11, 11] = 1.0
        K = K + (ins[2] * ee)[:, None, None] * D + (ins[1] * ee)[:, None, None] * E
        z = torch.zeros_like(du)[:, None]
        F = torch.cat([F2, (ins[2] * fu)[:, None], -(F1 + F2), z, F1, -(ins[1] * fu)[:, None]], 1)
        R_ = torch.where(k == 0, -1.0, 1.0).to(x)[:, None] * self.R[c][:, None]
        uv0 = pick(self.uv0, n1) - pick(self.uv0, n2)
        p = [x[n] + R_ * nrm[n] for n in (n2, n0, n1)]
        c1, c2, _, _, _, _, h1, h2, _ = self.bend_terms(*p, uv0, kb)
        sg = torch.where(k == 0, 1.0, -1.0).to(x)[:, None]
        slot = torch.cat([2 * n2 + k, 2 * n1 + k])
        fric = dict(FE=(slot, torch.cat([ins[2] * fu, -ins[1] * fu])), KEE=(slot, torch.cat([ins[2] * ee, ins[1] * ee])),
                    CL=(torch.cat([n2, n0, n1]), torch.cat([sg * c2, -sg * (c1 + c2), sg * c1])),
                    CLE=(slot, torch.cat([-sg * w2 * h2, sg * w1 * h1])))
        a3 = torch.arange(3, device=n0.device)
        dof = torch.cat([torch.cat([5 * n[:, None] + a3, (5 * n + 3 + k)[:, None]], 1) for n in (n2, n0, n1)], 1)
        return dof, -h * h * K, h * F, fric

    def shears(self, st, par, h, comp):
        n0, n1, n3 = self.shear.T
        c = self.cloth[n0]
        x = st["LPos"]
        Lc, R_, S, comp = self.L[c], self.R[c], par["S"][c], comp[n0]
        col, m = lambda s: s[:, None], lambda s: s[:, None, None]  # noqa: E731
        out = lambda a, b: a[:, :, None] * b[:, None, :]  # noqa: E731
        b1, b3 = x[n1] - x[n0], x[n3] - x[n0]
        l1, l3 = b1.norm(dim=1), b3.norm(dim=1)
        d1, d3 = b1 / col(l1), b3 / col(l3)
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        P1, P3 = eye - out(d1, d1), eye - out(d3, d3)
        co = (d1 * d3).sum(1)
        phi, s = torch.acos(co), torch.sqrt((1 - co) * (1 + co))
        a3, a1 = (P1 @ d3[:, :, None])[:, :, 0], (P3 @ d1[:, :, None])[:, :, 0]
        cs2 = co / (s * s)
        jam = (self.flip[n0] != self.flip[n1]) & (self.flip[n0] != self.flip[n3])
        # free shear
        kx, ph = (comp + 1) * S * R_ * R_ * PI, phi - PI / 2
        F1, F3 = col(kx * Lc * ph / (l1 * s)) * a3, col(kx * Lc * ph / (l3 * s)) * a1
        diag = lambda l, v, d, P: m(kx * Lc / (l * l * s)) * (m(ph) * (m(cs2) * out(v, v) - out(v, d) - out(d, v)  # noqa: E731
                                                              - m(co) * P) - m(1 / s) * out(v, v))
        mix = kx * Lc / (l1 * l3 * s) * ph * (cs2 - 1 / s)
        free = [F1, F3, diag(l1, a3, d1, P1), m(mix) * out(a3, a1), m(mix) * out(a1, a3), diag(l3, a1, d3, P3)]
        # shear lock
        pb, pl, sig = PI / 2, 2 * torch.asin(R_ / Lc), 0.6
        p1, p3 = -a3 / col(l1 * s), -a1 / col(l3 * s)
        sh, ch = torch.sqrt(0.5 * (1 - co)), torch.sqrt(0.5 * (1 + co))
        gam, kap = (Lc * math.sqrt(2.0) - 2 * Lc * sh) / R_, -Lc / R_ * ch
        A_, B_ = phi - pl, phi - pb
        phs, sgm, omg = phi * A_ * B_, A_ * B_ + phi * B_ + phi * A_, 2 * (A_ + B_ + phi)
        num, den = pb ** 5 * A_, phs * phs + pb ** 4 * sig * sig
        cf = torch.tanh(num / den)
        tau = pb ** 5 * den - num * 2 * phs * sgm
        mu = tau / den ** 2
        g3, base = gam ** 3, 0.5 * (comp + 1) * S * PI * R_ * R_
        kx = base * ((1 + g3) + (1 - g3) * cf)
        t0 = base * (1 - g3)
        t1 = base * (3 * gam ** 2 * kap * (1 - cf) - (1 - g3) * cf * cf * mu)
        F1 = -0.5 * (col(t0) + col(t1) * p1) * col(Lc * B_ * B_) + col(kx * Lc * B_ / (l1 * s)) * a3
        F3 = -0.5 * (col(t0) + col(t1) * p3) * col(Lc * B_ * B_) + col(kx * Lc * B_ / (l3 * s)) * a1
        e3 = (P3 @ d3[:, :, None])[:, :, 0]
        kO = 6 * gam * kap * kap * (1 - cf) - 6 * gam ** 2 * kap * (1 - cf * cf) * mu
        kG = 3 * gam ** 2 * (1 - cf)
        cq = -2 * cf * (1 - cf * cf) * mu * mu
        X4 = 4 * tau * den * phs * sgm / den ** 4
        hb, LB = 0.5 * Lc * B_ * B_ * 0.5 * (comp + 1) * S * R_ * R_, Lc * B_
        one, row = torch.ones_like(eye), lambda v: v[:, None, :]  # noqa: E731
        q1, q3 = 1 / (l1 * l1 * s), 1 / (l3 * l3 * s)
        q13 = 1 / (l1 * l3 * s)
        hs = 0.5 * Lc / R_ * sh

        def block(pxx, O, Ob, Rg, fo, same, mid):
            """one block of the lock's Hessian from phi_xx, phi_x phi_x^T and its mirror, the half-angle's
            remainder and the constant-kx part"""
            if same:
                psx, nx = m(sgm) * pxx + m(omg) * O, 0
            else:
                psx = m(sgm) * pxx + m(omg) * (0.5 * (O + Ob) if mid else O)
                nx = m(2 * phs * pb ** 5 * sgm) * (O - Ob)
            nx = nx + m(pb ** 5 * den) * pxx - m(2 * num * sgm * sgm) * O - m(2 * num * phs) * psx
            cfx = nx / m(den ** 2) - m(X4) * O
            cdd = m(cq) * (O if same else Ob) + (one - m(cf * cf) * cfx if same else m(1 - cf * cf) * cfx)
            kxx = m(kO) * O + m(kG) * (m(kap) * pxx + Rg) + m(1 - g3) * cdd
            return -m(hb) * kxx - m(2 * LB * t1) * O + fo

        A3, S1 = out(a3, a3), out(a3, d1) + out(d1, a3)
        O = m(q1 / s) * A3
        J11 = block(m(q1) * (S1 - m(cs2) * A3 + m(co) * P1), O, O, m(hs * q1 / s) * A3,
                    m(kx * Lc * q1) * (m(B_ * cs2 - 1 / s) * A3 - m(B_) * (S1 + m(co) * P1)), True, False)
        J11 = J11 - m(2 * LB * t0) * row(p1)
        A1, S3 = out(a1, a1), out(a1, d3) + out(d3, a1)
        O = m(q3 / s) * A1
        J33 = block(m(q3) * (S3 - m(cs2) * A1 + m(co) * P3), O, O, m(hs * q3 / s) * A1,
                    m(kx * Lc * q3) * (m(B_ * cs2 - 1 / s) * A1 - m(B_) * (S3 + m(co) * P3)), True, False)
        J33 = J33 - m(2 * LB * t0) * row(p3)
        M13, A13, A31 = P1 @ P3, out(a3, a1), out(a1, a3)
        kq = B_ * cs2 - 1 / s
        J13 = block(-m(q13) * (m(cs2) * A13 + M13), m(q13 / s) * A13, m(q13 / s) * A31, m(hs * q13 / s) * A13,
                    m(kx * Lc * q13) * (m(kq) * A13 + m(B_) * M13), False, True)
        J13 = J13 - m(LB * t0) * (row(p3) + p1[:, :, None])
        J31 = block(-m(q13) * (m(cs2) * out(a1, e3) + M13.transpose(1, 2)), m(q13 / s) * A31, m(q13 / s) * A13,
                    m(hs * q13 / s) * A31, m(kx * Lc * q13) * (m(kq) * A31 + m(B_) * M13.transpose(1, 2)), False, False)
        J31 = J31 - m(LB * t0) * (row(p1) + p3[:, :, None])
        lock = [F1, F3, J11, J13, J31, J33]
        F1, F3, J11, J13, J31, J33 = (torch.where(jam.view(-1, *([1] * (a.dim() - 1))), a, b) for a, b in zip(lock, free))
        J10, J30 = -(J11 + J13), -(J31 + J33)
        rows = [[-(J10 + J30), -(J11 + J31), -(J13 + J33)], [J10, J11, J13], [J30, J31, J33]]
        K = torch.cat([torch.cat([B.transpose(1, 2) for B in r], 2) for r in rows], 1)
        F = torch.cat([-(F1 + F3), F1, F3], 1)
        a3_ = torch.arange(3, device=n0.device)
        return torch.cat([5 * n[:, None] + a3_ for n in (n0, n1, n3)], 1), -h * h * K, h * F

    def winds(self, st, h):
        i = self.face
        p, v = st["LPos"][i], st["LVel"][i]
        c = self.cloth[i[:, 0]]
        n = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
        nc = n.norm(dim=1, keepdim=True)
        n, area = n / nc, 0.5 * nc
        rel = self.wind[c] - v.mean(1)
        vn = (n * rel).sum(1, keepdim=True)
        f = self.rho_air[c][:, None] * area * vn.abs() * vn * n + self.drag[c][:, None] * area * (rel - vn * n)
        return i, (h * f / 3)[:, None, :].expand(-1, 3, -1)

    def system(self, st, par, h, ext=None):
        """[(unknowns, matrices)] of the elements, b, and the slide indicator."""
        n = self.n
        nrm = self.normals(st["LPos"])
        ed, eA, eb, ef = self.edges(st, par, h)
        bd, bA, bb, bf = self.bends(st, par, h, nrm)
        tot = lambda k, size: sum(torch.zeros(size, *f[k][1].shape[1:], dtype=eb.dtype, device=eb.device).index_add(  # noqa: E731
            0, *f[k]) for f in (ef, bf) if k in f)
        FE, KEE, DEE, CLE = tot("FE", 2 * n).view(n, 2), tot("KEE", 2 * n).view(n, 2), tot("DEE", 2 * n).view(n, 2), \
            tot("CLE", 2 * n).view(n, 2, 3)
        inside = self.inside.to(eb)
        comp = torch.relu(0.5 * (nrm * tot("CL", n)).sum(1)) * inside
        cee = 0.5 * (nrm[:, None, :] * CLE).sum(2)
        mu, kf, df = par["mu"][self.cloth][:, None], self.kf[self.cloth][:, None], self.df[self.cloth][:, None]
        uvm, cm = st["EPos"] - st["EPosBar"], comp[:, None]
        lim = cm * mu
        slide = 1 / (1 + torch.exp(-1e4 * (FE.abs() - lim)))
        t, tl, tq = torch.tanh(10 * uvm), torch.tanh(10 * (lim - FE)), torch.tanh(10 * lim - FE)
        ud = st["EVel"]
        force = -0.5 * (kf * uvm - t * cm * mu) * tl + 0.5 * (kf * uvm + t * cm * mu) - df * ud
        pos = -0.5 * (kf - (1 - t * t) * mu * cm - t * mu * cee) * tl - 0.5 * (kf * uvm - t * mu * cm) * (1 - tl * tl) * (
            KEE - mu * cee) - 0.5 * (kf + (1 - t * t) * mu * cm + t * mu * cee)
        vel = -0.5 * (kf * uvm - t * mu * cm) * (1 - tq * tq) * DEE - df
        sd, sA, sb = self.shears(st, par, h, comp)
        fi, fb = self.winds(st, h)
        fx = self.fixed.to(eb)[:, None]
        kh = self.kh[self.cloth][:, None]
        one = inside[:, None]
        bx = torch.zeros(n, 3, dtype=eb.dtype, device=eb.device).index_add(0, fi.reshape(-1), fb.reshape(-1, 3))
        bx = bx - h * fx * kh * (st["LPos"] - st["LPosFix"])
        be = one * h * (force - vel * ud)
        diag = torch.cat([(h * h * fx * kh).expand(-1, 3), one * (-h * h * pos - h * vel) + (1 - one)], 1)
        b = torch.cat([bx, be], 1)
        if ext is not None:
            b = b + h * torch.cat([ext[:, :3], one * ext[:, 3:]], 1)
        b = b.reshape(-1)
        for d, v in ((ed, eb), (bd, bb), (sd, sb)):
            b = b.index_add(0, d.reshape(-1), v.reshape(-1))
        return [(ed, eA), (bd, bA), (sd, sA)], diag.reshape(-1), b, slide

    @staticmethod
    def apply(els, diag, q, trans=False):
        y = diag * q
        for d, A in els:
            v = ((A.transpose(1, 2) if trans else A) @ q[d][:, :, None])[:, :, 0]
            y = y.index_add(0, d.reshape(-1), v.reshape(-1))
        return y

    def solve(self, els, diag, b, trans=False):
        """Conjugate gradients, started again from the true residual until that stops falling."""
        dg = diag.clone()
        for d, A in els:
            dg = dg.index_add(0, d.reshape(-1), torch.diagonal(A, dim1=1, dim2=2).reshape(-1))
        x, best, r = torch.zeros_like(b), math.inf, b
        for _ in range(6):
            z = r / dg
            p, rz, y, r0 = z, r @ z, torch.zeros_like(b), r
            for _ in range(200):
                q = self.apply(els, diag, p, trans)
                a = rz / (p @ q)
                y, r0 = y + a * p, r0 - a * q
                z = r0 / dg
                new = r0 @ z
                if float(new) <= 1e-24 * float((r @ (r / dg))) or float(new) == 0.0:
                    break
                p, rz = z + (new / rz) * p, new
            r1 = b - self.apply(els, diag, x + y, trans)
            size = float((r1 / dg.abs().sqrt()).norm())
            if not size < 0.5 * best:
                break
            x, r, best = x + y, r1, size
        return x

    def update(self, st, q, slide, h):
        q = q.view(self.n, 5)
        one = self.inside.to(q)[:, None]
        x = st["LPos"] + h * q[:, :3]
        return dict(LPos=x, LPosFix=torch.where(self.fixed[:, None], st["LPosFix"], x), LVel=q[:, :3],
                    EPos=st["EPos"] + one * h * q[:, 3:], EPosBar=st["EPosBar"] + one * h * slide * q[:, 3:],
                    EVel=torch.where(self.inside[:, None], q[:, 3:], st["EVel"]))


def exact(case, seed):
    if case["kind"] == "respond":
        return None  # rounds of detection and projection: a sequence of choices, no formula to evaluate
    d = _inputs(case, seed)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    specs = d["specs"]
    if case["kind"] == "simstep":  # Cloth takes yarns, not lines: one for all, or two by parity
        p = specs[0]
        y = [p["warp"][0], p["warp"][1 if case["blend"] else 0]]
        for k in ("warp", "weft"):
            p[k] = np.array([y[i % 2] for i in range(len(p[k]))])
    m = _Model(specs, device)
    t = lambda a: None if a is None else torch.as_tensor(a, device=device)  # noqa: E731
    st, ext, h = {k: t(v) for k, v in d["state"].items()}, t(d["ext"]), case["h"]
    els, diag, b, slide = m.system(st, m.par, h, ext)
    q = m.solve(els, diag, b)
    if case["kind"] == "system":
        y = m.apply(els, diag, t(d["y"]).reshape(-1)).view(m.n, 5)
        return dict(x=q.view(m.n, 5), y=y, normals=m.normals(st["LPos"]), ok=None)
    if case["kind"] in ("simstep", "step", "learned"):
        return dict(m.update(st, q, slide, h), ok=None)
    names = ("LPos", "LVel", "EPos", "EVel", "EPosBar")

    def residual(state, par, force=None):
        e, g, rhs, sl = m.system(dict(state, LPosFix=st["LPosFix"]), par, h, force)
        return m.apply(e, g, q) - rhs, sl

    if case["kind"] == "adjoint":
        g = {k: t(v) for k, v in d["grad"].items()}
        one, qe = m.inside.to(q)[:, None], q.view(m.n, 5)[:, 3:]
        qb = torch.cat([g["LVel"] + h * g["LPos"], one * (g["EVel"] + h * g["EPos"] + h * slide * g["EPosBar"])], 1)
        lam = m.solve(els, diag, qb.reshape(-1), trans=True)
        del els
        leaf = {k: st[k].clone().requires_grad_(True) for k in names}
        par = {k: v.clone().requires_grad_(True) for k, v in m.par.items()}
        r, sl = residual(leaf, par, ext)
        loss = -(lam @ r) + (one * g["EPosBar"] * qe * h * sl).sum()
        order = [leaf[k] for k in names] + list(par.values())
        grads = torch.autograd.grad(loss, order, allow_unused=True)
        grads = [torch.zeros_like(a) if v is None else v for a, v in zip(order, grads)]
        out = dict(zip(names, grads))
        out["LPos"] = out["LPos"] + g["LPos"]
        out["EPos"] = out["EPos"] + g["EPos"]
        out["EPosBar"] = out["EPosBar"] + g["EPosBar"]
        out["EVel"] = out["EVel"] + (1 - one) * g["EVel"]
        force = h * torch.cat([lam.view(m.n, 5)[:, :3], one * lam.view(m.n, 5)[:, 3:]], 1) if case["ext"] else None
        return dict(state=out, params=dict(zip(par, grads[5:])), ext=force)
    # forward sensitivities: A dq = db - dA q along each direction
    line, cloth = _seeds(case["width"], case["length"])
    nl = case["width"] + case["length"]
    one = m.inside.to(q)[:, None]
    tan = {k: torch.zeros(4, 2 * m.n, st[k].shape[1], dtype=torch.float64, device=device) for k in names}
    src = dict(LPos="dlpos", LVel="dlvel", EPos="depos", EVel="devel", EPosBar="deposbar")
    for c in range(2):
        for k in range(4):
            ds = {a: t(d["tan"][src[a]][k, c * m.n:(c + 1) * m.n]) for a in names}
            dp = dict(zip(("rho", "Y", "B"), (t(line[j, k, c * nl:(c + 1) * nl]) for j in range(3))))
            dp.update(S=t(cloth[0, k, c:c + 1]), mu=t(cloth[1, k, c:c + 1]))
            _, (dr, dsl) = torch.func.jvp(residual, ({a: st[a] for a in names}, m.par), (ds, dp))
            dq = m.solve(els, diag, -dr).view(m.n, 5)
            qe = q.view(m.n, 5)[:, 3:]
            rows = slice(c * m.n, (c + 1) * m.n)
            tan["LPos"][k, rows] = ds["LPos"] + h * dq[:, :3]
            tan["LVel"][k, rows] = dq[:, :3]
            tan["EPos"][k, rows] = ds["EPos"] + one * h * dq[:, 3:]
            tan["EVel"][k, rows] = torch.where(m.inside[:, None], dq[:, 3:], ds["EVel"])
            tan["EPosBar"][k, rows] = ds["EPosBar"] + one * h * (dsl * qe + slide * dq[:, 3:])
    new = {k: torch.cat([v, v]) for k, v in m.update(st, q, slide, h).items()}
    return dict(state=new, tangents=tan, ok=None)
