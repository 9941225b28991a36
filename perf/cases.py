"""The workloads whose speed matters to a user of this package, as cases.

    listed()            the cases
    draw(rng)           another case of the same ranges
    prepare(case, seed) what a program holds before the call, on the GPU
    run(state)          one pass through the public entry points, its outputs
    work(case)          bytes and flops one pass cannot do without
    exact(case, seed)   run's outputs in 64 bits, by plain torch operations

A program loads a scene once and then steps it frame after frame, so a case's
bodies (sizes, hulls, masses) are fixed by the case and its state (poses and
velocities) comes from the seed: seeded velocities on the generated layout,
then untimed frames until the bodies lie in contact.  Every pass starts from
that state, as an episode or a rollout does, so all passes do the same work.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from seevr_b200 import (BROADPHASE_LBVH, BROADPHASE_N2, FLAG_CUDA_GRAPH, FLAG_SKIP_RENDER_VERTS,
                        SOLVER_COLORED, SOLVER_WAVEFRONT, Caps, Data, Physics, make_params)
from seevr_b200.bvh import BVH
from seevr_b200.grad import rollout
from seevr_b200.raytrace import Raytracer

DT, SUBSTEPS, G = 1.0 / 60.0, 10, (0.0, -9.81, 0.0)
STATE = (("body_pos", 3), ("body_quat", 4), ("body_vel", 3), ("body_omega", 3))
KEYS = ("pos", "quat", "vel", "omega")
BOXES = ("aabb_min", "aabb_max")


def listed():
    return [
        # A handful of bodies stepped once per display frame by an
        # interactive program, with the reference's settings: pure latency.
        {"name": "drop_in_24", "kind": "drop_in", "bodies": 24, "pgs": 4, "graph": False,
         "render": True, "settle": 90},
        # The reference's own kind of scene (512 bodies on a ground plane, 120
        # frames), at the solver quality its README names, frame graph replayed.
        {"name": "drop_in_512", "kind": "drop_in", "bodies": 512, "pgs": 30, "graph": True,
         "render": True, "settle": 90},
        # One scene too large for a solver block: islands of a pile.
        {"name": "drop_in_2600", "kind": "drop_in", "bodies": 2600, "pgs": 30, "graph": False,
         "render": False, "settle": 90},
        # Environments stepped together by a learning loop: many small scenes,
        # the handle's default launch shapes, frames queued without waiting.
        {"name": "batch_100", "kind": "batch", "scenes": 100, "max_bodies": 96, "pgs": 10,
         "groups": 1, "frames": 2, "settle": 75},
        # The headline workload's scenes (8 to 512 bodies each) at the size of
        # one simulator's share of a node, default shapes, device resident.
        {"name": "batch_1024", "kind": "batch", "scenes": 1024, "max_bodies": 512, "pgs": 30,
         "groups": 1, "frames": 1, "settle": 90},
        # The same through the call that takes a frame's state from pinned host
        # memory and returns it there, with the shapes the autotuner picks.
        {"name": "batch_io_1024", "kind": "batch_io", "scenes": 1024, "max_bodies": 512, "pgs": 30,
         "groups": 8, "settle": 90},
        # One large scene of boxes, spheres and convex hulls: LBVH broadphase.
        {"name": "large_32768", "kind": "large", "bodies": 32768, "pgs": 30, "settle": 30},
        # Stacks with persistent contacts, solved in colour order by islands.
        {"name": "towers_1024x256", "kind": "towers", "towers": 1024, "height": 256, "pgs": 30},
        # Gradient of a short horizon for a few scenes (a controller's inner loop).
        {"name": "rollout_6x20", "kind": "rollout", "scenes": 6, "bodies": 20, "pgs": 10,
         "frames": 1, "settle": 75},
        # Gradients of a batch of rollouts, forward and backward.
        {"name": "rollout_1024x64", "kind": "rollout", "scenes": 1024, "bodies": 64, "pgs": 30,
         "frames": 2, "settle": 75},
        # The triangle BVH of a scene's render mesh, rebuilt every frame.
        {"name": "bvh_512", "kind": "bvh", "bodies": 512, "settle": 60},
        # A path-traced frame of that scene.
        {"name": "render_640x480", "kind": "render", "bodies": 512, "width": 640, "height": 480,
         "settle": 60},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["drop_in", "drop_in", "batch", "batch", "batch_io", "large", "towers",
                       "rollout", "rollout", "bvh", "render"])
    c = {"kind": kind}
    if kind == "drop_in":
        c.update(bodies=_log(rng, 8, 2600), pgs=rng.choice([4, 10, 30]),
                 graph=rng.random() < 0.5, render=rng.random() < 0.5, settle=90)
    elif kind in ("batch", "batch_io"):
        c.update(scenes=_log(rng, 3, 900), max_bodies=_log(rng, 12, 512),
                 pgs=rng.choice([4, 10, 30]),
                 groups=rng.choice([1, 1, 4]) if kind == "batch" else rng.choice([4, 8]), settle=75)
        if kind == "batch":
            c["frames"] = rng.choice([1, 2])
    elif kind == "large":
        c.update(bodies=_log(rng, 3000, 32000), pgs=rng.choice([4, 30]), settle=30)
    elif kind == "towers":
        c.update(towers=_log(rng, 40, 1000), height=rng.randint(20, 250), pgs=rng.choice([10, 30]))
    elif kind == "rollout":
        c.update(scenes=_log(rng, 2, 1000), bodies=rng.randint(9, 64), pgs=rng.choice([4, 10, 30]),
                 frames=1, settle=75)
    elif kind == "bvh":
        c.update(bodies=_log(rng, 30, 2000), settle=30)
    else:
        w = _log(rng, 60, 620)
        c.update(bodies=_log(rng, 30, 500), width=w, height=max(40, int(w * 0.72)), settle=60)
    return c


# ---- scenes -------------------------------------------------------------------
def _side(bodies):
    """Half the side of the square a pile is dropped on: 10 m for 512 bodies
    (the reference scene), the same density of bodies for more and fewer."""
    return max(5.0 * math.sqrt(bodies / 512.0), 1.2)


def _height(bodies):
    """Metres a pile is dropped from: 20 (the reference scene), less for
    fewer bodies, so that they too have landed when the pass begins."""
    return 20.0 * min(1.0, (bodies / 512.0) ** (1.0 / 3.0))


@functools.lru_cache(maxsize=2)
def _scene(key):
    """The case's bodies on the GPU, loaded once."""
    c = dict(key)
    kind, pairs = c["kind"], 8.0
    if kind in ("drop_in", "bvh", "render"):
        n, s = c["bodies"], _side(c["bodies"])
        d = Data.pile(seed=n, n_boxes=(n + 1) // 2, n_spheres=n // 2, lo=(-s, 0.6, -s),
                      hi=(s, 0.6 + _height(n), s))
    elif kind in ("batch", "batch_io"):
        d = Data.batch(num_scenes=c["scenes"], min_bodies=8, max_bodies=c["max_bodies"],
                       seed_base=c["scenes"])
    elif kind == "large":
        d = Data.large(seed=0, n_bodies=c["bodies"])
    elif kind == "towers":
        d, pairs = Data.towers(seed=0, towers=c["towers"], height=c["height"], spacing=2.0,
                               overlap=0.002), 4.0
    else:
        d = Data.rollout(num_scenes=c["scenes"], bodies=c["bodies"], seed_base=1 << 32)
    return d, d.upload("cuda", Caps.for_data(d, pairs_per_body=pairs, contacts_per_body=4.0))


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def _params(case):
    kind = case["kind"]
    flags = 0
    if case.get("graph", kind not in ("bvh", "render")):
        flags |= FLAG_CUDA_GRAPH
    if not case.get("render", kind in ("batch_io", "bvh", "render")):
        flags |= FLAG_SKIP_RENDER_VERTS
    return make_params(pgs_iterations=case.get("pgs", 10),
                       solver=SOLVER_COLORED if kind == "towers" else SOLVER_WAVEFRONT,
                       broadphase=BROADPHASE_LBVH if kind in ("large", "towers") else BROADPHASE_N2,
                       flags=flags,
                       bundle_bodies=case["bodies"] + 1 if kind == "rollout" else 0)


def _start(case, seed):
    """The scene's buffers and handle, and the state every pass starts from."""
    d, master = _scene(_key(case))
    buf = dataclasses.replace(master, tensors={k: v.clone() for k, v in master.tensors.items()})
    nb, t = buf.num_bodies, buf.tensors
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dynamic = (t["body_inv_mass"][:nb] > 0).to(torch.float32)[:, None]
    size = 0.02 if case["kind"] == "towers" else 1.0  # towers stand: only stirred
    for name in ("body_vel", "body_omega"):
        v = torch.randn(nb, 3, generator=gen, device="cuda") * size * dynamic
        t[name][: 3 * nb].copy_(v.reshape(-1))
    ph = Physics(buf, _params(case))
    if case.get("groups", 1) > 1:
        ph.set_tuning(scene_groups=case["groups"])
    torch.cuda.synchronize()
    if case.get("settle"):
        ph.step_async(nb, buf.num_vertices, buf.num_hull_verts, SUBSTEPS, DT, G,
                      frames=case["settle"], stream=torch.cuda.current_stream())
        torch.cuda.synchronize()
    init = {k: t[n][: nb * c].clone() for k, (n, c) in zip(KEYS, STATE)}
    return d, buf, ph, init


def prepare(case, seed):
    kind = case["kind"]
    d, buf, ph, init = _start(case, seed)
    s = {"kind": kind, "buf": buf, "ph": ph, "init": init, "nb": buf.num_bodies,
         "nv": buf.num_vertices, "nhv": buf.num_hull_verts, "frames": case.get("frames", 1),
         "live": {k: buf.tensors[n][: buf.num_bodies * c] for k, (n, c) in zip(KEYS, STATE)},
         "boxes": {k: buf.tensors["body_" + k][: buf.num_bodies * 3] for k in BOXES}}
    if kind == "batch_io":
        s["in"] = {k: v.cpu().pin_memory() for k, v in init.items()}
        s["out"] = {k: torch.empty_like(v).pin_memory() for k, v in s["in"].items()}
    elif kind == "rollout":
        nb = buf.num_bodies
        off = torch.as_tensor(buf.scene_body_offset[:-1].astype(np.int64), device="cuda")
        s["first"] = off + 1  # a scene's body 0 is the ground
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        s["target"] = torch.rand(len(off), 3, generator=gen, device="cuda") * 2.0 - 1.0
        s["mu"] = buf.tensors["geom_friction"][:nb].clone()
        s["init"] = {k: v.reshape(nb, c) for (k, v), (_, c) in zip(init.items(), STATE)}
    elif kind in ("bvh", "render"):
        ntri = d.num_triangles
        idx = torch.from_numpy(d.array("indices").reshape(-1).view(np.int32)).cuda()
        s["bvh"] = BVH(buf.tensors["vertices"][: 3 * buf.num_vertices].clone(), idx)
        s["ntri"] = ntri
        if kind == "render":
            s["bvh"].build(ntri)
            s["rt"] = Raytracer(d, s["bvh"], case["width"], case["height"])
            cam = np.array([[0.0, 12.0, 24.0], [0.0, -0.35, -1.0], [1.0, 0.0, 0.0],
                            [0.0, 1.0, -0.35]])
            cam[1:] /= np.linalg.norm(cam[1:], axis=1, keepdims=True)
            s["cam"] = cam.tolist()
    return s


# ---- one pass -------------------------------------------------------------------
def _reset(s):
    for k, v in s["live"].items():
        v.copy_(s["init"][k])


def run(s):
    kind, ph = s["kind"], s["ph"]
    if kind == "drop_in":  # Physics.step waits, then Physics.readCounters
        _reset(s)
        torch.cuda.current_stream().synchronize()  # the handle steps on its own stream
        ph.step(s["nb"], s["nv"], s["nhv"], SUBSTEPS, DT, G)
        return {**s["live"], **s["boxes"], "counters": list(ph.read_counters())}
    if kind in ("batch", "large", "towers"):  # queued on the caller's stream, not waited for
        _reset(s)
        ph.step_async(s["nb"], s["nv"], s["nhv"], SUBSTEPS, DT, G, frames=s["frames"],
                      stream=torch.cuda.current_stream())
        return {**s["live"], **s["boxes"], "counters": s["buf"].tensors["counters"][:2]}
    if kind == "batch_io":  # host state in, host state out
        ph.step_io(s["nb"], s["nv"], s["nhv"], SUBSTEPS, DT, G, inputs=s["in"], outputs=s["out"])
        return s["out"]
    if kind == "rollout":
        x = s["init"]
        vel, omega, mu = (v.clone().requires_grad_() for v in (x["vel"], x["omega"], s["mu"]))
        out = rollout(ph, x["pos"], x["quat"], vel, omega, mu, frames=s["frames"],
                      substeps=SUBSTEPS, dt=DT, gravity=G)
        loss = ((out[0][s["first"]] - s["target"]) ** 2).sum()
        loss.backward()
        return {**{k: v.detach().reshape(-1) for k, v in zip(KEYS, out)}, "g_vel": vel.grad,
                "g_omega": omega.grad, "g_mu": mu.grad}
    if kind == "bvh":
        s["bvh"].build(s["ntri"])
        return {k: s["bvh"][k] for k in ("centroids", "scene_bounds", "morton", "sort_indices",
                                         "node_min", "node_max", "left", "right", "count",
                                         "parent", "prim_indices")}
    s["rt"].reset_accumulation()  # the same frame number (the random seed) every pass
    return s["rt"].render(*s["cam"], s["ntri"])


# ---- what a pass cannot do without -----------------------------------------------
def work(case):
    """Bytes and flops from the case's sizes.  A substep reads and writes each
    body's state (324 B), reads each hull vertex (12 B), reads a pair's shapes
    (72 B) and a contact's data (84 B); pairs and contacts per body as settled
    piles of this density hold them.  A support call is about 200 flops and
    MPR makes about 6 per pair; a contact update is about 420 flops."""
    kind = case["kind"]
    if kind in ("bvh", "render"):
        tri = 128 * case["bodies"] * 2 + 12 * case["bodies"] // 2
        build = {"bytes": tri * (12 + 36 + 12 + 16 + 2 * (24 + 16)), "flops": tri * 60}
        if kind == "bvh":
            return build
        rays = case["width"] * case["height"] * 16 * 2.0  # two segments per path
        return {"bytes": 16.0 * case["width"] * case["height"] + tri * 124.0,
                "flops": rays * (2 * math.log2(tri) * 20 + 4 * 50)}
    if kind in ("batch", "batch_io"):
        m = case["max_bodies"]
        bodies = case["scenes"] * ((m - 8) / math.log(m / 8.0) + 1.0)
    elif kind == "rollout":
        bodies = case["scenes"] * (case["bodies"] + 1)
    elif kind == "towers":
        bodies = case["towers"] * case["height"]
    else:
        bodies = case["bodies"] + 1
    hull = bodies * (8 if kind == "towers" else 122 if kind == "large" else 148)
    pairs = bodies * (1.0 if kind == "towers" else 1.2)
    contacts = bodies * (1.0 if kind == "towers" else 0.3)
    pgs = case.get("pgs", 10)
    sub = SUBSTEPS * case.get("frames", 1)
    once = {"bytes": 324.0 * bodies + 12.0 * hull + 72.0 * pairs + 84.0 * contacts,
            "flops": 18.0 * hull + 1200.0 * pairs + 420.0 * pgs * contacts}
    # the reverse pass recomputes a substep and differentiates it
    k = 3.5 if kind == "rollout" else 1.0
    return {"bytes": once["bytes"] * sub * k, "flops": once["flops"] * sub * k}


# ---- the frame in 64 bits ---------------------------------------------------------
def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


def _mat(q):
    x, y, z, w = q.unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x),
                        1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)


def _mv(m, v):
    return (m @ v[..., None])[..., 0]


class _Sim:
    """One substep after another of the rigid-body step: gravity, boxes,
    all pairs, Minkowski portal refinement, Gauss-Seidel contacts in order,
    integration."""

    def __init__(self, buf, state, pgs):
        t, nb = buf.tensors, buf.num_bodies
        f = lambda name, c: t[name][: nb * c].reshape(nb, c).double()
        self.nb, self.pgs = nb, pgs
        self.p, self.q, self.v, self.w = (state[k].reshape(nb, c).double()
                                          for k, (_, c) in zip(KEYS, STATE))
        self.im, self.ii = f("body_inv_mass", 1), f("body_inv_inertia", 3)
        self.mu, self.e = f("geom_friction", 1), f("geom_restitution", 1)
        self.dyn = self.im > 0
        self.hull = t["hull_verts"].reshape(-1, 3).double()
        self.hs, self.hc = (x.long() for x in t["hull_range"][: 2 * nb].reshape(nb, 2).unbind(1))
        self.lk = t["support_offset"][:nb].long()
        self.lut = t["support_lookup"].long()
        scene = np.repeat(np.arange(buf.num_scenes), np.diff(buf.scene_body_offset))
        self.scene = torch.as_tensor(scene, device="cuda")
        self.end = torch.as_tensor(np.asarray(buf.scene_body_offset[1:], np.int64),
                                   device="cuda")[self.scene]

    def substep(self, dt):
        d = self.dyn.double()
        g = torch.tensor(G, dtype=torch.float64, device="cuda")
        self.v = torch.where(self.dyn, self.v * 0.999 + g * dt, self.v)
        self.w = torch.where(self.dyn, self.w * 0.998, self.w)
        self.R = _mat(self.q)
        i, j = self.pairs()
        n, depth, cp, keep = self.mpr(i, j)
        self.solve(i[keep], j[keep], n[keep], depth[keep], cp[keep], dt)
        self.p = self.p + self.v * dt * d
        ox, oy, oz = self.w.unbind(1)
        x, y, z, w = self.q.unbind(1)
        dq = torch.stack([ox * w + oy * z - oz * y, -ox * z + oy * w + oz * x,
                          ox * y - oy * x + oz * w, -ox * x - oy * y - oz * z], 1)
        self.q = torch.where(self.dyn, _unit(self.q + 0.5 * dq * dt), self.q)

    def pairs(self):
        nb = self.nb
        owner = torch.repeat_interleave(torch.arange(nb, device="cuda"), self.hc)
        first = torch.cumsum(self.hc, 0) - self.hc
        idx = self.hs[owner] + torch.arange(len(owner), device="cuda") - first[owner]
        lo, hi = [], []
        for ax in range(3):  # one axis at a time: a batch holds millions of vertices
            x = (self.R[owner, ax] * self.hull[idx]).sum(-1) + self.p[owner, ax]
            z = torch.zeros(nb, dtype=torch.float64, device="cuda")
            lo.append(z.scatter_reduce(0, owner, x, "amin", include_self=False))
            hi.append(z.scatter_reduce(0, owner, x, "amax", include_self=False))
        lo, hi = self.lo, self.hi = torch.stack(lo, 1), torch.stack(hi, 1)
        rows, cols = [], []
        width = int((self.end - torch.arange(nb, device="cuda")).max())
        step = max(1, (1 << 25) // width)
        for r in range(0, nb, step):
            i = torch.arange(r, min(r + step, nb), device="cuda")[:, None]
            j = i + torch.arange(1, width + 1, device="cuda")
            ok = j < self.end[i]
            j = j.clamp(max=nb - 1)
            ok &= self.dyn[i, 0] | self.dyn[j, 0]
            for ax in range(3):
                ok &= (lo[i, ax] <= hi[j, ax]) & (lo[j, ax] <= hi[i, ax])
            a, b = ok.nonzero(as_tuple=True)
            rows.append(a + r)
            cols.append(j[a, b])
        return torch.cat(rows), torch.cat(cols)

    def support(self, b, d):
        """World point of body b farthest along d: over all hull vertices, or
        over the six that the body's angle tables name."""
        ld = _mv(self.R[b].transpose(1, 2), d)
        out = torch.empty_like(ld)
        table = self.lk[b] != 0
        for use, sel in ((True, table), (False, ~table)):
            k = sel.nonzero()[:, 0]
            if not len(k):
                continue
            bk, l = b[k], ld[k]
            if use:
                x, y, z = l.unbind(1)
                c = []
                for ax, (u, v) in enumerate(((y, z), (x, z), (x, y))):
                    a = torch.atan2(v, u)
                    a = torch.where(a < 0, a + 2 * math.pi, a)
                    n = (a / (2 * math.pi) * 64).long() % 64
                    c += [self.lk[bk] + ax * 64 + n, self.lk[bk] + ax * 64 + (n + 1) % 64]
                idx = self.hs[bk, None] + self.lut[torch.stack(c, 1)]
                ok = None
            else:
                m = torch.arange(int(self.hc[bk].max()), device="cuda")
                ok = m < self.hc[bk, None]
                idx = (self.hs[bk, None] + m).clamp(max=len(self.hull) - 1)
            pts = self.hull[idx]
            h = (pts * l[:, None]).sum(-1)
            h = h if ok is None else torch.where(ok, h, -math.inf)
            out[k] = pts[torch.arange(len(k), device="cuda"), h.argmax(1)]
        return self.p[b] + _mv(self.R[b], out)

    def mpr(self, i, j, eps=1e-6, tol=1e-6):
        n, m = len(i), 4
        S = torch.zeros(n, m, 3, 3, dtype=torch.float64, device="cuda")  # points: v, sa, sb
        S[:, 0] = torch.stack([self.p[i] - self.p[j], self.p[i], self.p[j]], 1)
        same = (S[:, 0, 0].abs() < eps).all(1)
        S[same, 0, 0, 0] += 10 * eps
        normal, cp = S[:, 0, 0].clone(), S[:, 0, 0].clone()
        depth = torch.zeros(n, dtype=torch.float64, device="cuda")
        found = torch.zeros(n, dtype=torch.bool, device="cuda")

        def point(k, d):
            a, b = self.support(i[k], d), self.support(j[k], -d)
            return torch.stack([a - b, a, b], 1)

        def portal(k):
            return _unit(_cross(S[k, 2, 0] - S[k, 1, 0], S[k, 3, 0] - S[k, 1, 0]))

        def tolerable(k, x, d):
            gap = (_dot(x[:, 0], d) - (S[k, 1:, 0] * d[:, None]).sum(-1)).amin(1)
            return gap < tol + eps * gap.clamp(min=1.0)

        def expand(k, x):
            c = _cross(x[:, 0], S[k, 0, 0])
            d1, d2, d3 = (_dot(S[k, a, 0], c)[:, 0] > 0 for a in (1, 2, 3))
            one = torch.ones_like(k)
            at = torch.where(d1, torch.where(d2, one, 3 * one), torch.where(d3, 2 * one, one))
            S[k, at] = x

        k = torch.arange(n, device="cuda")
        d = _unit(-S[:, 0, 0])
        x = point(k, d)
        go = _dot(x[:, 0], d)[:, 0] >= eps
        k, x = k[go], x[go]
        S[k, 1] = x
        c = _cross(S[k, 0, 0], x[:, 0])
        line = _dot(c, c)[:, 0] < eps  # the origin lies on the ray through the centres
        s, xs = k[line], x[line]
        found[s], cp[s] = True, 0.5 * (xs[:, 1] + xs[:, 2])
        depth[s], normal[s] = xs[:, 0].norm(dim=1), _unit(xs[:, 0])
        k, d = k[~line], _unit(c[~line])
        x = point(k, d)
        go = _dot(x[:, 0], d)[:, 0] >= eps
        k = k[go]
        S[k, 2] = x[go]
        d = _unit(_cross(S[k, 1, 0] - S[k, 0, 0], S[k, 2, 0] - S[k, 0, 0]))
        flip = (_dot(d, S[k, 0, 0]) > 0)[:, 0]
        f = k[flip]
        S[f, 1], S[f, 2] = S[f, 2].clone(), S[f, 1].clone()
        d = torch.where(flip[:, None], -d, d)
        refine = []
        for _ in range(15):  # portal discovery
            if not len(k):
                break
            x = point(k, d)
            go = _dot(x[:, 0], d)[:, 0] >= eps
            k, x = k[go], x[go]
            o = S[k, 0, 0]
            r2 = _dot(_cross(S[k, 1, 0], x[:, 0]), o)[:, 0] < -eps
            r1 = ~r2 & (_dot(_cross(x[:, 0], S[k, 2, 0]), o)[:, 0] < -eps)
            S[k[r2], 2], S[k[r1], 1] = x[r2], x[r1]
            done = ~(r1 | r2)
            S[k[done], 3] = x[done]
            refine.append(k[done])
            k = k[~done]
            d = _unit(_cross(S[k, 1, 0] - S[k, 0, 0], S[k, 2, 0] - S[k, 0, 0]))
        k = torch.cat(refine) if refine else k[:0]
        inside = []
        for _ in range(50):  # refinement until the portal holds the origin
            if not len(k):
                break
            d = portal(k)
            has = _dot(S[k, 1, 0], d)[:, 0] > -eps
            inside.append(k[has])
            k, d = k[~has], d[~has]
            x = point(k, d)
            go = (_dot(x[:, 0], d)[:, 0] > -eps) & ~tolerable(k, x, d)
            k, x = k[go], x[go]
            expand(k, x)
        k = torch.cat(inside + [k])
        for it in range(50):  # penetration
            if not len(k):
                break
            d = portal(k)
            x = point(k, d)
            end = tolerable(k, x, d) if it < 49 else torch.ones_like(k, dtype=torch.bool)
            s = k[end]
            found[s], normal[s], depth[s] = True, d[end], _dot(d[end], S[s, 1, 0])[:, 0]
            cp[s] = self.point(S[s], d[end], eps)
            k = k[~end]
            expand(k, x[~end])
        return normal, depth, cp, (found & (depth > 0)).nonzero()[:, 0]

    @staticmethod
    def point(S, d, eps):
        v0, v1, v2, v3 = S[:, :, 0].unbind(1)
        t = lambda a, b, c: _dot(_cross(a, b), c)
        b = torch.cat([t(v1, v2, v3), -t(v0, v2, v3), t(v0, v1, v3), -t(v0, v1, v2)], 1)
        z = torch.cat([torch.zeros_like(b[:, :1]), t(v2, v3, d), t(v3, v1, d), t(v1, v2, d)], 1)
        b = torch.where(b.sum(1, keepdim=True).abs() < eps, z, b)
        both = (b[:, :, None] * (S[:, :, 1] + S[:, :, 2])).sum(1)
        return 0.5 / b.sum(1, keepdim=True) * both

    def solve(self, a, b, n, depth, cp, dt):
        if not len(a):
            return
        # levels: a contact after every earlier one that shares a moving body
        dyn = self.dyn[:, 0].tolist()
        last, level = [0] * self.nb, []
        for x, y in zip(a.tolist(), b.tolist()):
            l = 1 + max(last[x] if dyn[x] else 0, last[y] if dyn[y] else 0)
            last[x] = last[y] = l
            level.append(l)
        level = torch.tensor(level, device="cuda")
        rows = []
        for l in range(1, int(level.max()) + 1):
            k = (level == l).nonzero()[:, 0]
            i, j = a[k], b[k]
            ra, rb = cp[k] - self.p[i], cp[k] - self.p[j]
            Ia = self.R[i] @ torch.diag_embed(self.ii[i]) @ self.R[i].transpose(1, 2)
            Ib = self.R[j] @ torch.diag_embed(self.ii[j]) @ self.R[j].transpose(1, 2)
            u = self.v[j] + _cross(self.w[j], rb) - self.v[i] - _cross(self.w[i], ra)
            e = torch.maximum(self.e[i], self.e[j])
            bias = 0.2 * (depth[k, None] - 0.005).clamp(min=0) / dt + \
                e * (-_dot(u, n[k])).clamp(min=0)
            rows.append([i, j, n[k], ra, rb, Ia, Ib, self.im[i], self.im[j], bias,
                         (self.mu[i] * self.mu[j]).sqrt(), torch.zeros_like(bias)])
        v, w = self.v.clone(), self.w.clone()
        for r in rows:
            ra, rb, N = r[3], r[4], r[2]
            ca, cb = _cross(ra, N), _cross(rb, N)
            r.append(r[7] + r[8] + _dot(ca, _mv(r[5], ca)) + _dot(cb, _mv(r[6], cb)))
        for _ in range(self.pgs):
            for r in rows:
                i, j, N, ra, rb, Ia, Ib, ma, mb, bias, mu, lam, kn = r
                va, wa, vb, wb = v[i], w[i], v[j], w[j]
                u = vb + _cross(wb, rb) - va - _cross(wa, ra)
                new = (lam + (bias - _dot(u, N)) / kn).clamp(min=0)
                P = (new - lam) * N
                r[11] = new
                va, vb = va - ma * P, vb + mb * P
                wa, wb = wa - _mv(Ia, _cross(ra, P)), wb + _mv(Ib, _cross(rb, P))
                u = vb + _cross(wb, rb) - va - _cross(wa, ra)
                s = u - _dot(u, N) * N
                size = s.norm(dim=1, keepdim=True)
                slip = size > 1e-6
                T = s / torch.where(slip, size, 1.0)
                ca, cb = _cross(ra, T), _cross(rb, T)
                kt = ma + mb + _dot(ca, _mv(Ia, ca)) + _dot(cb, _mv(Ib, cb))
                P = torch.where(slip, torch.minimum(size / kt, mu * new), 0.0) * T
                va, vb = va + ma * P, vb - mb * P
                wa, wb = wa + _mv(Ia, _cross(ra, P)), wb - _mv(Ib, _cross(rb, P))
                ia, jb = self.dyn[i], self.dyn[j]
                v[i[ia[:, 0]]], w[i[ia[:, 0]]] = va[ia[:, 0]], wa[ia[:, 0]]
                v[j[jb[:, 0]]], w[j[jb[:, 0]]] = vb[jb[:, 0]], wb[jb[:, 0]]
        self.v, self.w = v, w


def exact(case, seed):
    """A frame's poses and boxes in 64 bits.  Velocities, contact counts and
    gradients have no such value: a face that rests on a face touches at a corner that
    rounding chooses, and they jump with the corner.  Neither has the tree of
    a BVH (rounding of a centroid moves its Morton code).  The coloured
    solver visits contacts in an order of its own, and a path tracer's frame
    takes too long in plain operations."""
    kind = case["kind"]
    if kind in ("towers", "render"):
        return None
    d, buf, ph, init = _start(case, seed)
    if kind == "bvh":
        tri = torch.from_numpy(d.array("indices").astype(np.int64)).cuda()
        c = buf.tensors["vertices"][: 3 * buf.num_vertices].reshape(-1, 3).double()[tri].mean(1)
        names = ("morton", "sort_indices", "node_min", "node_max", "left", "right", "count",
                 "parent", "prim_indices")
        return {"centroids": c.reshape(-1), "scene_bounds": torch.cat([c.amin(0), c.amax(0)]),
                **dict.fromkeys(names)}
    ph.deinit()
    sim = _Sim(buf, init, case["pgs"])
    for _ in range(SUBSTEPS * case.get("frames", 1)):
        sim.substep(DT / SUBSTEPS)
    got = {"pos": sim.p.reshape(-1), "quat": sim.q.reshape(-1), "vel": None, "omega": None}
    if kind == "batch_io":
        return got
    if kind == "rollout":
        return {**got, **dict.fromkeys(("g_vel", "g_omega", "g_mu"))}
    return {**got, "aabb_min": sim.lo.reshape(-1), "aabb_max": sim.hi.reshape(-1), "counters": None}
