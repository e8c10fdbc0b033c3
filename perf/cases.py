"""The work that users of this renderer have it do, as cases that can be timed and compared.

Each case is one call, or one short sequence of calls, that a program makes through the package's
public surface: single images (preview to full HD), progressive passes, FP64 films, one-shot renders
that build and upload their scene, batches of jobs, served requests, SPPM and ray queries. Scenes come
from the repository's own generator (orion_gb300/scenegen.py); every state is made from a seed, which
moves the camera, picks the range of sample passes and, where the generator takes one, seeds the
geometry.

    listed()              the cases, by name
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   what a program holds before the call: resident scene, jobs, server, rays
    run(state)            one pass; returns every film, count or hit array whole
    work(case)            bytes and operations that a pass cannot do without
    exact(case, seed)     ray queries: hit distance and barycentrics in 64 bits
"""
import math
import random

import numpy as np
import torch

import orion_gb300 as og
from orion_gb300 import scenegen

FLOAT_MAX = float(np.finfo(np.float32).max)


def listed():
    return [
        # The smallest call: one pass of a thumbnail while a scene is being edited.
        {"name": "preview", "kind": "render", "scene": "cornell", "subdiv": 3, "width": 64, "height": 64, "spp": 1,
         "depth": 5, "fp64": False},
        # The Cornell box of the benchmark: a small image where launches and kernel tails count.
        {"name": "cornell", "kind": "render", "scene": "cornell", "subdiv": 4, "width": 256, "height": 256, "spp": 16,
         "depth": 5, "fp64": False},
        # Every material and every light type at an odd film size: material look-development.
        {"name": "zoo", "kind": "render", "scene": "zoo", "subdiv": 4, "width": 333, "height": 217, "spp": 48,
         "depth": 6, "fp64": False},
        # Image textures on all material inputs, film as FP64 sums and sums of squares (error estimates).
        {"name": "textured_fp64", "kind": "render", "scene": "textured", "subdiv": 4, "width": 640, "height": 359,
         "spp": 32, "depth": 6, "fp64": True},
        # One sample pass of a 720p view: the step of a progressive viewer.
        {"name": "progressive", "kind": "render", "scene": "displaced", "subdiv": 7, "width": 1280, "height": 720,
         "spp": 1, "depth": 8, "fp64": False},
        # The benchmark's headline workload: 1.3M triangles, glossy conductor, 67M paths.
        {"name": "displaced", "kind": "render", "scene": "displaced", "subdiv": 8, "width": 1024, "height": 1024,
         "spp": 64, "depth": 8, "fp64": False},
        # The largest: full HD, five materials, thin lens, 265M paths.
        {"name": "mixed", "kind": "render", "scene": "mixed", "subdiv": 7, "width": 1920, "height": 1080, "spp": 128,
         "depth": 16, "fp64": False},
        # From host arrays to an image: scene build, upload, render, release (one image per program run).
        {"name": "one_shot", "kind": "one_shot", "scene": "displaced", "subdiv": 6, "width": 640, "height": 480,
         "spp": 16, "depth": 8},
        # Eight jobs of the benchmark's job distribution in one batched launch, FP32 films.
        {"name": "batch", "kind": "batch", "jobs": 8, "spp": 16, "res": 384},
        # Twelve requests (four scenes, three views each) through the serving loop.
        {"name": "served", "kind": "served", "scenes": 4, "views": 3, "spp": 16, "res": 256},
        # The benchmark's SPPM workload: 16 iterations of one photon per pixel.
        {"name": "sppm", "kind": "sppm", "subdiv": 5, "width": 512, "height": 512, "iterations": 16,
         "photons": 262144, "depth": 5},
        # Closest hits of incoherent rays (picking, visibility, light baking) against a resident scene.
        {"name": "rays", "kind": "rays", "subdiv": 5, "rays": 262144, "any_hit": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges that the listed ones stand for; sizes log-uniform, mostly odd."""
    kind = rng.choice(["render"] * 6 + ["one_shot", "batch", "served", "sppm", "rays"])
    if kind == "render":
        scene = rng.choice(["cornell", "zoo", "textured", "envlit", "displaced", "mixed"])
        width = _log_int(rng, 64, 1920)
        height = max(48, int(width * rng.uniform(0.5, 1.0)))
        spp = min(128, _log_int(rng, 1, 128))
        spp = max(1, min(spp, 100_000_000 // (width * height)))
        return {"kind": kind, "scene": scene, "subdiv": rng.randint(3, 8 if scene == "displaced" else 6),
                "width": width, "height": height, "spp": spp, "depth": rng.randint(4, 16),
                "fp64": rng.random() < 0.25}
    if kind == "one_shot":
        return {"kind": kind, "scene": rng.choice(["cornell", "zoo", "displaced"]), "subdiv": rng.randint(3, 7),
                "width": _log_int(rng, 128, 1024), "height": _log_int(rng, 128, 1024), "spp": _log_int(rng, 1, 32),
                "depth": rng.randint(4, 12)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 16), "spp": rng.choice([4, 16, 64]),
                "res": _log_int(rng, 96, 640)}
    if kind == "served":
        return {"kind": kind, "scenes": rng.randint(1, 5), "views": rng.randint(1, 4), "spp": rng.choice([4, 16, 32]),
                "res": _log_int(rng, 96, 512)}
    if kind == "sppm":
        width, height = _log_int(rng, 64, 512), _log_int(rng, 64, 512)
        return {"kind": kind, "subdiv": rng.randint(3, 5), "width": width, "height": height,
                "iterations": rng.randint(2, 16), "photons": _log_int(rng, 4096, 262144), "depth": rng.randint(3, 8)}
    return {"kind": kind, "subdiv": rng.randint(3, 7), "rays": _log_int(rng, 100, 2_000_000),
            "any_hit": rng.random() < 0.5}


# ------------------------------------------------------------------ states

_context = None


def context():
    """One context per process, as a program keeps one per device: its path state is allocated once."""
    global _context
    if _context is None:
        _context = og.Context(0)
    return _context


class State:
    """A prepared case; its resident scenes leave the device with it."""

    def __init__(self, case, **kw):
        self.case, self.sids, self.server = case, [], None
        self.__dict__.update(kw)

    def __del__(self):
        if self.server is not None:
            self.server.close()
        for sid in self.sids:
            context().release(sid)


def _scene(case, seed):
    """The case's generated scene, its camera moved and (where it has a seed) its geometry made by the seed."""
    rng = random.Random(seed)
    name, sub = case["scene"], case["subdiv"]
    if name == "cornell":
        s = scenegen.cornell(subdiv=sub)
    elif name == "zoo":
        s = scenegen.zoo(subdiv=sub)
    elif name == "textured":
        s = scenegen.textured(subdiv=sub)
    elif name == "envlit":
        s = scenegen.envlit(subdiv=sub)
    elif name == "displaced":
        s = scenegen.displaced(subdiv=sub, seed=1 + seed % 1000)
    else:  # the eight spheres, the finest at subdivision `sub`
        s = scenegen.mixed(subdivs=tuple(max(0, sub - d) for d in (2, 1, 0, 2, 1, 0, 1, 0)), seed=3 + seed % 1000)
    s.width, s.height, s.spp, s.max_depth = case["width"], case["height"], case["spp"], case["depth"]
    s.eye = tuple(e + rng.uniform(-0.15, 0.15) for e in s.eye)
    s.fov *= rng.uniform(0.9, 1.1)
    return s


def _jobs(case, count, seed):
    """`count` scenes of the job distribution at the case's film size and sample count."""
    out = []
    for k in range(count):
        s = scenegen.job((seed * 64 + k) % 100_003, tri_budget_scale=0.25)
        # A spread of film sizes around the case's, as the distribution has.
        s.width = max(32, case["res"] * (3 + k % 4) // 4)
        s.height = max(32, case["res"] * (3 + (k + 1) % 4) // 4)
        s.spp = case["spp"]
        out.append(s)
    return out


def _rays(case, seed):
    """Rays from a shell around the displaced sphere towards points near it; some miss."""
    g = np.random.RandomState(seed % (1 << 31))
    n = case["rays"]
    o = g.normal(size=(n, 3))
    o *= (g.uniform(1.5, 6.0, size=(n, 1)) / np.linalg.norm(o, axis=1, keepdims=True))
    d = g.uniform(-1.1, 1.1, size=(n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 3:6], rays[:, 7] = o, d, FLOAT_MAX
    return rays


def prepare(case, seed):
    ctx, kind = context(), case["kind"]
    if kind == "one_shot":  # the program's arrays are host data
        s = _scene(case, seed)
        return State(case, arrays=scenegen.scene_arrays(s), first_pass=0)
    if kind in ("render", "rays"):
        s = _scene(case, seed) if kind == "render" else scenegen.displaced(subdiv=case["subdiv"], seed=1 + seed % 1000)
        host = scenegen.to_host_scene(s)
        st = State(case, host=host, first_pass=(seed % 997) * case["spp"] if kind == "render" else 0)
        st.sids = [ctx.upload(host)]
        if kind == "rays":
            st.rays = _rays(case, seed)
        return st
    if kind == "batch":
        scenes = _jobs(case, case["jobs"], seed)
        st = State(case, hosts=[scenegen.to_host_scene(s) for s in scenes])
        st.sids = [ctx.upload(h) for h in st.hosts]
        st.jobs = [dict(sid=sid, width=s.width, height=s.height, spp=s.spp, max_depth=s.max_depth)
                   for sid, s in zip(st.sids, scenes)]
        return st
    if kind == "served":
        scenes = _jobs(case, case["scenes"], seed)
        st = State(case, hosts=[scenegen.to_host_scene(s) for s in scenes])
        st.requests = [(h, s.spp, s.max_depth, cam) for s, h in zip(scenes, st.hosts)
                       for cam in scenegen.job_views(s, case["views"])]
        st.server = og.Server(ctx, spp_chunk=16)
        return st
    s = scenegen.caustics(subdiv=case["subdiv"])
    rng = random.Random(seed)
    s.width, s.height = case["width"], case["height"]
    s.eye = tuple(e + rng.uniform(-0.15, 0.15) for e in s.eye)
    host = scenegen.to_host_scene(s)
    st = State(case, host=host, radius=0.05)
    st.sids = [ctx.upload(host)]
    return st


def run(st):
    ctx, c = context(), st.case
    kind = c["kind"]
    if kind == "render":
        return ctx.render(st.sids[0], c["width"], c["height"], spp=c["spp"], max_depth=c["depth"],
                          first_pass=st.first_pass, fp64=c["fp64"])
    if kind == "one_shot":
        host = og.HostScene.from_arrays(**st.arrays)
        sid = ctx.upload(host)
        film = ctx.render(sid, c["width"], c["height"], spp=c["spp"], max_depth=c["depth"])
        ctx.release(sid)
        return film
    if kind == "batch":
        outs, _ = ctx.render_batch(st.jobs, fp32=True)
        return [(s, n) for s, _, n in outs]
    if kind == "served":
        tickets = [st.server.submit(h, spp=spp, max_depth=depth, camera=cam) for h, spp, depth, cam in st.requests]
        films = []
        for t in tickets:
            st.server.wait(t)
            films.append(st.server.result(t))
            st.server.release(t)
        return films
    if kind == "sppm":
        return ctx.render_sppm(st.sids[0], c["width"], c["height"], iterations=c["iterations"], photons=c["photons"],
                               radius=st.radius, max_depth=c["depth"])
    if c["any_hit"]:  # occlusion queries report hit or miss
        return ctx.trace_wave(st.sids[0], st.rays, any_hit=True)[3]
    return ctx.trace(st.sids[0], st.rays)


# -------------------------------------------------------------------- work


def _triangles(scene, sub):
    ball = 20 * 4 ** sub
    if scene == "mixed":
        return sum(20 * 4 ** max(0, sub - d) for d in (2, 1, 0, 2, 1, 0, 1, 0)) + 6
    return {"cornell": 2 * ball + 12, "zoo": 7 * ball + 6, "textured": 5 * ball + 4, "envlit": 4 * ball + 2,
            "caustics": 3 * ball + 12, "displaced": ball + 2}[scene]


def _ray_flops(tris):
    """Operations of one ray in a binary tree over `tris` triangles: two boxes a level (24 operations
    each) on the way to one leaf, and its triangle (50)."""
    return 48 * math.log2(max(2, tris)) + 50


def work(case):
    """Bytes: corner positions and normals of each triangle (72) read once, films (or rays and hits)
    written or read once. Operations: each path's camera ray and, for half of the paths, one more bounce
    with a light sample (three rays, 600 operations of shading a bounce)."""
    kind = case["kind"]
    if kind in ("render", "one_shot"):
        tris = _triangles(case["scene"], case["subdiv"])
        px = case["width"] * case["height"]
        paths = px * case["spp"]
        return {"bytes": 72 * tris + px * (48 if case.get("fp64") else 16),
                "flops": paths * (2.5 * _ray_flops(tris) + 900)}
    if kind in ("batch", "served"):
        n = case["jobs"] if kind == "batch" else case["scenes"] * case["views"]
        scenes = case["jobs"] if kind == "batch" else case["scenes"]
        px, tris = case["res"] ** 2, 20_000
        return {"bytes": scenes * 72 * tris + n * px * (16 if kind == "batch" else 52),
                "flops": n * px * case["spp"] * (2.5 * _ray_flops(tris) + 900)}
    if kind == "sppm":
        tris, px = _triangles("caustics", case["subdiv"]), case["width"] * case["height"]
        return {"bytes": 72 * tris + 16 * px,
                "flops": case["iterations"] * (3 * px + 2 * case["photons"]) * (_ray_flops(tris) + 600)}
    tris = _triangles("displaced", case["subdiv"])
    return {"bytes": 72 * tris + case["rays"] * (32 + (4 if case["any_hit"] else 16)),
            "flops": case["rays"] * _ray_flops(tris)}


def exact(case, seed):
    """Closest hits by testing every triangle in 64 bits. A film has no such value: it is the sum of
    paths whose branches (which lobe, which triangle at an edge) depend on the last bits of 32-bit
    sampling, so two exact renderers differ by whole paths."""
    if case["kind"] != "rays" or case["any_hit"]:
        return None
    tris = _triangles("displaced", case["subdiv"])
    if case["rays"] * tris > 1.2e10:  # about ten seconds
        return None
    pos = scenegen.scene_arrays(scenegen.displaced(subdiv=case["subdiv"], seed=1 + seed % 1000))["positions"]
    p = torch.from_numpy(np.ascontiguousarray(pos, np.float32).reshape(-1, 3, 3)).double().cuda()
    p0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    rays = torch.from_numpy(_rays(case, seed)).double().cuda()
    out = torch.zeros((case["rays"], 3), dtype=torch.float64, device="cuda")
    chunk = max(1, 20_000_000 // tris)
    for a in range(0, case["rays"], chunk):
        o, d = rays[a:a + chunk, 0:3], rays[a:a + chunk, 3:6]
        # Moeller-Trumbore with the triple products written as matrix products over (ray, triangle):
        # det = -d.n, t = (o - p0).n / det, and u, v from the moment o x d.
        m = torch.linalg.cross(o, d)
        det = -(d @ nrm.T)
        t = (o @ nrm.T - (p0 * nrm).sum(1)) / det
        u = (m @ e2.T + d @ torch.linalg.cross(p0, e2).T) / det
        v = -(m @ e1.T + d @ torch.linalg.cross(p0, e1).T) / det
        hit = (t > 0) & (u >= 0) & (v >= 0) & (u + v <= 1)
        t = torch.where(hit, t, torch.inf)
        best, k = t.min(1)
        any_ = torch.isfinite(best)
        pick = torch.stack([best, u.gather(1, k[:, None])[:, 0], v.gather(1, k[:, None])[:, 0]], 1)
        out[a:a + chunk] = torch.where(any_[:, None], pick, torch.zeros_like(pick))
    return [out[:, 0].contiguous(), out[:, 1].contiguous(), out[:, 2].contiguous(), None]
