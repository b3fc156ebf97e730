"""Performance cases of the renderer: what a program that uses this library has it do.

A case is a dict of plain values; ``prepare`` makes what the program holds before the
call (a Context with its scene, host arrays, network weights), ``run`` makes one pass
through the public entry points and returns everything it computed.  ``kind`` says
which path of the library a case takes:

* frame     — one image of a triangle scene: the Cornell box (reference estimator or
              next-event estimation) or a bumpy sphere of any triangle count; with
              ``motion`` the vertices are replaced first (an animated mesh: upload and
              BVH rebuild), with ``rebuild`` the BVH is rebuilt on the device;
* world     — a voxel-world frame under sun and sky, then the bilateral denoiser;
* views     — many cameras of uneven sizes traced together from a CUDA graph;
* adjoint   — image and material gradient by path replay (inverse rendering step);
* probe     — closest-hit queries of caller-made rays (picking, visibility, audio);
* train     — one optimisation step of the radiance cache's network on host samples;
* cached    — rendering with a frozen radiance cache;
* terrain   — voxel terrain generated and meshed (greedy as the reference's mesher, or
              one quad per exposed face), the mesh read back;
* obj       — Wavefront OBJ text parsed into the device mesh, the mesh read back.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import mcrt_gb300 as M
from mcrt_gb300 import scenes

PARAMS = ((96, 64), (64, 64), (64, 64), (64, 64), (64, 64), (64, 16))   # (inputs, outputs) per layer
LO, HI = np.float32([0.0, 0.0, 0.0]), np.float32([1.0, 1.0, 1.0])       # the Cornell box


def listed():
    return [
        # an interactive window's progressive frame: one sample per pixel of a tiny image, where latency and launches count
        dict(name="progressive_frame", kind="frame", scene="cornell", width=160, height=120, spp=1, depth=8, nee=False),
        # the reference's offline render of the Cornell box with next-event estimation, at the benchmark's size
        dict(name="cornell_nee", kind="frame", scene="cornell", width=512, height=512, spp=64, depth=8, nee=True),
        # preview of an animated mesh: new vertices each frame, ragged triangle count and image
        dict(name="animated_preview", kind="frame", scene="sphere", triangles=80001, width=637, height=359, spp=2, depth=6,
             nee=False, motion=True),
        # the benchmark frame: 1.3 million triangles, full HD, BVH rebuilt
        dict(name="mesh_frame_1080p", kind="frame", scene="sphere", triangles=1310720, width=1920, height=1080, spp=16,
             depth=12, nee=False, rebuild=True),
        # the voxel-world workload: 720p, 8 samples, sun and sky, 5 x 5 denoiser
        dict(name="world_denoised_720p", kind="world", nx=256, ny=128, nz=256, width=1280, height=720, spp=8, depth=6, radius=2),
        # batched cameras (data sets, thumbnails) over a smaller world, from a graph
        dict(name="batched_views", kind="views", views=9, layout=3, nx=128, ny=96, nz=128, spp=4, depth=6),
        # one step of inverse rendering at the differentiable Cornell box's size
        dict(name="inverse_step", kind="adjoint", width=256, height=256, spp=32, depth=8, nee=True),
        # a batch of probe rays into a mesh of ordinary size
        dict(name="probe_rays", kind="probe", triangles=81920, rays=250007),
        # one training step of the radiance cache
        dict(name="cache_train_step", kind="train", samples=131072),
        # rendering with a frozen radiance cache, half of the paths' length saved
        dict(name="cached_render", kind="cached", width=512, height=512, spp=16, depth=8, query_vertex=2),
        # a streamed region of terrain, greedy-meshed
        dict(name="terrain_greedy", kind="terrain", nx=128, ny=128, nz=128, place=5, greedy=True),
        # a mesh file of ordinary size
        dict(name="obj_import", kind="obj", triangles=81920),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["frame", "frame", "motion", "world", "views", "adjoint", "probe", "train", "cached", "terrain", "obj"])
    if kind in ("frame", "motion"):
        scene = "sphere" if kind == "motion" else rng.choice(["cornell", "sphere"])
        w, h = _log(rng, 100, 1600), _log(rng, 75, 900)
        spp = max(1, min(_log(rng, 1, 64), 16_000_000 // (w * h)))
        c = dict(kind="frame", scene=scene, width=w, height=h, spp=spp, depth=rng.randint(3, 12), nee=scene == "cornell" and rng.random() < 0.6)
        if scene == "sphere":
            c["triangles"] = _log(rng, 1000, 1_300_000)
            c["motion"] = kind == "motion"
            c["rebuild"] = not c["motion"] and rng.random() < 0.5
        return c
    if kind == "world":
        return dict(kind="world", nx=16 * rng.randint(3, 14), ny=rng.randint(40, 128), nz=16 * rng.randint(3, 14), width=_log(rng, 200, 1280),
                    height=_log(rng, 150, 720), spp=rng.randint(1, 8), depth=rng.randint(2, 6), radius=rng.randint(1, 5))
    if kind == "views":
        return dict(kind="views", views=rng.randint(2, 16), layout=rng.randint(0, 999), nx=16 * rng.randint(3, 9), ny=rng.randint(48, 96),
                    nz=16 * rng.randint(3, 9), spp=rng.randint(1, 6), depth=rng.randint(2, 6))
    if kind == "adjoint":
        return dict(kind="adjoint", width=_log(rng, 60, 320), height=_log(rng, 60, 320), spp=_log(rng, 4, 32), depth=rng.randint(3, 9),
                    nee=rng.random() < 0.7)
    if kind == "probe":
        return dict(kind="probe", triangles=_log(rng, 1000, 300_000), rays=_log(rng, 1000, 1_000_000))
    if kind == "train":
        return dict(kind="train", samples=_log(rng, 1000, 500_000))
    if kind == "cached":
        w, h = _log(rng, 128, 900), _log(rng, 128, 600)
        return dict(kind="cached", width=w, height=h, spp=max(1, min(_log(rng, 2, 32), 8_000_000 // (w * h))), depth=rng.randint(4, 10),
                    query_vertex=rng.randint(1, 3))
    if kind == "terrain":
        return dict(kind="terrain", nx=16 * rng.randint(2, 9), ny=rng.randint(32, 160), nz=16 * rng.randint(2, 9), place=rng.randint(0, 999),
                    greedy=rng.random() < 0.6)
    return dict(kind="obj", triangles=_log(rng, 500, 160_000))


# ---------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=4)
def _icosphere(level):
    return scenes.icosphere(level)


def _bumpy_sphere(n_tri, seed):
    """A unit icosphere cut to n_tri faces, displaced along its normals by seeded waves, with smooth normals, over a ground
    plane: (vertices, triangles, materials); groups of neighbouring faces share one of 12 materials, half of them
    Lambertian, then GGX conductors and glass (the benchmark mesh's mix)."""
    rng = np.random.default_rng(seed)
    level = max(1, math.ceil(math.log(max(n_tri, 21) / 20.0) / math.log(4.0) - 1e-9))
    p, f = _icosphere(level)
    f = f[:n_tri]
    k = rng.standard_normal((8, 3)) * (2.0 ** np.arange(8))[:, None] * 1.5
    ph = rng.uniform(0, 2 * np.pi, 8)
    disp = (np.sin(p @ k.T + ph) * 0.5 ** np.arange(8)).sum(1) * 0.04
    pos = p * (1.0 + disp)[:, None] + (0.0, 1.2, 0.0)
    fn = np.cross(pos[f[:, 1]] - pos[f[:, 0]], pos[f[:, 2]] - pos[f[:, 0]])
    vn = np.stack([sum(np.bincount(f[:, c], fn[:, a], len(pos)) for c in range(3)) for a in range(3)], 1)
    vn /= np.maximum(np.linalg.norm(vn, axis=1, keepdims=True), 1e-12)
    nv, nt = len(pos), len(f)
    V = np.zeros(nv + 4, M.VERTEX)
    V["position"][:nv, :3] = pos
    V["position"][:, 3] = 1.0
    V["normal"][:nv, :3] = vn
    V["position"][nv:, :3] = [(-6, 0, 6), (6, 0, 6), (6, 0, -6), (-6, 0, -6)]
    V["normal"][nv:, :3] = (0, 1, 0)
    T = np.zeros(nt + 2, M.TRIANGLE)
    T["v"][:nt] = f
    T["mat_idx"][:nt] = rng.integers(0, 12, 321)[np.arange(nt) * 320 // max(nt, 1)]
    T["v"][nt:] = [(nv, nv + 1, nv + 2), (nv, nv + 2, nv + 3)]
    T["mat_idx"][nt:] = 12
    mats = [(0, rng.uniform(0.2, 0.8, 3), 0.0, 1.0) for _ in range(6)]
    mats += [(4, rng.uniform(0.5, 0.95, 3), rng.uniform(0.05, 0.5), 1.0) for _ in range(4)]
    mats += [(2, (1.0, 1.0, 1.0), 0.0, 1.5) for _ in range(2)] + [(0, (0.5, 0.5, 0.5), 0.0, 1.0)]
    return V, T, M.materials(mats)


def _sky(seed):
    """A smooth HDR sky, 1024 x 512, brighter towards a seeded sun."""
    rng = np.random.default_rng(seed)
    th = (0.5 - (np.arange(512) + 0.5) / 512)[:, None] * np.pi
    ph = ((np.arange(1024) + 0.5) / 1024 - 0.5)[None, :] * 2 * np.pi
    s = rng.normal(size=3)
    s[1] = abs(s[1]) + 0.3
    s /= np.linalg.norm(s)
    c = np.cos(th) * np.cos(ph) * s[0] + np.sin(th) * s[1] + np.cos(th) * np.sin(ph) * s[2]
    base = 0.3 + 1.2 * np.clip(np.sin(th), 0, 1) + 4.0 * np.exp(20.0 * (c - 1.0))
    env = np.ones((512, 1024, 4), np.float32)
    env[..., :3] = base[..., None] * np.float32([0.9, 0.95, 1.1])
    return env


def _pinned(h, w):
    return torch.empty((h, w, 4), dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()


def _cornell(seed, ggx=False):
    return scenes.cornell_box_ggx(seed) if ggx else scenes.cornell_box(seed)


def _camera(c, w, h):
    return M.compute_camera(w, h, c["look_from"], c["look_at"], c["vfov"], c.get("aperture", 0.0))


def _world(ctx, case, seed):
    sc = scenes.voxel_world(seed, case["nx"], case["ny"], case["nz"])
    ctx.world_generate(sc["params"])
    ctx.world_mesh(sc["block_material"], sc["voxel_size"], greedy=False)
    ctx.upload_scene(materials=sc["materials"], env=M.gradient_env_map(), sun_dir=sc["sun_dir"],
                     sun_irradiance=sc["sun_irradiance"], world_mesh=True)
    return sc


def _views(case, seed):
    """Sizes from the case alone (every seed asks for the same images), poses from the seed."""
    r, g = random.Random(case["layout"]), random.Random(seed)
    s = 0.125
    ex, ey, ez = case["nx"] * s, case["ny"] * s, case["nz"] * s
    out = []
    for _ in range(case["views"]):
        w, h = r.randint(128, 640), r.randint(128, 480)
        a, d = g.uniform(0.0, 2.0 * math.pi), g.uniform(0.25, 0.48)
        eye = [d * ex * math.cos(a), g.uniform(0.75, 1.0) * ey, d * ez * math.sin(a)]
        at = [g.uniform(-0.2, 0.2) * ex, g.uniform(0.3, 0.5) * ey, g.uniform(-0.2, 0.2) * ez]
        out.append((M.compute_camera(w, h, eye, at, g.uniform(40.0, 70.0)), w, h))
    return out


def _network(seed):
    """He-initialised weights, the outputs near a grey radiance."""
    rng = np.random.default_rng(seed)
    parts = []
    for l, (i, o) in enumerate(PARAMS):
        w = rng.standard_normal((o, i)) * math.sqrt((2.0 if l < 5 else 0.3) / i)
        b = np.zeros(o)
        if l == 5:
            w[3:] = 0.0
            b[:3] = 0.4
        parts += [w.ravel(), b]
    return np.concatenate(parts).astype(np.float32)


def _samples(n, seed):
    """Training samples in the Cornell box: position, directions, albedo, the radiance of a smooth field, weight."""
    rng = np.random.default_rng(seed)
    s = np.ones((n, 16), np.float32)
    s[:, 0:3] = rng.random((n, 3), np.float32)
    for k in (3, 6):
        d = rng.standard_normal((n, 3), np.float32)
        s[:, k:k + 3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    s[:, 9:12] = rng.random((n, 3), np.float32)
    base = 0.6 + 0.3 * np.sin(5 * s[:, 0:1]) * np.cos(3 * s[:, 2:3]) + 0.2 * s[:, 4:5]
    s[:, 12:15] = base * (0.3 + s[:, 9:12])
    return s


def _rays(n, seed):
    """Half of the rays from a few eyes towards the sphere (coherent), half between random points (incoherent)."""
    rng = np.random.default_rng(seed + 1)
    k = n // 2
    eye = rng.uniform(-1, 1, (8, 3)) * (3.0, 1.0, 3.0) + (0.0, 2.5, 0.0)
    o = np.concatenate([eye[np.arange(k) * 8 // max(k, 1)], rng.uniform(-2, 2, (n - k, 3)) + (0.0, 2.0, 0.0)])
    to = rng.standard_normal((n, 3))
    to = to / np.linalg.norm(to, axis=1, keepdims=True) * 1.1 + (0.0, 1.2, 0.0)
    d = to - o
    return M.make_rays(o, d / np.linalg.norm(d, axis=1, keepdims=True))


def _obj(n_tri, seed):
    V, T, _ = _bumpy_sphere(n_tri, seed)
    return V["position"][:-4, :3], V["normal"][:-4, :3], T["v"][:-2].astype(np.int64)


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, k = case, case["kind"]
    if k != "train" or torch.cuda.is_available():
        s.ctx = M.Context(0)
    w, h = case.get("width"), case.get("height")
    if w:
        s.out = _pinned(h, w)
    if k == "frame":
        if case["scene"] == "cornell":
            sc = _cornell(seed)
            s.ctx.upload_scene(vertices=sc["vertices"], triangles=sc["triangles"], materials=sc["materials"], env=M.gradient_env_map())
            s.cam = _camera(sc["camera"], w, h)
        else:
            V, T, md = _bumpy_sphere(case["triangles"], seed)
            s.ctx.upload_scene(vertices=V, triangles=T, materials=md, env=_sky(seed))
            s.cam = M.compute_camera(w, h, [0.0, 2.2, 4.2], [0.0, 1.1, 0.0], 40.0)
            if case.get("motion"):
                s.vertices = V.copy()
                s.vertices["position"][:-4, 0] += np.float32(0.1) * np.sin(3 * V["position"][:-4, 1])
    elif k == "world":
        sc = _world(s.ctx, case, seed)
        s.cam = _camera(sc["camera"], w, h)
    elif k == "views":
        _world(s.ctx, case, seed)
        s.views = _views(case, seed)
    elif k == "adjoint":
        sc = _cornell(seed, ggx=True)
        s.ctx.upload_scene(vertices=sc["vertices"], triangles=sc["triangles"], materials=sc["materials"], env=M.gradient_env_map())
        s.cam = _camera(sc["camera"], w, h)
        s.d_image = np.random.default_rng(seed).standard_normal((h, w, 4)).astype(np.float32)
    elif k == "probe":
        V, T, md = _bumpy_sphere(case["triangles"], seed)
        s.ctx.upload_scene(vertices=V, triangles=T, materials=md)
        s.rays = _rays(case["rays"], seed)
    elif k == "train":
        s.ctx.cache_set_bounds(LO, HI)
        s.params, s.samples = _network(seed), _samples(case["samples"], seed)
    elif k == "cached":
        sc = _cornell(seed)
        s.ctx.upload_scene(vertices=sc["vertices"], triangles=sc["triangles"], materials=sc["materials"], env=M.gradient_env_map())
        s.cam = _camera(sc["camera"], w, h)
        s.ctx.cache_config(query_vertex=case["query_vertex"], train_stride=64, train_steps=0, lo=LO, hi=HI)
        s.ctx.cache_set_params(_network(seed))
    elif k == "terrain":
        # the place is the case's (every seed gives a mesh of one size); block materials and scale are the seed's
        s.params = scenes.world_params(case["place"], case["nx"], case["ny"], case["nz"])
        rng = np.random.default_rng(seed)
        s.blocks, s.voxel_size = rng.integers(0, 64, 256).astype(np.uint32), float(rng.uniform(0.05, 1.0))
    elif k == "obj":
        P, Nn, F = _obj(case["triangles"], seed)
        s.text = scenes.obj_text(P, F, normals=Nn)
    return s


# ---------------------------------------------------------------- one pass

def _mesh(v, t):
    return [v.view(np.float32).reshape(-1, 12), t.view(np.int32).reshape(-1, 4)]


def run(s):
    c, ctx, k = s.case, s.ctx, s.case["kind"]
    w, h, spp, depth = c.get("width"), c.get("height"), c.get("spp"), c.get("depth")
    if k == "frame":
        if c.get("motion"):
            ctx.update_vertices(s.vertices)
        if c.get("rebuild"):
            ctx.rebuild_bvh()
        ctx.render(s.cam, w, h, spp, max_depth=depth, nee=c["nee"], outputs=(), out_rgba=s.out)
        return s.out
    if k == "world":
        ctx.render(s.cam, w, h, spp, max_depth=depth, nee=True, outputs=(), out_rgba=s.out)
        return [s.out, ctx.denoise_accum(radius=c["radius"], sigma_color=0.1, sigma_normal=0.2)]
    if k == "views":
        return ctx.render_views(s.views, spp, max_depth=depth, nee=True, graph=True)
    if k == "adjoint":
        grad, image = ctx.adjoint(s.cam, w, h, spp, s.d_image, max_depth=depth, nee=c["nee"], with_image=True)
        return [grad, image]
    if k == "probe":
        hits = ctx.trace_closest(s.rays)
        return [np.ascontiguousarray(hits[f]) for f in ("t", "u", "v")] + [hits["prim"].view(np.int32)]
    if k == "train":
        ctx.cache_set_params(s.params)
        loss, grad = ctx.cache_train(s.samples, steps=1, lr=1e-3, want_grad=True)
        return [loss, grad, ctx.cache_params()]
    if k == "cached":
        ctx.render(s.cam, w, h, spp, max_depth=depth, nee=True, cache=True, outputs=(), out_rgba=s.out)
        return s.out
    if k == "terrain":
        ctx.world_generate(s.params)
        ctx.world_mesh(s.blocks, s.voxel_size, greedy=c["greedy"])
        return _mesh(*ctx.world_read_mesh())
    ctx.mesh_reset()
    ctx.mesh_append_obj(s.text)
    return _mesh(*ctx.mesh_read())


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    """Bytes: the scene and host inputs read once, the outputs written once.  Operations: paths x the mean number of
    segments that such a scene's paths have (two extend on an open scene, depth-limited in a closed box), each a walk of
    log2(triangles) boxes of 24 operations, one triangle and one shading point of about 150; the network's products; a
    hash and a comparison per voxel and octave."""
    k, nt = case["kind"], case.get("triangles", 36)
    px = case.get("width", 0) * case.get("height", 0)

    def paths(n, tri, seg):
        return n * seg * (24 * math.log2(tri + 2) + 150)

    mesh = nt * 0.5 * 48 + nt * 16
    if k == "frame":
        seg = 0.7 * case["depth"] if case["scene"] == "cornell" else 2.0
        seg *= 2 if case["nee"] else 1
        build = nt * math.log2(nt + 2) * 30 if case.get("motion") or case.get("rebuild") else 0
        return {"bytes": mesh + px * 16 + (mesh if case.get("motion") else 0), "flops": paths(px * case["spp"], nt, seg) + build}
    if k in ("world", "views"):
        tri = case["nx"] * case["nz"] * 75
        if k == "views":
            r = random.Random(case["layout"])
            px = sum(r.randint(128, 640) * r.randint(128, 480) for _ in range(case["views"]))
        flops = paths(px * case["spp"], tri, 3.0)
        if k == "world":
            flops += px * (2 * case["radius"] + 1) ** 2 * 40
        return {"bytes": tri * 40 + px * 16 * (2 if k == "world" else 1), "flops": flops}
    if k == "adjoint":
        return {"bytes": px * 32, "flops": 1.5 * paths(px * case["spp"], 36, 0.7 * case["depth"] * (2 if case["nee"] else 1))}
    if k == "probe":
        return {"bytes": mesh + case["rays"] * 48, "flops": paths(case["rays"], nt, 1.0)}
    if k == "train":
        return {"bytes": case["samples"] * 64 + 4 * 23888 * 4, "flops": case["samples"] * 129024}
    if k == "cached":
        n = px * case["spp"]
        return {"bytes": px * 16, "flops": paths(n, 36, 2.0 * case["query_vertex"]) + n * 47104}
    if k == "terrain":
        cells = case["nx"] * case["ny"] * case["nz"]
        quads = case["nx"] * case["nz"] * (8 if case["greedy"] else 37)
        return {"bytes": cells + quads * 224, "flops": cells * 150}
    return {"bytes": nt * (0.5 * 76 + 42) + nt * (0.5 * 48 + 16), "flops": nt * 100}


# ---------------------------------------------------------------- the same in 64 bits

def _exact_hits(case, seed):
    V, T, _ = _bumpy_sphere(case["triangles"], seed)
    rays = _rays(case["rays"], seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    P = torch.from_numpy(V["position"][:, :3].astype(np.float64)).to(dev)
    idx = torch.from_numpy(T["v"].astype(np.int64)).to(dev)
    a = P[idx[:, 0]]
    e1, e2 = P[idx[:, 1]] - a, P[idx[:, 2]] - a
    n = torch.linalg.cross(e1, e2)
    org = torch.from_numpy(np.ascontiguousarray(rays["org"]).astype(np.float64)).to(dev)
    dr = torch.from_numpy(np.ascontiguousarray(rays["dir"]).astype(np.float64)).to(dev)
    out = []
    step = max(1, (1 << 27) // len(T))
    for i in range(0, len(rays), step):      # Cramer's rule, every ray against every triangle, by matrix products
        o, d = org[i:i + step], dr[i:i + step]
        det = -(d @ n.T)
        m = torch.linalg.cross(o, d)
        # with s = o - a, m = o x d: s.(d x e2) = m.e2 - d.(e2 x a), d.(s x e1) = d.(e1 x a) - m.e1, e2.(s x e1) = s.n
        u = (m @ e2.T - d @ torch.linalg.cross(e2, a).T) / det
        v = (d @ torch.linalg.cross(e1, a).T - m @ e1.T) / det
        t = (o @ n.T - (a * n).sum(1)[None, :]) / det
        ok = (det.abs() > 1e-8) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 1e-4)
        t = torch.where(ok, t, torch.inf)
        best, j = t.min(1)
        hit = torch.isfinite(best)
        pick = lambda x: torch.where(hit, x.gather(1, j[:, None])[:, 0], torch.zeros_like(best))  # noqa: E731
        out.append(torch.stack([torch.where(hit, best, -torch.ones_like(best)), pick(u), pick(v)]))
    r = torch.cat(out, 1).cpu().numpy()
    return [r[0], r[1], r[2], None]


def _exact_train(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    s = torch.from_numpy(_samples(case["samples"], seed)).to(dev, torch.float64)
    p = torch.from_numpy(_network(seed)).to(dev, torch.float64).requires_grad_(True)
    u = s[:, :3].clamp(0, 1)
    feats = []
    for a in range(3):
        for b in range(12):
            x = u[:, a] * math.pi * 2.0 ** b
            feats += [torch.sin(x), torch.cos(x)]
    x = torch.cat([torch.stack(feats, 1), s[:, 3:12], u, torch.zeros_like(s[:, :12])], 1)
    at = 0
    for l, (i, o) in enumerate(PARAMS):
        W, b = p[at:at + i * o].reshape(o, i), p[at + i * o:at + i * o + o]
        at += i * o + o
        x = x @ W.T + b
        if l < 5:
            x = torch.relu(x)
    y = x[:, :3]
    terms = (y - s[:, 12:15]) ** 2 / (y.detach() ** 2 + 0.01)
    loss = terms.sum()
    grad = torch.autograd.grad(loss / (3.0 * len(s)), p)[0]
    new = p.detach() - 1e-3 * grad / (grad.abs() + 1e-8)          # Adam's first step from cleared moments
    return [loss.detach().reshape(1).cpu().numpy(), grad.cpu().numpy(), new.cpu().numpy()]


def _exact_obj(case, seed):
    P, Nn, F = _obj(case["triangles"], seed)
    uniq, first = np.unique(F.ravel(), return_index=True)
    order = uniq[np.argsort(first, kind="stable")]                # vertices are numbered at their first use
    v = np.zeros((len(order), 12))
    v[:, 0:3] = np.rint(P[order].astype(np.float64) * 1e6) / 1e6  # six decimals in the text
    v[:, 3] = 1.0
    v[:, 4:7] = np.rint(Nn[order].astype(np.float64) * 1e6) / 1e6
    return [v, None]


def exact(case, seed):
    """Sampled images have no 64-bit value (each sample's path follows from 32-bit rounding); a terrain mesh is lattice
    points and block ids."""
    k = case["kind"]
    if k == "probe":
        return _exact_hits(case, seed) if case["rays"] * case["triangles"] < 3e10 else None
    if k == "train":
        return _exact_train(case, seed)
    if k == "obj":
        return _exact_obj(case, seed)
    return None
