"""The calls whose time is watched, as a user's program makes them.

Every case goes through the package's public classes (Scene, Renderer, Server,
Guide).  ``listed()`` names the ones looked at first, ``draw()`` gives more of
the same ranges.  A case is a dict of plain values with a ``kind``:

* ``pick``     Renderer.trace() on a host batch: mouse picking, line of sight,
               focus distance.  A few rays to a few ten thousand; the smallest
               calls there are, where latency is everything.
* ``rays``     Renderer.trace_device() on rays already on the GPU, leaving
               surface points in random directions: light-map baking (closest
               hit) and ambient occlusion (any hit with a finite reach).
* ``render``   one Render() and the download of its image, for each of the
               scene families: the Cornell box, the textured room, the
               2.6M-triangle spheres scene and the participating media, with
               either random stream, one sample per pixel (a viewer's frame)
               up to a final frame's 64, and the denoiser.
* ``guided``   a Render() that samples a path-guiding network which the
               program has loaded (a network trained earlier).
* ``gradients``  Guide.gradients(): loss and gradients of one training batch.
* ``serve``    a batch of mixed jobs through the render server.
* ``open``     a scene turned into a renderer, its first frame, and the
               renderer closed again: what the command line program does.

All inputs come from the seed: camera, random streams, the placement of the
geometry, the sky's orientation, rays, network parameters and samples.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import optixrender_b200 as rt
from optixrender_b200 import scenes, serve_bench

FLT_MAX = float(np.finfo(np.float32).max)


def listed():
    return [
        # 200 rays picked in the Cornell box: the smallest call
        {"name": "pick-200", "kind": "pick", "scene": "cornell", "rays": 200},
        # light-map baking: closest hits of 2^22 rays leaving the surfaces of the spheres scene
        {"name": "bake-4m", "kind": "rays", "any_hit": False, "rays": 1 << 22, "level": 8},
        # ambient occlusion at a ragged number of points
        {"name": "occlusion-1m", "kind": "rays", "any_hit": True, "rays": 1000003, "level": 8},
        # the Cornell configuration: 256 x 256, 16 spp, depth 8
        {"name": "cornell-256", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16,
         "depth": 8, "rr": 3, "rng": "pcg", "denoise": False},
        # a small preview of odd size with textures, shown denoised
        {"name": "textured-preview", "kind": "render", "scene": "textured", "width": 641, "height": 359, "spp": 4,
         "depth": 8, "rr": 3, "rng": "pcg", "denoise": True},
        # a viewer's frame while the camera moves: the defaults (1 spp, the reference's stream, depth 25)
        {"name": "viewer-1080p", "kind": "render", "scene": "spheres", "width": 1920, "height": 1080, "spp": 1,
         "depth": 25, "rr": 0, "rng": "lcg", "denoise": False},
        # the final frame of the spheres configuration: 1920 x 1080, 64 spp, depth 16
        {"name": "spheres-1080p-64", "kind": "render", "scene": "spheres", "width": 1920, "height": 1080, "spp": 64,
         "depth": 16, "rr": 0, "rng": "pcg", "denoise": False},
        # the media configuration at an eighth of its samples: 1280 x 720, 32 spp, depth 32
        {"name": "media-720p-32", "kind": "render", "scene": "media", "width": 1280, "height": 720, "spp": 32,
         "depth": 32, "rr": 0, "rng": "pcg", "denoise": False},
        # guided sampling of the portal room with a loaded network
        {"name": "guided-512", "kind": "guided", "width": 512, "height": 512, "spp": 16, "depth": 8},
        # one training batch of the renderer's own size
        {"name": "gradients-256k", "kind": "gradients", "samples": 1 << 18},
        # a burst of small and middling jobs on three resident scenes
        {"name": "serve-24", "kind": "serve", "jobs": 24, "largest": 512, "spp": 16},
        # the spheres scene opened, shown once and closed
        {"name": "open-spheres", "kind": "open", "width": 1920, "height": 1080, "spp": 1, "level": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pick", "rays", "rays", "render", "render", "render", "render", "guided", "gradients", "serve", "open"])
    if kind == "pick":
        return {"kind": kind, "scene": rng.choice(["cornell", "textured"]), "rays": _log_int(rng, 1, 50000)}
    if kind == "rays":
        return {"kind": kind, "any_hit": rng.random() < 0.5, "rays": _log_int(rng, 5000, 1 << 22),
                "level": rng.choice([6, 7, 8])}
    if kind == "render":
        scene = rng.choice(["cornell", "textured", "spheres", "media"])
        w = _log_int(rng, 96, 1920)
        h = min(1200, max(64, int(w * rng.uniform(0.45, 1.1))))
        lcg = rng.random() < 0.3
        top = 4 if lcg else min(64, max(1, int(3e7 if scene == "media" else 1.2e8) // (w * h)))
        depth, rr = {"cornell": (8, 3), "textured": (8, 3), "spheres": (16, 0), "media": (32, 0)}[scene]
        return {"kind": kind, "scene": scene, "width": w, "height": h, "spp": _log_int(rng, 1, top), "depth": depth,
                "rr": rr, "rng": "lcg" if lcg else "pcg", "denoise": rng.random() < 0.25}
    if kind == "guided":
        w = _log_int(rng, 96, 768)
        return {"kind": kind, "width": w, "height": max(64, int(w * rng.uniform(0.5, 1.0))),
                "spp": _log_int(rng, 1, 16), "depth": 8}
    if kind == "gradients":
        return {"kind": kind, "samples": _log_int(rng, 1000, 1 << 18)}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(3, 24), "largest": _log_int(rng, 96, 512), "spp": _log_int(rng, 2, 16)}
    w = _log_int(rng, 240, 1920)
    return {"kind": kind, "width": w, "height": max(64, int(w * 0.5625)), "spp": 1, "level": rng.choice([5, 6, 7, 8])}


# ------------------------------------------------------------------ scenes
# The fractal noise of a scene's base geometry takes seconds in numpy, so it is
# computed once; a seed turns, flips and rescales what it is given.
@functools.lru_cache(maxsize=None)
def _spheres(level):
    return scenes.spheres(ico_level=level)


@functools.lru_cache(maxsize=None)
def _media(grid):
    return scenes.media(grid_res=grid)


def _turn(p, angle):
    c, s = math.cos(angle), math.sin(angle)
    return (p @ np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]], np.float32).T).astype(np.float32)


def _spec(scene, seed, level=8, grid=128):
    """The named scene as this seed has it."""
    g = np.random.default_rng([seed, 77])
    if scene == "cornell":
        spec = scenes.cornell()
    elif scene == "textured":
        spec = scenes.textured(seed=1 + seed % 1000)
    elif scene == "portal":
        spec = scenes.portal()
    elif scene == "spheres":
        base = _spheres(level)
        meshes = []
        for m in base.meshes:  # the ground body turned one way, every sphere about the axis by its own angle
            a = g.uniform(-0.1, 0.1) if len(meshes) else g.uniform(0, 2 * math.pi)
            meshes.append(scenes.MeshSpec(_turn(m.positions, a), m.indices, m.material))
        spec = scenes.SceneSpec(base.name, meshes, [], [], base.env, base.camera, base.settings)
    else:
        base = _media(grid)
        media = [dict(m) for m in base.media]
        d = np.transpose(media[1]["density"], g.permutation(3))
        media[1]["density"] = np.ascontiguousarray(d * np.float32(g.uniform(0.8, 1.0)))
        spec = scenes.SceneSpec(base.name, base.meshes, base.lights, media, base.env, base.camera, base.settings)
    if spec.env is not None:
        spec.env = np.roll(spec.env, int(g.integers(spec.env.shape[1])), axis=1)
    cam = dict(spec.camera)
    f, a = np.array(cam["from_"], np.float64), np.array(cam["at"], np.float64)
    f = a + (f - a) * g.uniform(0.95, 1.0) + g.uniform(-0.02, 0.02, 3)
    cam["from_"] = tuple(float(x) for x in f)
    spec.camera = cam
    return spec


def _settings(case, seed, **more):
    o = dict(width=case["width"], height=case["height"], spp=case["spp"], max_depth=case.get("depth", 25),
             rr_depth=case.get("rr", 0), rng=rt.RNG_LCG if case.get("rng") == "lcg" else rt.RNG_PCG32,
             seed=1 + seed, denoise=int(case.get("denoise", False)))
    o.update(more)
    return o


def _triangles(spec):
    return np.concatenate([m.triangles() for m in spec.meshes]).reshape(-1, 3, 3)


def _camera_rays(spec, n, g):
    """Rays of a pinhole camera through n points of its image."""
    f, a = np.array(spec.camera["from_"]), np.array(spec.camera["at"])
    fwd = (a - f) / np.linalg.norm(a - f)
    right = np.cross(fwd, [0.0, 1.0, 0.0])
    right /= np.linalg.norm(right)
    up = np.cross(right, fwd)
    d = fwd + g.uniform(-0.3, 0.3, (n, 1)) * right + g.uniform(-0.3, 0.3, (n, 1)) * up
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3], r[:, 3], r[:, 4:7], r[:, 7] = f, 1e-4, d / np.linalg.norm(d, axis=1, keepdims=True), FLT_MAX
    return r


def _surface_rays(spec, n, g, reach):
    """Rays from points of the surfaces, in the order of the triangles, into
    the outward half space (cosine distributed); `reach`: their length or None."""
    tri = _triangles(spec)
    pick = np.sort(g.integers(0, len(tri), n))
    t = torch.from_numpy(tri[pick].astype(np.float32)).cuda().double()
    u = torch.from_numpy(g.random((n, 4))).cuda()
    s = u[:, 0:1].sqrt()
    p = t[:, 0] * (1 - s) + t[:, 1] * (s * (1 - u[:, 1:2])) + t[:, 2] * (s * u[:, 1:2])
    nrm = torch.linalg.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
    z = 1 - 2 * u[:, 2:3]
    ph = 2 * math.pi * u[:, 3:4]
    q = (1 - z * z).clamp_min(0).sqrt()
    d = nrm + 0.999 * torch.cat([q * ph.cos(), q * ph.sin(), z], 1)
    d = d / d.norm(dim=1, keepdim=True).clamp_min(1e-30)
    r = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    r[:, 0:3] = (p + 2e-4 * nrm).float()
    r[:, 3] = 1e-4
    r[:, 4:7] = d.float()
    r[:, 7] = FLT_MAX if reach is None else reach
    return r


# ------------------------------------------------------------------ prepare
def _network(seed):
    """Parameters of a guiding network with the spread of a trained one: features of order 0.1, He-sized weights."""
    g = np.random.default_rng([seed, 5])
    sizes = [(64, 32), (64, 64), (64, 64), (32, 64)]
    ws = [g.standard_normal(s, dtype=np.float32) * np.float32(math.sqrt(2.0 / s[1])) for s in sizes]
    table = (g.random(16 * (1 << 19) * 2, dtype=np.float32) - np.float32(0.5)) * np.float32(0.4)
    return table, np.concatenate([w.reshape(-1) for w in ws])


def _samples(n, seed):
    """A training batch: points of a room's surfaces, directions towards a bright patch or anywhere, noisy weights."""
    g = np.random.default_rng([seed, 9])
    pos = g.random((n, 3), dtype=np.float32)
    face = g.integers(0, 6, n)
    pos[np.arange(n), face // 2] = (face % 2).astype(np.float32)
    aim = np.array([0.5, 0.5, 0.5]) + 0.1 * g.standard_normal((n, 3)) - pos
    d = np.where(g.random((n, 1)) < 0.6, aim, g.standard_normal((n, 3)))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    w = np.exp(g.standard_normal(n) * 1.5)
    return pos, d.astype(np.float32), w.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    g = np.random.default_rng([seed, 3])
    if kind == "pick":
        spec = _spec(case["scene"], seed)
        scene = scenes.build_scene(spec)
        return {"kind": kind, "renderer": rt.Renderer(scene, rt.options(width=16, height=16)),
                "rays": _camera_rays(spec, case["rays"], g)}
    if kind == "rays":
        spec = _spec("spheres", seed, case["level"])
        scene = scenes.build_scene(spec)
        rays = _surface_rays(spec, case["rays"], g, 0.8 if case["any_hit"] else None)
        hits = torch.empty((case["rays"], 4), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return {"kind": kind, "renderer": rt.Renderer(scene, rt.options(width=16, height=16)), "rays": rays,
                "hits": hits, "any_hit": case["any_hit"]}
    if kind == "render":
        spec = _spec(case["scene"], seed)
        r = rt.Renderer(scenes.build_scene(spec), rt.options(**_settings(case, seed)))
        h, w = case["height"], case["width"]
        return {"kind": kind, "renderer": r, "camera": rt.camera(**spec.camera), "denoise": case["denoise"],
                "pixels": np.empty((h, w), np.uint32), "linear": np.empty((h, w, 4), np.float32),
                "viewer": case["rng"] == "lcg"}
    if kind == "guided":
        spec = _spec("portal", seed)
        r = rt.Renderer(scenes.build_scene(spec), rt.options(**_settings(case, seed, rr_depth=3, guided=1, guide_train_spp=0)))
        r.guide().set_params(*_network(seed))
        return {"kind": kind, "renderer": r, "camera": rt.camera(**spec.camera),
                "linear": np.empty((case["height"], case["width"], 4), np.float32)}
    if kind == "gradients":
        net = rt.Guide()
        net.set_params(*_network(seed))
        return {"kind": kind, "guide": net, "batch": _samples(case["samples"], seed)}
    if kind == "serve":
        specs = [_spec("cornell", seed), _spec("spheres", seed, 6), _spec("media", seed, grid=64)]
        server = rt.Server(rt.server_options(max_depth=32))
        ids = [server.add_scene(scenes.build_scene(s)) for s in specs]
        top, spp = case["largest"], case["spp"]
        sizes = [(top, top), (top, max(1, top * 9 // 16)), (max(1, top // 2), max(1, top // 2)), (top // 4 + 1, max(1, top // 4))]
        jobs = []
        for i in range(case["jobs"]):  # every size at both sample counts on every scene in turn
            w, h = sizes[i % 4]
            st = specs[i % 3].settings
            jobs.append(rt.job(ids[i % 3], rt.camera(**serve_bench.orbit_camera(specs[i % 3].camera, g)), w, h,
                               spp if i // 4 % 2 else max(1, spp // 4), max_depth=st["max_depth"],
                               rr_depth=st["rr_depth"], seed=int(g.integers(1 << 62))))
        return {"kind": kind, "server": server, "jobs": jobs}
    spec = _spec("spheres", seed, case["level"])
    return {"kind": kind, "scene": scenes.build_scene(spec), "options": rt.options(**_settings(case, seed)),
            "camera": rt.camera(**spec.camera)}


# ------------------------------------------------------------------ run
def run(state):
    kind = state["kind"]
    if kind == "pick":
        hits = state["renderer"].trace(state["rays"])
        return {"hit": hits[:, :3], "triangle": hits[:, 3].view(np.int32)}
    if kind == "rays":
        hits, rays = state["hits"], state["rays"]
        state["renderer"].trace_device(rays.data_ptr(), rays.shape[0], hits.data_ptr(), any_hit=state["any_hit"])
        return {"hit": hits[:, :3], "triangle": hits.view(torch.int32)[:, 3]}
    if kind == "render":
        r = state["renderer"]
        r.set_camera(state["camera"])
        r.render()
        if state["viewer"]:
            return {"pixels": r.download_pixels(state["pixels"]).view(np.int32)}
        out = {"linear": r.download_linear(state["linear"])}
        if state["denoise"]:
            out["denoised"] = r.download_aov(rt.AOV_DENOISED)
        return out
    if kind == "guided":
        r = state["renderer"]
        r.set_camera(state["camera"])
        r.render()
        return {"linear": r.download_linear(state["linear"])}
    if kind == "gradients":
        loss, table, mlp = state["guide"].gradients(*state["batch"])
        return {"loss": loss, "table": table, "mlp": mlp}
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(j) for j in state["jobs"]]
        images = []
        for i in ids:
            server.wait(i)
            images.append(server.download_pixels(i).view(np.int32))
            server.release(i)
        return images
    r = rt.Renderer(state["scene"], state["options"])
    r.set_camera(state["camera"])
    r.render()
    out = {"pixels": r.download_pixels().view(np.int32), "linear": r.download_linear()}
    r.close()
    return out


# ------------------------------------------------------------------ work
# What a ray cannot do without, counted on an ideal 8-wide tree: one node (eight
# boxes of six planes, a multiply-add each) per three halvings of the
# triangles, two watertight triangle tests; and about 400 operations to shade
# its hit.  Bounces are the mean path lengths of the scenes.
_BOUNCES = {"cornell": 3.5, "textured": 3.5, "spheres": 4.0, "media": 8.0, "portal": 5.0}
_TRIANGLES = {"cornell": 34, "textured": 24, "media": 7212, "portal": 36}


def _ray_flops(triangles):
    return 96.0 * max(1.0, math.log2(max(2, triangles)) / 3.0) + 2 * 60.0


def _count(scene, level):
    return 20 * 4 ** level + 64 * 20000 if scene == "spheres" else _TRIANGLES[scene]


def _render_work(scene, level, pixels, spp, env):
    t = _count(scene, level)
    rays = pixels * spp * _BOUNCES[scene]
    return {"bytes": 36.0 * t + 100.0 * min(t, rays) + (32e6 if env else 0.0) + 20.0 * pixels,
            "flops": rays * (1.5 * _ray_flops(t) + 400.0)}


def work(case):
    kind = case["kind"]
    if kind in ("pick", "rays"):
        t = _count(case.get("scene", "spheres"), case.get("level", 8))
        return {"bytes": 48.0 * case["rays"] + 36.0 * min(t, case["rays"]), "flops": case["rays"] * _ray_flops(t)}
    if kind == "render":
        return _render_work(case["scene"], 8, case["width"] * case["height"], case["spp"], case["scene"] in ("spheres", "media"))
    if kind == "guided":
        w = _render_work("portal", 0, case["width"] * case["height"], case["spp"], False)
        n = case["width"] * case["height"] * case["spp"] * _BOUNCES["portal"]
        return {"bytes": w["bytes"] + 4e6, "flops": w["flops"] + 2 * 12288.0 * n}
    if kind == "gradients":
        n = case["samples"]  # each sample once, the addressed half of the table's levels once, the gradients written
        return {"bytes": 28.0 * n + 4.0 * (16 << 20) + 1e7, "flops": 3 * 2 * 12288.0 * n}
    if kind == "serve":
        pixels, parts = case["largest"] ** 2 * (1 + 0.5625 + 0.25 + 0.0625) / 4 * case["jobs"], []
        for scene in ("cornell", "spheres", "media"):
            parts.append(_render_work(scene, 6, pixels / 3, case["spp"] * 0.625, scene != "cornell"))
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    t = _count("spheres", case["level"])
    w = _render_work("spheres", case["level"], case["width"] * case["height"], case["spp"], True)
    return {"bytes": w["bytes"] + 96.0 * t + 64e6, "flops": w["flops"] + t * 20 * 100.0}


# ------------------------------------------------------------------ exact
def _exact_pick(case, seed):
    """Nearest hits by testing every triangle in double precision."""
    spec = _spec(case["scene"], seed)
    rays = _camera_rays(spec, case["rays"], np.random.default_rng([seed, 3])).astype(np.float64)
    tri = _triangles(spec).astype(np.float64)
    best = np.full((len(rays), 3), 0.0)
    best[:, 0] = FLT_MAX
    o, d = rays[:, 0:3], rays[:, 4:7]
    for a, b, c in tri:
        e1, e2 = b - a, c - a
        p = np.cross(d, e2)
        det = p @ e1
        ok = det != 0
        inv = 1.0 / np.where(ok, det, 1.0)
        s = o - a
        u = (s * p).sum(1) * inv
        q = np.cross(s, e1)
        v = (d * q).sum(1) * inv
        t = (q @ e2) * inv
        hit = ok & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > rays[:, 3]) & (t < best[:, 0])
        best[hit] = np.stack([t, u, v], 1)[hit]
    return {"hit": best, "triangle": None}


def _exact_gradients(case, seed):
    """The network's loss and gradients in double precision, by automatic differentiation."""
    table, mlp = (torch.from_numpy(p).cuda().double().requires_grad_() for p in _network(seed))
    pos, d, w = (torch.from_numpy(x).cuda() for x in _samples(case["samples"], seed))
    n_levels, size = 16, 1 << 19
    feats = []
    for level in range(n_levels):
        res = int(math.floor(16 * 4.0 ** (level / 15.0) + 1e-6))  # 16 .. 64, geometric: dense levels all
        p = pos * res  # the cell and the fraction are those of the single-precision product
        cell = p.floor().clamp_max(res - 1)
        f = (p - cell).double()
        tab = table[level * size * 2:(level + 1) * size * 2].view(size, 2)
        acc = 0
        for corner in range(8):
            bits = [(corner >> a) & 1 for a in range(3)]
            i = sum((cell[:, a].long() + bits[a]) * (res + 1) ** a for a in range(3))
            k = 1.0
            for a in range(3):
                k = k * (f[:, a] if bits[a] else 1 - f[:, a])
            acc = acc + k[:, None] * tab[i]
        feats.append(acc)
    x, at = torch.cat(feats, 1), 0
    for i, (rows, cols) in enumerate([(64, 32), (64, 64), (64, 64), (32, 64)]):
        x = x @ mlp[at:at + rows * cols].view(rows, cols).T
        at += rows * cols
        x = torch.relu(x) if i < 3 else x
    o = x.view(-1, 8, 4)
    kappa = o[..., 1].clamp(-2.0, 4.0).exp()
    th, ph = math.pi * torch.sigmoid(o[..., 2]), 2 * math.pi * torch.sigmoid(o[..., 3])
    mu = torch.stack([th.sin() * ph.cos(), th.sin() * ph.sin(), th.cos()], -1)
    cos = (mu * d.double()[:, None, :]).sum(-1)
    dens = kappa / (2 * math.pi * -torch.expm1(-2 * kappa)) * (kappa * (cos - 1)).exp()
    q = (torch.softmax(o[..., 0], 1) * dens).sum(1)
    loss = -(w.double() * q.log()).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "table": table.grad, "mlp": mlp.grad}


def exact(case, seed):
    """The values that have one without a random walk: hits of few rays by brute force, a batch's gradients."""
    if case["kind"] == "pick":
        return _exact_pick(case, seed)
    if case["kind"] == "gradients":
        return _exact_gradients(case, seed)
    return None
