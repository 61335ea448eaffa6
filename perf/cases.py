"""Timed workloads of the path tracer, through its public Python interface.

listed() names the workloads, draw() makes further ones of the same ranges.
Per case, prepare() builds what a program holds before the call (the uploaded
scene, films, rays, targets), run() makes one pass through the public entry
points and returns its outputs whole, work() says what the pass cannot do
without and exact() gives 64-bit results where an output has one.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sol_b200 import capi, scenes
from sol_b200.renderer import BatchRenderer, GpuPathTracer, GpuScene, Image, image_l2
from sol_b200.scene import Camera


def listed():
    return [
        # Camera preview while a scene is edited: one sample of a thumbnail, where the call itself is the cost.
        {"name": "preview", "kind": "render", "scene": "cornell", "width": 64, "height": 48, "spp": 1},
        # Progressive viewer: one more sample added into the host film that is shown, per call.
        {"name": "progressive", "kind": "host", "scene": "spheres", "spheres": 4, "textured": False,
         "width": 960, "height": 540, "spp": 1},
        # The Cornell box of the benchmark: long paths (up to 16 vertices), small scene.
        {"name": "cornell", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16},
        # Image textures (full shading), a ragged film and an odd sample count.
        {"name": "textured", "kind": "render", "scene": "spheres", "spheres": 12, "textured": True,
         "width": 701, "height": 389, "spp": 7},
        # The headline frame: 1,048,586 triangles, full HD, 64 samples.
        {"name": "frame", "kind": "render", "scene": "spheres", "spheres": 64, "textured": False,
         "width": 1920, "height": 1080, "spp": 64},
        # Views of one scene in one call (a multi-camera data set), through the wavefront.
        {"name": "views", "kind": "batch", "schedule": "wavefront", "scenes": 1, "spheres": 16, "views": 24,
         "min_side": 64, "max_side": 512, "max_spp": 32},
        # One view each of independent textured scenes in one call, through the multi-view megakernel.
        {"name": "scenes", "kind": "batch", "schedule": "megakernel", "scenes": 6, "spheres": 6, "views": 6,
         "min_side": 128, "max_side": 384, "max_spp": 16},
        # A step of texture optimisation: forward, L2 loss, path-replay adjoint.
        {"name": "train_step", "kind": "train", "scene": "cornell", "textured": True, "width": 128, "height": 128,
         "spp": 16},
        # The same for several scenes in one fused launch.
        {"name": "train_batch", "kind": "fused", "scenes": 6, "spheres": 6, "min_side": 128, "max_side": 320,
         "spp": 16},
        # Closest hits of scattered rays (bounce rays of an integrator that does its own shading).
        {"name": "closest", "kind": "trace", "spheres": 4, "rays": 300003, "any_hit": False},
        # Visibility of many point pairs: a batch of shadow rays in a larger mesh.
        {"name": "visibility", "kind": "trace", "spheres": 16, "rays": 1500000, "any_hit": True},
        # Moving geometry: upload the mesh with a device-built hierarchy and render a first sample.
        {"name": "rebuild", "kind": "rebuild", "spheres": 16, "textured": False, "width": 640, "height": 360,
         "spp": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "host", "batch", "train", "fused", "trace", "rebuild"])
    if kind in ("render", "host", "train"):
        c = {"kind": kind, "scene": rng.choice(["cornell", "spheres"]), "textured": kind == "train" or rng.random() < 0.3}
        if c["scene"] == "spheres":
            c["spheres"] = _log_int(rng, 1, 48)
        top = {"render": 1920, "host": 1280, "train": 320}[kind]
        c["width"] = _log_int(rng, 48, top)
        c["height"] = max(24, int(c["width"] * rng.uniform(0.5, 1.0)))
        most = {"render": 3e7, "host": 4e6, "train": 1e6}[kind]
        c["spp"] = _log_int(rng, 1, max(1, min(64 if kind != "train" else 16, int(most / (c["width"] * c["height"])))))
        return c
    if kind == "batch":
        n = rng.choice([1, 1, 2, 3, 5])
        return {"kind": kind, "schedule": rng.choice(["wavefront", "megakernel"]), "scenes": n,
                "spheres": _log_int(rng, 1, 16 if n == 1 else 6), "views": max(n, _log_int(rng, 2, 40)), "min_side": 64,
                "max_side": _log_int(rng, 96, 512), "max_spp": _log_int(rng, 1, 32)}
    if kind == "fused":
        return {"kind": kind, "scenes": rng.randint(1, 8), "spheres": _log_int(rng, 1, 6), "min_side": 48,
                "max_side": _log_int(rng, 64, 320), "spp": _log_int(rng, 1, 24)}
    if kind == "trace":
        return {"kind": kind, "spheres": _log_int(rng, 1, 32), "rays": _log_int(rng, 1000, 4000000),
                "any_hit": rng.random() < 0.5}
    w = _log_int(rng, 64, 1280)
    return {"kind": kind, "spheres": _log_int(rng, 1, 24), "textured": rng.random() < 0.3, "width": w,
            "height": max(24, int(w * rng.uniform(0.5, 1.0))), "spp": 1}


# --------------------------------------------------------------------------- inputs

def _scene(case, seed):
    """The case's mesh, its configuration and its camera."""
    if case.get("scene") == "cornell":
        s = scenes.cornell_box(seed, textured=bool(case.get("textured")), tex_seed=3 + seed)
        cfg = scenes.CORNELL_CONFIG
    else:
        s = scenes.sphere_field(case["spheres"], seed=seed, textured=bool(case.get("textured")))
        cfg = scenes.SPHERES_CONFIG
    c = s.camera
    return s, cfg, Camera(c.eye, c.dir, c.up, c.fov, case["width"] / case["height"]) if "width" in case else c


def _film(w, h):
    return torch.zeros((3, h, w), device="cuda")


def _scene_set(case, seed):
    """Independent textured scenes, each with a square film side in the case's range; sizes do not depend on the seed."""
    rng = scenes.Pcg(4)
    out = []
    for k in range(case["scenes"]):
        n = 1 + int(rng() * case["spheres"])
        seg = 2 * int(rng.uniform(24, 64))
        s = scenes.sphere_field(n, seed=1000 * seed + k, textured=True, sphere_sizes=[(seg // 2 + 1, seg)] * n, aspect=1.0)
        out.append((s, int(round(math.exp(rng.uniform(math.log(case["min_side"]), math.log(case["max_side"])))))))
    return out


def _grad(scene):
    """A gradient vector with room for the parameters of any scene of that size."""
    texels = sum(im.size for im in scene.images)
    return torch.zeros(64 + 4 * (scene.num_triangles // 100 + 16) + texels, device="cuda")


def _rays(case, seed):
    """Scattered rays inside the sphere field, or (any hit) segments from points in it to points on its lights."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["rays"]
    r = torch.empty((n, 8), device="cuda")
    r[:, 0:3] = torch.rand((n, 3), generator=g, device="cuda") * 10.0
    r[:, 3] = 1e-4
    if case["any_hit"]:
        to = torch.rand((n, 3), generator=g, device="cuda") * 10.0
        to[:, 1] = 11.0
        r[:, 4:7] = to - r[:, 0:3]
        r[:, 7] = 1.0 - 1e-4
    else:
        d = torch.randn((n, 3), generator=g, device="cuda")
        r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
        r[:, 7] = float(np.finfo(np.float32).max)
    return r


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "stream": torch.cuda.current_stream().cuda_stream}
    if kind in ("render", "host", "train"):
        s, cfg, cam = _scene(case, seed)
        st["pt"] = GpuPathTracer(GpuScene(s), cfg, cam)
        if kind == "host":
            st["image"], st["index"] = Image(case["width"], case["height"]), 0
        else:
            st["film"] = _film(case["width"], case["height"])
        if kind == "train":
            g = torch.Generator(device="cuda").manual_seed(seed)
            st["target"] = torch.rand(st["film"].shape, generator=g, device="cuda")
            st["dl"] = torch.empty_like(st["film"])
            st["grad"] = _grad(s)
            st["loss"] = torch.zeros((), dtype=torch.float64, device="cuda")
    elif kind == "batch":
        st["films"], specs = [], []
        if case["scenes"] == 1:
            s = scenes.sphere_field(case["spheres"], seed=seed)
            st["scenes"] = [GpuScene(s)]
            views = scenes.view_set(case["views"], min_side=case["min_side"], max_side=case["max_side"],
                                    max_spp=case["max_spp"])
            for cam, side, spp in views:
                st["films"].append(_film(side, side))
                specs.append((0, cam, side, side, 0, spp, st["films"][-1].data_ptr()))
        else:
            made = _scene_set(case, seed)
            st["scenes"] = [GpuScene(s) for s, _ in made]
            for v in range(case["views"]):
                s, side = made[v % len(made)]
                st["films"].append(_film(side, side))
                specs.append((v % len(made), s.camera, side, side, v // len(made) * case["max_spp"], case["max_spp"],
                              st["films"][-1].data_ptr()))
        schedule = capi.BATCH_WAVEFRONT if case["schedule"] == "wavefront" else capi.BATCH_MEGAKERNEL
        st["batch"] = BatchRenderer(st["scenes"], schedule=schedule)
        st["views"] = st["batch"].views(specs)
    elif kind == "fused":
        made = _scene_set(case, seed)
        st["scenes"] = [GpuScene(s) for s, _ in made]
        st["batch"] = BatchRenderer(st["scenes"])
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["films"] = [_film(side, side) for _, side in made]
        st["targets"] = [torch.rand(f.shape, generator=g, device="cuda") for f in st["films"]]
        st["grads"] = [_grad(s) for s, _ in made]
        st["losses"] = torch.zeros(len(made), dtype=torch.float64, device="cuda")
        st["specs"] = [(k, s.camera, side, side, 0, case["spp"], st["films"][k].data_ptr(), st["targets"][k].data_ptr(),
                        st["grads"][k].data_ptr(), st["losses"][k:k + 1].data_ptr()) for k, (s, side) in enumerate(made)]
    elif kind == "trace":
        st["scene"] = GpuScene(scenes.sphere_field(case["spheres"], seed=seed))
        st["rays"] = _rays(case, seed)
        st["hits"] = torch.empty((case["rays"], 4), dtype=torch.int32, device="cuda")
    else:
        st["mesh"], st["cfg"], st["cam"] = _scene(case, seed)
        st["film"] = _film(case["width"], case["height"])
    return st


# --------------------------------------------------------------------------- one pass

def run(st):
    case, stream = st["case"], st["stream"]
    kind = case["kind"]
    if kind == "render":
        st["film"].zero_()
        st["pt"].render_device(st["film"].data_ptr(), case["width"], case["height"], 0, case["spp"], stream)
        return st["film"]
    if kind == "host":
        st["pt"].render(st["image"], st["index"], case["spp"])
        st["index"] += case["spp"]
        return st["image"].channels
    if kind == "train":
        w, h, spp, film, dl = case["width"], case["height"], case["spp"], st["film"], st["dl"]
        film.zero_()
        st["loss"].zero_()
        st["grad"].zero_()
        st["pt"].render_device(film.data_ptr(), w, h, 0, spp, stream)
        image_l2(film.data_ptr(), st["target"].data_ptr(), film.numel(), 1.0 / spp, dl.data_ptr(),
                 st["loss"].data_ptr(), stream)
        st["pt"].adjoint(dl.data_ptr(), st["grad"].data_ptr(), w, h, 0, spp, stream)
        return {"film": film, "loss": st["loss"], "dl": dl, "grad": st["grad"]}
    if kind == "batch":
        torch._foreach_zero_(st["films"])
        st["batch"].render(scenes.SPHERES_CONFIG, st["views"], stream)
        return st["films"]
    if kind == "fused":
        torch._foreach_zero_(st["films"])
        torch._foreach_zero_(st["grads"])
        st["losses"].zero_()
        st["batch"].forward_adjoint(scenes.SPHERES_CONFIG, st["specs"], stream)
        return {"films": st["films"], "grads": st["grads"], "losses": st["losses"]}
    if kind == "trace":
        hits = st["hits"]
        st["scene"].trace(st["rays"].data_ptr(), case["rays"], case["any_hit"], hits.data_ptr(), stream)
        if case["any_hit"]:
            return hits[:, 0] >= 0
        return {"tri": hits[:, 0], "tuv": hits.view(torch.float32)[:, 1:]}
    st["scene"] = GpuScene(st["mesh"], gpu_bvh=True)
    st["film"].zero_()
    pt = GpuPathTracer(st["scene"], st["cfg"], st["cam"])
    pt.render_device(st["film"].data_ptr(), case["width"], case["height"], 0, case["spp"], stream)
    return st["film"]


# --------------------------------------------------------------------------- what a pass cannot do without

TRIANGLES = 16384      # per sphere of sphere_field
SCENE_BYTES = 192      # per triangle: its node, vertices and shading data, read once
RAY_FLOPS = 500        # about ten box pairs and one triangle per ray
VERTEX_FLOPS = 300     # surface, light sample, BSDF value and sample, with two rays per vertex


def work(case):
    kind = case["kind"]
    if kind == "trace":
        return {"bytes": case["rays"] * 48 + case["spheres"] * TRIANGLES * 112, "flops": case["rays"] * RAY_FLOPS}
    if kind in ("batch", "fused"):
        mean = (case["max_side"] ** 2 - case["min_side"] ** 2) / (2.0 * math.log(case["max_side"] / case["min_side"]))
        n = case.get("views", case["scenes"])
        spp = case.get("spp") or (case["max_spp"] if case["scenes"] > 1 else 0.5 * (1 + case["max_spp"]))
        pixels, paths = n * mean, n * mean * spp
        tris = case["spheres"] * TRIANGLES if case["scenes"] == 1 else case["scenes"] * case["spheres"] * 2048
        rays = 2.6
    else:
        pixels = case["width"] * case["height"]
        paths = pixels * case["spp"]
        cornell = case.get("scene") == "cornell"
        tris = 36 if cornell else case["spheres"] * TRIANGLES
        rays = 6.0 if cornell else 2.6
    flops = paths * rays * (RAY_FLOPS + VERTEX_FLOPS / 2)
    back = 2 if kind in ("train", "fused") else 1
    return {"bytes": tris * SCENE_BYTES + pixels * 24 * back, "flops": flops * back}


# --------------------------------------------------------------------------- 64-bit results

def exact(case, seed):
    """Hits by testing every ray against every triangle in 64 bits (small queries); a film is one draw of a random
    estimate, which has no value of its own to compare with."""
    tris = case.get("spheres", 0) * TRIANGLES
    if case["kind"] != "trace" or case["any_hit"] or case["rays"] * tris > 2e10:
        return None
    s = scenes.sphere_field(case["spheres"], seed=seed)
    v = torch.tensor(s.vertices, device="cuda", dtype=torch.float64)[torch.tensor(s.indices.astype(np.int64), device="cuda")]
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    n = torch.linalg.cross(e1, e2)
    rays = _rays(case, seed).double()
    tuv = torch.zeros((case["rays"], 3), dtype=torch.float64, device="cuda")
    step = max(1, int(2e7 // len(v0)))
    for a in range(0, case["rays"], step):
        o, d, lo, hi = rays[a:a + step, 0:3], rays[a:a + step, 4:7], rays[a:a + step, 3], rays[a:a + step, 7]
        # With m = o x d: det = -d.n, t = (o - v0).n / det, and the edge products from the scalar triple products.
        det = -(d @ n.T)
        t = (o @ n.T - (v0 * n).sum(1)) / det
        m = torch.linalg.cross(o, d)
        u = (m @ e2.T - d @ torch.linalg.cross(e2, v0).T) / det
        w = (d @ torch.linalg.cross(e1, v0).T - m @ e1.T) / det
        t[~((u >= 0) & (w >= 0) & (u + w <= 1) & (t > lo[:, None]) & (t < hi[:, None]))] = math.inf
        best, at = t.min(1)
        k = torch.arange(len(at), device="cuda")
        hit = torch.isfinite(best)
        tuv[a:a + step] = torch.where(hit[:, None], torch.stack([best, u[k, at], w[k, at]], 1), 0.0)
    return {"tri": None, "tuv": tuv}
