"""Rays that graze boxes and triangles (coordinates on a grid, origins in box faces,
targets at corners and on edges): closest-hit and any-hit queries agree on what is
hit, and renders of such a scene are those of the counting kernels, which walk the
nodes in the host's order.  At large coordinates the triangle test finds the
surface that a ray leaves again beyond the ray offset, so it is the box test that
decides, to the last bit."""
import numpy as np
import pytest

from test_gpu_ray_lengths import _trace

pytestmark = pytest.mark.gpu


def _scene(v, light, scale):
    """Diffuse triangles (n, 3, 3) with a point light, seen along z."""
    from sol_b200 import abi
    from sol_b200.scene import Bsdf, Camera, Light, Scene, Texture
    normal = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    area = np.linalg.norm(normal, axis=1)
    v, normal = v[area > 0].reshape(-1, 3), normal[area > 0] / area[area > 0, None]
    nt = len(normal)
    return Scene(vertices=np.float32(v * scale), normals=np.float32(np.repeat(normal, 3, axis=0)),
                 tex_coords=np.zeros((3 * nt, 2), np.float32), indices=np.arange(3 * nt, dtype=np.uint32).reshape(-1, 3),
                 tri_bsdf=np.zeros(nt, np.int32), tri_light=np.full(nt, -1, np.int32),
                 textures=[Texture(abi.TEX_CONSTANT_COLOR, (0.8, 0.8, 0.8))], bsdfs=[Bsdf(abi.BSDF_DIFFUSE, (0, -1, -1))],
                 lights=[Light(abi.LIGHT_POINT, v0=tuple(scale * x for x in light), intensity=(9.0 * scale * scale,) * 3)],
                 camera=Camera((0.3 * scale, 0.2 * scale, -9.0 * scale), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0), 60.0, 1.0))


def _grid_scene(seed, n=300):
    rng = np.random.default_rng(seed)
    v = rng.integers(-4, 5, (n, 3, 3)).astype(np.float64)
    flat = rng.integers(0, 4, n)   # three of four lie in an axis plane
    for k in range(3):
        v[flat == k, :, k] = v[flat == k, :1, k]
    return _scene(v, (1.0, 3.0, 2.0), 1.0)


def _boxes_scene(seed, scale, n=40):
    """Axis-parallel boxes, their faces split along random lines: leaves whose boxes have the
    surface that a ray leaves as a face."""
    rng = np.random.default_rng(seed)
    tris = []
    for _ in range(n):
        lo, size = rng.uniform(-4, 3, 3), rng.uniform(0.3, 1.5, 3)
        for k in range(3):
            for side in (0, 1):
                a, b = (k + 1) % 3, (k + 2) % 3
                cut = rng.uniform(0.2, 0.8)
                for s0, s1 in ((0.0, cut), (cut, 1.0)):
                    q = np.repeat(lo[None], 4, axis=0)
                    q[:, k] += size[k] * side
                    q[[1, 2], a] += size[a]
                    q[:, b] += size[b] * np.array([s0, s0, s1, s1])
                    q[[0, 3], a] = lo[a]
                    if side == 0:
                        q = q[::-1]
                    tris += [q[[0, 1, 2]], q[[0, 2, 3]]]
    return _scene(np.array(tris), (0.5, 6.0, -5.0), scale)


def _grazing_rays(scene, n, seed):
    rng = np.random.default_rng(seed)
    tri = scene.vertices[scene.indices[rng.integers(0, len(scene.indices), n)]].astype(np.float64)   # (n, corner, xyz)
    w = rng.dirichlet([1, 1, 1], n)
    part = rng.integers(0, 3, n)   # a corner, an edge, the inside
    w[part == 0] = np.eye(3)[rng.integers(0, 3, (part == 0).sum())]
    w[part == 1, 2] = 0.0
    at = (tri * (w / w.sum(1, keepdims=True))[..., None]).sum(1)
    d = np.where((rng.random(n) < 0.5)[:, None], rng.integers(-2, 3, (n, 3)), rng.uniform(-1, 1, (n, 3)))
    d[~d.any(1)] = (1, 0, 0)
    d = np.float32(d)
    org = np.float32(at - d.astype(np.float64) * np.exp(rng.uniform(-4, 2, (n, 1))))
    k = np.arange(n), rng.integers(0, 3, n)
    face = np.where(rng.random(n) < 0.5, tri.min(1)[k], tri.max(1)[k])
    org[k] = np.where(rng.random(n) < 0.4, face, org[k])
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7] = org, d
    rays[:, 3] = np.where(rng.random(n) < 0.5, 0.0, 1e-4)
    rays[:, 7] = np.finfo(np.float32).max
    return rays


@pytest.mark.parametrize("gpu_bvh", [False, True])
@pytest.mark.parametrize("seed", [1, 2])
def test_both_queries_hit_or_miss(built, seed, gpu_bvh):
    from sol_b200.renderer import GpuScene
    scene = _grid_scene(seed)
    gs = GpuScene(scene, gpu_bvh=gpu_bvh)
    rays = _grazing_rays(scene, 400_000, seed)
    closest, any_hit = _trace(gs, rays)[:, 0].view(np.int32) >= 0, _trace(gs, rays, True)[:, 0].view(np.int32) >= 0
    assert 0.3 < closest.mean() < 0.99
    assert np.array_equal(closest, any_hit), (closest != any_hit).sum()


@pytest.mark.parametrize("scale", [1.0, 1000.0, 8000.0])
@pytest.mark.parametrize("seed", [1, 2])
def test_films_are_the_counting_kernels(built, seed, scale):
    import torch
    from sol_b200 import capi
    from sol_b200.renderer import BatchRenderer, GpuPathTracer, GpuScene
    from sol_b200.scene import Config
    cfg = Config(max_path_len=6)
    scene = _grid_scene(seed) if scale == 1.0 else _boxes_scene(seed, scale)
    gs = GpuScene(scene)
    films = {}
    for name in ("counting", "split", "single", "wavefront", "views"):
        film = torch.zeros((3, 65, 65), device="cuda")
        if name in ("wavefront", "views"):
            b = BatchRenderer([gs], schedule=capi.BATCH_WAVEFRONT if name == "wavefront" else capi.BATCH_MEGAKERNEL)
            b.render(cfg, b.views([(0, scene.camera, 65, 65, 0, 8, film.data_ptr())]))
            b.stats()
        else:
            gs.set_instrumented(name == "counting")
            pt = GpuPathTracer(gs, cfg)
            for k in range(8 if name == "single" else 1):
                pt.render_device(film.data_ptr(), 65, 65, k, 1 if name == "single" else 8)
            pt.stats()
        torch.cuda.synchronize()
        films[name] = film.cpu().numpy()
    want = films["counting"]
    assert want.any()
    for name in ("split", "wavefront", "views"):
        assert np.array_equal(films[name], want), (name, (films[name] != want).sum())
    # single samples are summed into the film one by one instead of as one sum of 8
    assert np.abs(films["single"] - want).max() <= 8 * 2.0 ** -23 * np.abs(want).max()
