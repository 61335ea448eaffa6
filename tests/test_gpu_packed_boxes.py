"""Closest hits through the packed box nodes against the exact traversal: at
exactly equal distances (coincident triangles) and at scales near the ends
of the range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _coincident(copies, seed):
    """The Cornell box with every triangle `copies` times, in random order and with random BSDFs."""
    from sol_b200 import scenes
    s = scenes.cornell_box(1)
    rng = np.random.default_rng(seed)
    at = rng.permutation(np.tile(np.arange(s.num_triangles), copies))
    s.indices = np.ascontiguousarray(s.indices[at])
    s.tri_light = np.ascontiguousarray(s.tri_light[at])
    s.tri_bsdf = rng.integers(0, len(s.bsdfs), len(at)).astype(np.int32)
    return s


@pytest.mark.parametrize("copies", [1, 2, 9])   # 9: more coincident triangles than a leaf holds
@pytest.mark.parametrize("gpu_bvh", [False, True])
def test_equal_distances_resolve_as_in_the_exact_traversal(built, copies, gpu_bvh):
    import torch
    from sol_b200 import capi, scenes
    from sol_b200.renderer import BatchRenderer, GpuPathTracer, GpuScene
    s = _coincident(copies, 5)
    gs = GpuScene(s, gpu_bvh=gpu_bvh)
    pt = GpuPathTracer(gs, scenes.CORNELL_CONFIG)
    w, h, spp = 51, 37, 3
    films = {}
    for name in ("exact", "packed", "wavefront", "megakernel"):
        film = torch.zeros((3, h, w), device="cuda")
        if name in ("wavefront", "megakernel"):
            b = BatchRenderer([gs], schedule=capi.BATCH_WAVEFRONT if name == "wavefront" else capi.BATCH_MEGAKERNEL)
            b.render(scenes.CORNELL_CONFIG, b.views([(0, s.camera, w, h, 0, spp, film.data_ptr())]))
            b.stats()
        else:
            gs.set_instrumented(name == "exact")   # the counting kernels walk the exact nodes
            pt.render_device(film.data_ptr(), w, h, 0, spp)
            pt.stats()
        torch.cuda.synchronize()
        films[name] = film.cpu().numpy()
    assert films["exact"].any()
    for name, f in films.items():
        assert np.array_equal(f, films["exact"]), name


@pytest.mark.parametrize("num_tris", [1, 2, 8, 9])   # one leaf (both children of the root), and just more
@pytest.mark.parametrize("scale", [1e-8, 1.0, 1e8, 1e12])   # (beyond, the triangle test's products overflow)
def test_axis_parallel_rays_at_any_scale(built, num_tris, scale):
    """Rays along +-z through stacked triangles in planes of constant z: the nearest one ahead."""
    import torch
    from sol_b200 import abi
    from sol_b200.renderer import GpuScene
    from sol_b200.scene import Bsdf, Scene, Texture
    z = np.arange(num_tris, dtype=np.float32)
    v = np.array([[[-4, -4, k], [8, -4, k], [-4, 8, k]] for k in z], np.float32).reshape(-1, 3) * np.float32(scale)
    s = Scene(vertices=v, normals=np.tile(np.float32([0, 0, 1]), (len(v), 1)), tex_coords=np.zeros((len(v), 2), np.float32),
              indices=np.arange(len(v), dtype=np.uint32).reshape(-1, 3), tri_bsdf=np.zeros(num_tris, np.int32),
              tri_light=np.full(num_tris, -1, np.int32), textures=[Texture(abi.TEX_CONSTANT_COLOR, (0.5, 0.5, 0.5))],
              bsdfs=[Bsdf(abi.BSDF_DIFFUSE, (0, -1, -1))])
    rng = np.random.default_rng(3)
    n = 500
    rays = np.zeros((n, 8), np.float32)
    at = rng.integers(-1, num_tris, n) + 0.5
    rays[:, 0:2] = rng.uniform(-1, 1, (n, 2)) * scale
    rays[:, 2] = at * scale
    sign = np.where(rng.random(n) < 0.5, 1.0, -1.0)
    rays[:, 6] = sign
    rays[:, 7] = np.finfo(np.float32).max
    want = np.where(sign > 0, np.ceil(at), np.floor(at)).astype(int)
    want = np.where((want < 0) | (want >= num_tris), -1, want)
    for gpu_bvh in (False, True):
        hits = torch.zeros((n, 4), device="cuda")
        r = torch.from_numpy(rays).cuda()
        GpuScene(s, gpu_bvh=gpu_bvh).trace(r.data_ptr(), n, False, hits.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(hits.cpu().numpy()[:, 0].view(np.int32), want)
