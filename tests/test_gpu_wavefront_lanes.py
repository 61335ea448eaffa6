"""Wavefront queues of few rays are traced with few lanes per warp: films of batches
whose queues start and end at either side of the lane counts, against plain renders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(1, 1, 1)], [(5, 3, 2), (1, 7, 1)], [(60, 59, 1)], [(61, 59, 2), (8, 8, 3)],
                                   [(240, 241, 2)], [(241, 240, 4), (3, 2, 1)]])
@pytest.mark.parametrize("host_loop", [False, True])
def test_films_match_plain_renders(built, sizes, host_loop):
    import torch
    from sol_b200 import capi, scenes
    from sol_b200.renderer import BatchRenderer, GpuPathTracer, GpuScene
    gs = GpuScene(scenes.cornell_box(3))
    pt = GpuPathTracer(gs, scenes.CORNELL_CONFIG)
    films = [torch.zeros((3, h, w), device="cuda") for w, h, _ in sizes]
    b = BatchRenderer([gs], schedule=capi.BATCH_WAVEFRONT, host_loop=host_loop)
    b.render(scenes.CORNELL_CONFIG, b.views([(0, gs.scene.camera, w, h, 2, spp, f.data_ptr())
                                             for (w, h, spp), f in zip(sizes, films)]))
    assert b.stats().paths == sum(w * h * spp for w, h, spp in sizes)
    for (w, h, spp), f in zip(sizes, films):
        want = torch.zeros((3, h, w), device="cuda")
        pt.render_device(want.data_ptr(), w, h, 2, spp)
        torch.cuda.synchronize()
        assert np.array_equal(f.cpu().numpy(), want.cpu().numpy())


def test_large_scene_build_matches_plain_render(built):
    """Nodes and triangles beyond 48 MB: the traversal stages' other build."""
    import torch
    from sol_b200 import capi, scenes
    from sol_b200.renderer import BatchRenderer, GpuPathTracer, GpuScene
    gs = GpuScene(scenes.sphere_field(28, seed=3), gpu_bvh=True)
    info = gs.info()
    assert 64 * info.num_nodes + 48 * info.num_triangles > 48 << 20
    w, h, spp = 93, 61, 3
    film, want = torch.zeros((3, h, w), device="cuda"), torch.zeros((3, h, w), device="cuda")
    b = BatchRenderer([gs], schedule=capi.BATCH_WAVEFRONT)
    b.render(scenes.SPHERES_CONFIG, b.views([(0, gs.scene.camera, w, h, 0, spp, film.data_ptr())]))
    b.stats()
    GpuPathTracer(gs, scenes.SPHERES_CONFIG).render_device(want.data_ptr(), w, h, 0, spp)
    torch.cuda.synchronize()
    assert want.any() and torch.equal(film, want)
