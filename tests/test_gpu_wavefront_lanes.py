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
