"""What a call uploads has landed when it returns: renders on streams that do not wait
for the default stream see all of it (a copy from pageable memory may return
before its data has reached the device)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_new_parameters_are_seen_by_the_next_render(built):
    import torch
    from sol_b200 import scenes
    from sol_b200.renderer import GpuPathTracer, GpuScene, Image
    gs = GpuScene(scenes.cornell_box(0, textured=True, tex_size=512))
    pt = GpuPathTracer(gs, scenes.CORNELL_CONFIG)
    first = gs.get_params()
    rng = np.random.default_rng(0)
    for k in range(6):
        values = first * np.float32(rng.uniform(0.2, 1.0))
        gs.set_params(values)
        at_once, later = Image(48, 48), Image(48, 48)
        pt.render(at_once, 0, 1)          # on the handle's own stream
        torch.cuda.synchronize()
        pt.render(later, 0, 1)
        assert at_once.channels.any() and np.array_equal(at_once.channels, later.channels), k


def test_new_batch_renders_on_another_stream(built):
    import torch
    from sol_b200 import capi, scenes
    from sol_b200.renderer import BatchRenderer, GpuPathTracer, GpuScene
    made = [scenes.cornell_box(k) for k in range(24)]
    gs = [GpuScene(s) for s in made]
    stream = torch.cuda.Stream()
    films = [torch.zeros((3, 16, 16), device="cuda") for _ in gs]
    want = torch.zeros((3, 16, 16), device="cuda")
    torch.cuda.synchronize()
    for schedule in (capi.BATCH_MEGAKERNEL, capi.BATCH_WAVEFRONT):
        for f in films:
            f.zero_()
        torch.cuda.synchronize()
        b = BatchRenderer(gs, schedule=schedule)
        views = b.views([(k, s.camera, 16, 16, 0, 2, films[k].data_ptr()) for k, s in enumerate(made)])
        b.render(scenes.CORNELL_CONFIG, views, stream.cuda_stream)
        b.stats()
        for k in (0, 11, 23):
            want.zero_()
            GpuPathTracer(gs[k], scenes.CORNELL_CONFIG).render_device(want.data_ptr(), 16, 16, 0, 2)
            torch.cuda.synchronize()
            assert torch.equal(films[k], want), (schedule, k)
