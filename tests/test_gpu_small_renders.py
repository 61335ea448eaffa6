"""Single-sample and small renders (one path per work item, few lanes per warp, the
6-block build) against the counting kernel's per-pixel loop, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _render(pt, w, h, spp, index):
    import torch
    film = torch.full((3, h, w), 0.25, device="cuda")   # added into, not overwritten
    pt.render_device(film.data_ptr(), w, h, index, spp)
    st = pt.stats()
    return film.cpu().numpy(), st


# 3552 warps of the 6-block build: one lane up to 3552 paths, two up to 7104, ...; 227,328 lanes of the full one
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (7, 1, 2), (96, 37, 1), (97, 37, 1), (119, 60, 2), (113, 63, 8),
                                     (476, 477, 1), (478, 477, 1), (641, 363, 2)])
@pytest.mark.parametrize("textured", [False, True])
def test_matches_the_per_pixel_loop(built, w, h, spp, textured):
    from sol_b200 import capi, scenes
    from sol_b200.renderer import GpuPathTracer, GpuScene
    gs = GpuScene(scenes.cornell_box(2, textured=textured, tex_size=16))
    pt = GpuPathTracer(gs, scenes.CORNELL_CONFIG)
    got, st = _render(pt, w, h, spp, 5)
    assert st.paths == w * h * spp
    assert (st.launches, st.sample_chunk) == ((1, 0) if spp == 1 else (2, spp))
    gs.set_instrumented(True)
    gs.set_schedule(capi.SCHEDULE_PER_PIXEL)
    want, st2 = _render(pt, w, h, spp, 5)
    assert np.array_equal(got, want)
    assert (st.rays, st.shadow_rays) == (st2.rays, st2.shadow_rays)
    assert (got != 0.25).any()


@pytest.mark.parametrize("spp", [1, 3])
def test_empty_paths(built, spp):
    from sol_b200 import scenes
    from sol_b200.renderer import GpuPathTracer
    from sol_b200.scene import Config
    got, st = _render(GpuPathTracer(scenes.cornell_box(2), Config(max_path_len=0)), 33, 9, spp, 0)
    assert st.paths == 33 * 9 * spp and st.rays == 0
    assert (got == 0.25).all()
