"""Ray queries with direction vectors of any length: scaled by a power of two, a
ray hits the same triangle at the same place, its distance scaled the other way
(every operation of the triangle test scales exactly).  Rays with a component
that the box test's own floor of 1e-30 would replace are left out."""
import numpy as np
import pytest

from helpers import random_rays

pytestmark = pytest.mark.gpu


def _trace(gs, rays, any_hit=False):
    import torch
    r = torch.from_numpy(rays).cuda()
    hits = torch.zeros((len(rays), 4), device="cuda")
    gs.trace(r.data_ptr(), len(rays), any_hit, hits.data_ptr())
    torch.cuda.synchronize()
    return hits.cpu().numpy()


@pytest.mark.parametrize("gpu_bvh", [False, True])
@pytest.mark.parametrize("exponent", [-95, -80, -75, -48, -47, 49, 50, 51, 80])
def test_scaled_directions_hit_the_same(built, exponent, gpu_bvh):
    from sol_b200 import scenes
    from sol_b200.renderer import GpuScene
    gs = GpuScene(scenes.sphere_field(4, seed=5, bands=17, segments=32), gpu_bvh=gpu_bvh)
    rays = random_rays(4000, (0, 0.2, 0), (10, 10, 10), seed=6)
    rays = rays[np.ldexp(np.abs(rays[:, 4:7]).min(1).astype(np.float64), exponent) > 1e-30]
    want = _trace(gs, rays)
    scaled = rays.copy()
    scaled[:, 4:7] = np.ldexp(rays[:, 4:7], exponent)
    scaled[:, 7] = np.inf
    got = _trace(gs, scaled)
    assert (want[:, 0].view(np.int32) >= 0).mean() > 0.3
    assert np.array_equal(got[:, 0].view(np.int32), want[:, 0].view(np.int32))
    assert np.array_equal(got[:, 1], np.ldexp(want[:, 1], -exponent))
    assert np.array_equal(got[:, 2:], want[:, 2:])
    assert np.array_equal(_trace(gs, scaled, True)[:, 0].view(np.int32) >= 0, got[:, 0].view(np.int32) >= 0)
