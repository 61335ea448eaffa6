"""Ray batches of few rays are spread over more warps: a prefix of a batch gives the
prefix of its hits, at either side of each lane count."""
import numpy as np
import pytest

from helpers import random_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("any_hit", [False, True])
def test_prefixes_agree(built, any_hit):
    import torch
    from sol_b200 import scenes
    from sol_b200.renderer import GpuScene
    gs = GpuScene(scenes.cornell_box(0))
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 32
    rays = torch.from_numpy(random_rays(5 * warps, (0.05, 0.05, 0.05), (0.95, 0.95, 0.95), seed=6)).cuda()

    def trace(n):
        hits = torch.full((n + 1, 4), -7.0, device="cuda")
        gs.trace(rays.data_ptr(), n, any_hit, hits.data_ptr())
        torch.cuda.synchronize()
        return hits.cpu().numpy().view(np.int32)
    whole = trace(5 * warps)
    assert (whole[:-1, 0] >= 0).mean() > 0.3
    for n in (1, 2, 63, 65, warps - 1, warps, warps + 1, 2 * warps, 2 * warps + 1, 4 * warps, 4 * warps + 1):
        got = trace(n)
        assert np.array_equal(got[:n], whole[:n]), n
        assert (got[n].view(np.float32) == -7.0).all()   # nothing written behind the batch
