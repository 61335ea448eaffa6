"""The adjoint's builds (picked by the size of the call) against each other.

Gradients are sums of 32-bit terms added in any order: N terms of one sign err
by about sqrt(N) 2^-24 of the sum, under 1e-4 for the up to 1e6 terms here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-4


def _tracer():
    from sol_b200 import scenes
    from sol_b200.renderer import GpuPathTracer, GpuScene
    return GpuPathTracer(GpuScene(scenes.cornell_box(1, textured=True, tex_size=32)), scenes.CORNELL_CONFIG)


def _close(a, b):
    return np.abs(a - b).max() <= TOL * np.abs(b).max() and np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)


# 75,776 lanes of the 4-block build: at limit 16 small up to 94,720 paths, middle up to 198,912
@pytest.mark.parametrize("w,h,spp", [(1, 1, 3), (33, 7, 2), (97, 51, 16), (128, 128, 8), (131, 129, 16)])
def test_a_call_is_the_sum_of_its_samples(built, w, h, spp):
    import torch
    pt = _tracer()
    n = pt.scene.param_layout()[0]
    whole, parts = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    dl = torch.rand((3, h, w), device="cuda", generator=torch.Generator("cuda").manual_seed(1)) + 0.1
    dl[:, :, w // 2] = 0.0 if w > 1 else 1.0   # pixels without a gradient are skipped
    pt.adjoint(dl.data_ptr(), whole.data_ptr(), w, h, 4, spp)
    st = pt.stats()
    for k in range(spp):   # single samples of these images: the small build
        pt.adjoint(dl.data_ptr(), parts.data_ptr(), w, h, 4 + k, 1)
    torch.cuda.synchronize()
    assert st.paths == spp * h * (w - (1 if w > 1 else 0))
    assert np.abs(whole.cpu().numpy()).max() > 0
    assert _close(whole.double().cpu().numpy(), parts.double().cpu().numpy())


@pytest.mark.parametrize("w,h,spp", [(31, 17, 3), (96, 80, 5), (128, 100, 16)])
def test_fused_matches_render_loss_and_adjoint(built, w, h, spp):
    import torch
    from sol_b200 import scenes
    from sol_b200.renderer import BatchRenderer, image_l2
    pt = _tracer()
    cam = pt.scene.scene.camera
    n = pt.scene.param_layout()[0]
    z = lambda *s: torch.zeros(s, device="cuda")   # noqa: E731
    target = torch.zeros((3, h, w), device="cuda")  # residuals of one sign, so the sums do not cancel
    film, film2, dl, g, g2 = z(3, h, w), z(3, h, w), z(3, h, w), z(n), z(n)
    loss = torch.zeros(2, dtype=torch.float64, device="cuda")
    br = BatchRenderer([pt.scene])
    br.forward_adjoint(scenes.CORNELL_CONFIG, [(0, cam, w, h, 9, spp, film.data_ptr(), target.data_ptr(), g.data_ptr(),
                                                loss.data_ptr())])
    pt.render_device(film2.data_ptr(), w, h, 9, spp)
    image_l2(film2.data_ptr(), target.data_ptr(), film2.numel(), 1.0 / spp, dl.data_ptr(), loss[1:].data_ptr())
    pt.adjoint(dl.data_ptr(), g2.data_ptr(), w, h, 9, spp)
    torch.cuda.synchronize()
    assert torch.equal(film, film2)
    a, b = loss.tolist()
    assert abs(a - b) <= 1e-6 * abs(b)   # the residual's rounding (sum * (1 / spp) in either order)
    assert _close(g.double().cpu().numpy(), g2.double().cpu().numpy())


def test_no_samples_add_nothing(built):
    import torch
    pt = _tracer()
    grad = torch.full((pt.scene.param_layout()[0],), 0.5, device="cuda")
    dl = torch.ones((3, 9, 7), device="cuda")
    pt.adjoint(dl.data_ptr(), grad.data_ptr(), 7, 9, 2, 0)
    st = pt.stats()
    assert (st.paths, st.rays) == (0, 0)
    assert (grad == 0.5).all()
