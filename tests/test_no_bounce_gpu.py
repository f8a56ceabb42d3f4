"""Frames and gradient steps without bounces in scenes of RAY_MAT_PRINCIPLED
materials only, whose shading is that material's own kernel: against the path
kernel, and against the same scene with an unused material of another type
beside, which takes the kernels of all materials."""
import numpy as np
import pytest

from raydemo_b200 import api, diff, scenes

pytestmark = pytest.mark.gpu


def _build(spec, other):
    from render_scenes import build_gpu

    if other:
        spec["materials"].append({"type": 0, "main_color": (0.5, 0.5, 0.5)})
    spec["camera"]["skip_indirect_lighting"] = True
    r = api.Renderer(*spec["size"])
    return r, build_gpu(r, spec)


def _image(kernel, other):
    r, sc = _build(scenes.atrium(1, 90, 70, 4, level=2, n_spheres=9, tex_res=32), other)
    r.set_kernel(kernel)
    reg = api.RegionContext()
    for _ in range(2):
        r.RenderScene(sc, reg)
    info = r.frame_info()
    assert info.error_flags == 0 and info.kernel == kernel
    return r.get_pixels_ref().copy(), r.debug_read(1)[: 90 * 70].copy()


def test_image_and_payloads(cuda_device):
    image, pay = _image(1, False)
    assert image[..., :3].max() > 0.1
    general, general_pay = _image(1, True)
    assert np.array_equal(image.view(np.uint32), general.view(np.uint32))
    assert np.array_equal(pay.view(np.uint32), general_pay.view(np.uint32))
    assert np.array_equal(image.view(np.uint32), _image(2, False)[0].view(np.uint32))


def test_gradient_step(cuda_device):
    import torch

    def step(other):
        spec = scenes.diff_atrium(0, 48, 40, 4, level=2, n_spheres=6, tex_res=64)
        r, sc = _build(spec, other)
        albedo = torch.full_like(torch.from_numpy(spec["albedo_target"]).cuda(), 0.4).requires_grad_()
        rough = torch.full_like(torch.from_numpy(spec["rough_target"]).cuda(), 0.5).requires_grad_()
        img = diff.render(albedo, rough, r, sc, spec["material_slot"] + [-1] * other, 1, 3)
        img.backward(torch.ones_like(img))
        return img.detach(), albedo.grad, rough.grad

    a, b = step(False), step(True)
    assert torch.equal(a[0], b[0]) and a[1].abs().max() > 0
    for x, y in zip(a[1:], b[1:]):  # sums in the atomics' order: some thousand terms of float rounding
        assert torch.allclose(x, y, rtol=1e-4, atol=1e-5 * float(y.abs().max()))
