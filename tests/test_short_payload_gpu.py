"""Wavefronts of scenes with RAY_MAT_PRINCIPLED materials only, whose payloads
hold the colour, the depth and the pdf: the image equals the path kernel's bit
for bit without and with ray sorting (which moves the payloads), in a batch and
next to a scene of other materials (full payloads); a frame without bounces
keeps the primary rays' full payloads for read-back."""
import numpy as np
import pytest

from raydemo_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _spec(w=90, h=70, bounces=5):
    return scenes.atrium(1, w, h, bounces, level=2, n_spheres=9, tex_res=32)


def _build(spec):
    from render_scenes import build_gpu

    r = api.Renderer(*spec["size"])
    return r, build_gpu(r, spec)


def _image(spec, kernel, sort=0):
    r, sc = _build(spec)
    r.set_kernel(kernel)
    r.set_ray_sort(sort)
    reg = api.RegionContext()
    for _ in range(2):
        r.RenderScene(sc, reg)
    assert r.frame_info().error_flags == 0
    return r.get_pixels_ref()


@pytest.mark.parametrize("bounces", [1, 2, 8])
@pytest.mark.parametrize("sort", [0, 0x3FF, 0x2])
def test_equal_to_the_path_kernel(cuda_device, bounces, sort):
    spec = _spec(bounces=bounces)
    a = _image(spec, 1, sort)
    assert a[..., :3].max() > 0.0
    assert np.array_equal(a.view(np.uint32), _image(spec, 2).view(np.uint32))


def test_batch_with_and_without_other_materials(cuda_device):
    specs = [_spec(64, 48), _spec(33, 57), scenes.cornell_box(0, 40, 40)]
    for group in (specs[:2], specs):
        for sort in (0, 0x3FF):
            built = [_build(s) for s in group]
            for r, _ in built:
                r.set_kernel(1)
                r.set_ray_sort(sort)
            api.render_batch([r for r, _ in built], [s for _, s in built], [api.RegionContext() for _ in built], 2)
            for (r, _), spec in zip(built, group):
                assert np.array_equal(r.get_pixels_ref().view(np.uint32), _image(spec, 2).view(np.uint32))


def test_payload_read_back(cuda_device):
    spec = _spec(24, 16)
    r, sc = _build(spec)
    r.set_kernel(1)
    r.set_ray_sort(0)
    cam = sc.GetCamera(0)
    cam.skip_indirect_lighting = True
    sc.SetCamera(0, cam)
    r.RenderScene(sc, api.RegionContext())
    pay = r.debug_read(1)[: 24 * 16]
    assert np.all(pay[:, :4] == 1.0) and np.abs(pay[:, 7:10]).min() > 0.0 and np.all(pay[:, 16].view(np.int32) == 0)
    cam.skip_indirect_lighting = False
    cam.max_total_depth = cam.max_diff_depth = 1
    sc.SetCamera(0, cam)
    r.RenderScene(sc, api.RegionContext())  # the buffer's second generation: rays that went on would have depth 2
    pay = r.debug_read(1)[: 24 * 16]
    assert pay.shape == (24 * 16, 20) and np.all(pay[:, 3] == 1.0) and np.all(pay[:, 4:16] == 0.0)
