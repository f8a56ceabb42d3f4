"""The reference's lights whose shadow rays go through the wavefront's queue (up
to four lights per scene, no area lights) against the path kernel, which traces
them where it shades: the same image bit for bit, for every count around the
limit, with a transparent and a mixed occluder in the rays' way, in a batch of
scenes with different light counts, and next to an area light (not queued)."""
import numpy as np
import pytest

from raydemo_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _spec(n_lights, seed=0, transparent=True):
    spec = scenes.cornell_box(seed, 72, 56, 4)
    if transparent:
        tex = spec["materials"][0]["main_texture"]
        spec["materials"].append({"type": 5, "main_color": (1.0, 1.0, 1.0), "main_texture": tex})
        t = len(spec["materials"]) - 1
        spec["materials"].append({"type": 4, "main_texture": tex, "strength": 0.5, "mix_materials": (0, t), "int_ior": 1.0, "ext_ior": 1.0})
        for k, m in enumerate((t, t + 1)):  # two panes below the lights
            y = 0.8 - 0.1 * k
            a, i = scenes._quad((0.1, y, 0.1), (0.1, y, 0.9), (0.9, y, 0.9), (0.9, y, 0.1), (0, -1, 0))
            spec["meshes"].append((a, i, [(m, m, 0, 6)], 0))
            spec["instances"].append((len(spec["meshes"]) - 1, np.eye(4, dtype=np.float32).reshape(-1)))
    kinds = [{"type": 0, "position": (0.5, 0.9, 0.4), "radius": 0.05, "color": (2.0, 1.5, 1.0)},
             {"type": 1, "position": (0.2, 0.95, 0.5), "radius": 0.02, "color": (3.0, 3.0, 2.0), "direction": (0.2, -1.0, 0.1), "angle": 50.0},
             {"type": 2, "position": (0.0, 0.0, 0.0), "radius": 0.0, "color": (0.4, 0.5, 0.6), "direction": (0.1, -0.3, 1.0), "angle": 2.0},
             {"type": 0, "position": (0.8, 0.5, 0.1), "radius": 0.01, "color": (0.5, 0.5, 2.0)},
             {"type": 0, "position": (0.3, 0.3, -0.2), "radius": 0.1, "color": (0.2, 0.9, 0.3)}]
    spec["lights"] = kinds[:n_lights]
    return spec


def _build(spec):
    from render_scenes import build_gpu

    r = api.Renderer(*spec["size"])
    return r, build_gpu(r, spec)


def _image(spec, kernel, area=None):
    r, sc = _build(spec)
    if area:
        sc.AddLight(**area)
    r.set_kernel(kernel)
    reg = api.RegionContext()
    for _ in range(3):
        r.RenderScene(sc, reg)
    info = r.frame_info()
    assert info.error_flags == 0 and info.kernel == kernel
    return r.get_pixels_ref(), info.shadow_rays


@pytest.mark.parametrize("n_lights", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("transparent", [False, True])
def test_queued_lights_equal_the_path_kernel(cuda_device, n_lights, transparent):
    spec = _spec(n_lights, 0, transparent)
    (a, rays_a), (b, rays_b) = _image(spec, 1), _image(spec, 2)
    assert a[..., :3].max() > 0.1 and rays_a > 0
    if not transparent:
        assert rays_a == rays_b
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_lights_beside_an_area_light_equal_the_path_kernel(cuda_device):
    area = {"type": 3, "position": (0.35, 0.99, 0.35), "edge_u": (0.3, 0.0, 0.0), "edge_v": (0.0, 0.0, 0.3), "color": (4.0, 4.0, 4.0)}
    spec = _spec(2)
    assert np.array_equal(_image(spec, 1, area)[0].view(np.uint32), _image(spec, 2, area)[0].view(np.uint32))


def test_batch_of_scenes_with_different_light_counts(cuda_device):
    specs = [_spec(n, n) for n in (0, 1, 3, 4)]
    built = [_build(s) for s in specs]
    for r, _ in built:
        r.set_kernel(1)
    api.render_batch([r for r, _ in built], [s for _, s in built], [api.RegionContext() for _ in built], 3)
    for (r, _), spec in zip(built, specs):
        assert np.array_equal(r.get_pixels_ref().view(np.uint32), _image(spec, 2)[0].view(np.uint32))


def test_no_memory_for_the_queue_traces_the_lights_where_they_shade(cuda_device):
    """The k-th device allocation of a frame fails, for every k: the frame ends
    with an error, or (the queue's allocations) with the same image."""
    from raydemo_b200 import capi

    lib, spec = capi.lib(), _spec(2)

    def frame(k):
        r, sc = _build(spec)
        r.set_kernel(1)
        lib.ray_debug_fail_device_alloc(k)
        try:
            r.RenderScene(sc, api.RegionContext())
        except capi.RayError as e:
            assert e.code == capi.RAY_ERR_OUT_OF_MEMORY, e
            return None
        finally:
            lib.ray_debug_fail_device_alloc(-1)
        return r.get_pixels_ref().view(np.uint32)

    want = frame(-1)
    images = [frame(k) for k in range(240)]
    failed = [k for k, im in enumerate(images) if im is None]
    assert failed and failed[-1] < 230
    assert any(im is not None for im in images[:failed[-1]])  # the queue's
    assert all(np.array_equal(im, want) for im in images if im is not None)
