"""Memory of the queued lights: the queue stays below 1 GiB. A frame whose four
lights would need more traces them in the shading kernel, as one with five
lights (never queued) does, with the path kernel's image; one light of the same
frame is queued."""
import gc

import numpy as np
import pytest

from raydemo_b200 import api, scenes

pytestmark = pytest.mark.gpu

W, H = 2400, 2300  # 5.52 million pixels: 0.64 GB of queue per light


def _frame(n_lights, kernel=1):
    """The frame's pixels and the device memory it took."""
    import torch
    from render_scenes import build_gpu

    spec = scenes.cornell_box(0, W, H, 2)
    spec["lights"] = [{"type": 0, "position": (0.2 + 0.15 * k, 0.9, 0.4), "radius": 0.05, "color": (1.0, 1.0, 1.0)} for k in range(n_lights)]
    r = api.Renderer(W, H)
    sc = build_gpu(r, spec)
    r.set_kernel(kernel)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    r.RenderScene(sc, api.RegionContext())
    info = r.frame_info()
    assert info.error_flags == 0 and info.kernel == kernel
    px = r.get_pixels_ref().copy()
    used = free - torch.cuda.mem_get_info()[0]
    del r, sc
    gc.collect()
    return px, used


def test_the_queue_is_bounded(cuda_device):
    image, four = _frame(4)
    _, five = _frame(5)
    _, one = _frame(1)
    assert four - five < 64 << 20, (four, five)  # one GiB at the most, here none
    assert (256 << 20) < one - five < (1 << 30) + (64 << 20), (one, five)
    assert np.array_equal(image.view(np.uint32), _frame(4, 2)[0].view(np.uint32))
