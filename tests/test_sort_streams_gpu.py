"""Ray sorts of one renderer in flight on several streams: they share the
renderer's scratch, so each waits on the GPU for the one before it; every
call's permutation and rays are those of the call alone."""
import pytest

from raydemo_b200 import api, scenes

pytestmark = pytest.mark.gpu

COUNTS = (2000000, 921600, 1000, 500001)


def test_overlapping_sorts_of_one_renderer(cuda_device):
    import torch

    r = api.Renderer(16, 16)
    rays = [torch.from_numpy(scenes.incoherent_rays(n, seed=60 + k)).cuda() for k, n in enumerate(COUNTS)]
    streams = [torch.cuda.Stream() for _ in COUNTS]

    def sort(overlap):
        out = [(torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros((n, 8), device="cuda")) for n in COUNTS]
        torch.cuda.synchronize()
        for q, (perm, moved), s in zip(rays, out, streams):
            r.sort_rays_device(q.data_ptr(), len(q), (0.0, 0.0, 0.0), (1.0 / 255.0,) * 3, perm.data_ptr(), 0, moved.data_ptr(), s.cuda_stream)
            if not overlap:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return [t for pair in out for t in pair]

    want = sort(False)
    for k, q in enumerate(rays):
        assert torch.equal(q[want[2 * k].long()], want[2 * k + 1])
    for _ in range(4):
        assert all(torch.equal(a, b) for a, b in zip(sort(True), want))
