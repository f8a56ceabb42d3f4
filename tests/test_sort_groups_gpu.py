"""The radix sort's look-back at its grain: tiles of 4,096 keys in groups of 16,
eight groups a round. Ray counts around a group's and a round's edges, with
few and many distinct keys: hashes and permutation equal a stable argsort of the
hashes, and the moved rays the gathered ones."""
import numpy as np
import pytest

from raydemo_b200 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4095, 4097, 65535, 65536, 65537, 69633, 524287, 524289, 593921, 1048577, 2200001])
@pytest.mark.parametrize("spread", [0.0, 1.0])
def test_counts_at_group_edges(cuda_device, n, spread):
    import torch

    r = api.Renderer(16, 16)
    rays = scenes.incoherent_rays(n, seed=n)
    rays[:, :3] *= spread  # 0: every origin in one cell, the keys' low 24 bits equal
    d = torch.from_numpy(rays).cuda()
    keys, perm = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    out = torch.zeros((n, 8), device="cuda")
    s = torch.cuda.Stream()
    for moved in (True, False):
        torch.cuda.synchronize()
        r.sort_rays_device(d.data_ptr(), n, (0.0, 0.0, 0.0), (1.0 / 255.0,) * 3, perm.data_ptr(), keys.data_ptr(),
                           out.data_ptr() if moved else 0, s.cuda_stream)
        torch.cuda.synchronize()
        k = keys.cpu().numpy().view(np.uint32)
        exp = np.argsort(k, kind="stable")
        assert np.array_equal(perm.cpu().numpy(), exp)
        assert np.array_equal(out.cpu().numpy(), rays[exp])
