"""Traces of one scene in flight on several streams: the calls share the scene's
work counters (and the orders of reordered traces), so each waits on the GPU for
the one before it; every ray of every call gets its hit, the same as alone."""
import numpy as np
import pytest

from raydemo_b200 import api, scenes

pytestmark = pytest.mark.gpu

COUNTS = (1500000, 700001, 1000, 300000)


@pytest.mark.parametrize("reorder", [0, 1], ids=["input order", "reordered"])
def test_overlapping_traces_of_one_scene(cuda_device, reorder):
    import torch

    r = api.Renderer(16, 16)
    attrs, idx = scenes.triangle_soup_mesh(scenes.random_triangles(100000, seed=31, mean_edge=0.02))
    sc = r.CreateScene()
    m = sc.AddMaterial()
    sc.AddMeshInstance(sc.AddMesh(attrs, idx, [(m, 0, len(idx))]))
    sc.set_trace_tuning(reorder=reorder)
    rays = [torch.from_numpy(scenes.incoherent_rays(n, seed=40 + k)).cuda() for k, n in enumerate(COUNTS)]
    streams = [torch.cuda.Stream() for _ in COUNTS]

    def trace(overlap):
        hits = [torch.full((n, 4), -7, dtype=torch.int32, device="cuda") for n in COUNTS]
        torch.cuda.synchronize()
        for q, h, s in zip(rays, hits, streams):
            sc.trace_closest_device(q.data_ptr(), len(q), h.data_ptr(), 0, s.cuda_stream)
            if not overlap:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        assert sc.last_trace_info().error_flags == 0
        return hits

    want = trace(False)
    for _ in range(4):
        assert all(torch.equal(a, b) for a, b in zip(trace(True), want))


def test_host_trace_beside_a_device_trace(cuda_device):
    """A host-buffer call on one stream while a device-buffer call runs on another."""
    import torch

    r = api.Renderer(16, 16)
    attrs, idx = scenes.triangle_soup_mesh(scenes.random_triangles(100000, seed=32, mean_edge=0.02))
    sc = r.CreateScene()
    m = sc.AddMaterial()
    sc.AddMeshInstance(sc.AddMesh(attrs, idx, [(m, 0, len(idx))]))
    host = scenes.incoherent_rays(50000, seed=50)
    dev = torch.from_numpy(scenes.incoherent_rays(2000000, seed=51)).cuda()
    want = sc.trace_closest(host)
    stream = torch.cuda.Stream()
    hits = [torch.full((len(dev), 4), -7, dtype=torch.int32, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    sc.trace_closest_device(dev.data_ptr(), len(dev), hits[0].data_ptr(), 0, stream.cuda_stream)
    torch.cuda.synchronize()
    sc.trace_closest_device(dev.data_ptr(), len(dev), hits[1].data_ptr(), 0, stream.cuda_stream)
    got = sc.trace_closest(host)
    torch.cuda.synchronize()
    assert np.array_equal(np.asarray(got).view(np.uint32), np.asarray(want).view(np.uint32))
    assert torch.equal(hits[0], hits[1])


def test_captured_trace(cuda_device):
    """A device-buffer trace captured after one on another stream, its graph launched twice."""
    import torch

    r = api.Renderer(16, 16)
    attrs, idx = scenes.triangle_soup_mesh(scenes.random_triangles(5000, seed=33, mean_edge=0.05))
    sc = r.CreateScene()
    m = sc.AddMaterial()
    sc.AddMeshInstance(sc.AddMesh(attrs, idx, [(m, 0, len(idx))]))
    rays = torch.from_numpy(scenes.incoherent_rays(60000, seed=52)).cuda()
    want = torch.full((len(rays), 4), -7, dtype=torch.int32, device="cuda")
    hits = torch.full_like(want, -7)
    other, stream = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    sc.trace_closest_device(rays.data_ptr(), len(rays), want.data_ptr(), 0, other.cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sc.trace_closest_device(rays.data_ptr(), len(rays), hits.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        hits.fill_(-7)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(hits, want)
    sc.trace_closest_device(rays.data_ptr(), len(rays), hits.data_ptr(), 0, other.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(hits, want)
