"""Scenes of 8 to 31 instances: batch traces test the instances in turn, and
the wavefront's frames walk an instance tree that the first one after a commit
builds or refits. Hits and images equal those without a tree bit for bit, with
instances moved and added between the calls."""
import numpy as np
import pytest

from raydemo_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _build(w, h, tree):
    from render_scenes import build_gpu

    spec = scenes.atrium(2, w, h, 3, level=2, n_spheres=9, tex_res=32)
    r = api.Renderer(w, h)
    sc = build_gpu(r, spec)
    sc.set_trace_tuning(instance_tree=tree)
    r.set_kernel(1)
    r.set_ray_sort(0)
    return r, sc, spec


def _frame(r, sc):
    r.Clear()
    r.RenderScene(sc, api.RegionContext())
    assert r.frame_info().error_flags == 0
    return r.get_pixels_ref().view(np.uint32).copy()


def test_tree_of_frames(cuda_device):
    (r, sc, spec), (r0, sc0, _) = _build(256, 144, 0), _build(256, 144, -1)
    n = len(spec["instances"])
    assert 8 <= n < 32
    rays = scenes.incoherent_rays(50000, seed=3, tmax=100.0)
    rays[:, :3] = rays[:, :3] * 20 - 10

    def state():
        i = sc.instance_tree_info()
        return i.instances, i.refit

    def both():
        hits, want = sc.trace_closest(rays, with_obj=True), sc0.trace_closest(rays, with_obj=True)
        assert np.array_equal(np.asarray(hits[0]).view(np.uint32), np.asarray(want[0]).view(np.uint32))
        assert np.array_equal(hits[1], want[1])

    both()
    assert state() == (0, 0)  # a trace builds none
    assert np.array_equal(_frame(r, sc), _frame(r0, sc0))
    assert state() == (n, 0)
    both()
    moved = np.array(spec["instances"][n - 1][1], np.float32).reshape(4, 4)
    for step in (1.0, -2.5):
        moved[3, :3] += step
        for s in (sc, sc0):
            s.SetMeshInstanceTransform(n - 1, moved.reshape(-1))
        both()
        assert state()[0] == 0  # not up to date, and not used
        assert np.array_equal(_frame(r, sc), _frame(r0, sc0))
        assert state() == (n, 1)
    for s in (sc, sc0):
        s.AddMeshInstance(spec["instances"][n - 1][0], np.eye(4, dtype=np.float32).reshape(-1))
    assert np.array_equal(_frame(r, sc), _frame(r0, sc0))
    assert state() == (n + 1, 0)
    both()


def test_small_frames_and_batches(cuda_device):
    """A frame below the tree's ray count leaves it; a batch counts all its frames' rays."""
    (a, sa, _), (b, sb, _) = _build(160, 120, 0), _build(160, 120, 0)
    (c, s_c, _) = _build(160, 120, -1)
    want = _frame(c, s_c)
    assert np.array_equal(_frame(a, sa), want)
    assert sa.instance_tree_info().instances == 0
    for r in (a, b):
        r.Clear()
    api.render_batch([a, b], [sa, sb], [api.RegionContext(), api.RegionContext()], 1)
    assert sa.instance_tree_info().instances > 0 and sb.instance_tree_info().instances > 0
    for r in (a, b):
        assert np.array_equal(r.get_pixels_ref().view(np.uint32), want)
