"""A corrupt instance tree whose root is its own child beside an instance: the
walk returns to the root after every instance without growing its stack. The
bound on node visits ends it and reports it for every block shape of the
trace kernels, the one without shared memory for the tree's visit count among
them, with one lane to a ray and with eight."""
import numpy as np
import pytest

from raydemo_b200 import api, capi, scenes

pytestmark = pytest.mark.gpu

SHAPES = [(1, 0, 0), (2, 64, 16), (3, 64, 16), (3, 128, 24), (2, 256, 24), (3, 256, 24)]


def _scene(r, shape):
    attrs, idx = scenes.triangle_soup_mesh(scenes.random_triangles(400, seed=5, mean_edge=0.1))
    sc = r.CreateScene()
    m = sc.AddMaterial()
    mesh = sc.AddMesh(attrs, idx, [(m, 0, len(idx))])
    rng = np.random.default_rng(6)
    for _ in range(24):
        x = np.eye(4, dtype=np.float32)
        x[3, :3] = rng.uniform(-0.5, 0.5, 3)
        sc.AddMeshInstance(mesh, x.reshape(-1))
    sc.set_trace_tuning(kernel=shape[0], block=shape[1], smem_stack=shape[2], instance_tree=1)
    return sc


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("n", [300, 100000], ids=["eight lanes", "one lane"])
def test_a_cycle_through_an_instance_is_ended(cuda_device, shape, n):
    r = api.Renderer(16, 16)
    sc = _scene(r, shape)
    rays = scenes.incoherent_rays(n, seed=7, tmax=10.0)
    ref = _scene(r, SHAPES[0])
    ref.set_trace_tuning(kernel=1, instance_tree=-1)
    hits, obj = sc.trace_closest(rays, with_obj=True)
    want, want_obj = ref.trace_closest(rays, with_obj=True)
    assert np.array_equal(np.asarray(hits).view(np.uint32), np.asarray(want).view(np.uint32)) and np.array_equal(obj, want_obj)
    # the root: infinite quanta over zero plane bytes (unbounded), slot 0 the
    # internal child 0 (itself), slot 1 a leaf with the first instance entry
    node = np.zeros(20, np.uint32)
    node[3] = 0x01FFFFFF
    node[6] = (0x20 | 24) | (0x20 << 8)
    sc.debug_write(3, 0, node.tobytes())
    with pytest.raises(capi.RayError) as e:
        sc.trace_closest(rays)
    assert e.value.code == capi.RAY_ERR_CUDA, e.value
    assert sc.last_trace_info().error_flags == 4  # the visit bound
