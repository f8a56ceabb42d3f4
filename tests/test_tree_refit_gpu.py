"""The instance tree over instances that a transform with infinities or NaN
places nowhere (how a program hides one), freshly built and refitted from
finite boxes: the finite instances' hits equal the walk that tests every
instance in turn, bit for bit, for rays with one, two and no zero direction
component, eight lanes to a ray and one."""
import numpy as np
import pytest

from raydemo_b200 import api, scenes

pytestmark = pytest.mark.gpu

N_INST = 40


def _xforms():
    rng = np.random.default_rng(17)
    out = np.tile(np.eye(4, dtype=np.float32), (N_INST, 1, 1))
    for x in out:
        x[0, 0] = x[1, 1] = x[2, 2] = rng.uniform(0.2, 0.5)
        x[3, :3] = rng.uniform(0.0, 2.0, 3)
    return out


def _rays(n):
    """Every third ray with one zero direction component, every third along an axis."""
    r = scenes.incoherent_rays(n, seed=71, tmax=10.0)
    r[:, 0:3] *= 2.5
    k = np.arange(n)
    r[k % 3 == 0, 4 + k[k % 3 == 0] % 2] = 0.0
    along = k[k % 3 == 1]
    r[along, 4:7] = 0.0
    r[along, 4 + along % 2 * 2] = np.where(along % 4 < 2, 1.0, -1.0)
    return r


def _scene(r, xf, tree):
    attrs, idx = scenes.triangle_soup_mesh(scenes.random_triangles(500, seed=18, mean_edge=0.1))
    sc = r.CreateScene()
    m = sc.AddMaterial()
    mesh = sc.AddMesh(attrs, idx, [(m, 0, len(idx))])
    for x in xf:
        sc.AddMeshInstance(mesh, x.reshape(-1))
    sc.set_trace_tuning(instance_tree=tree)
    return sc


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("refit", [False, True], ids=["build", "refit"])
@pytest.mark.parametrize("n", [900, 60000], ids=["eight lanes", "one lane"])
def test_finite_instances_beside_a_non_finite_one(cuda_device, value, refit, n):
    r = api.Renderer(16, 16)
    finite = _xforms()
    moved = finite.copy()
    for k in (3, 21):
        moved[k, 3, 0] = value
    rays = _rays(n)
    tree = _scene(r, finite if refit else moved, 1)
    if refit:
        tree.trace_closest(rays)
        for k in (3, 21):
            tree.SetMeshInstanceTransform(k, moved[k].reshape(-1))
    flat = _scene(r, moved, -1)
    hits, obj = tree.trace_closest(rays, with_obj=True)
    assert tree.last_trace_info().error_flags == 0
    info = tree.instance_tree_info()
    assert info.instances == N_INST and bool(info.refit) == refit
    want, want_obj = flat.trace_closest(rays, with_obj=True)
    axis = (rays[:, 4:7] == 0.0).any(axis=1)
    assert (want["prim"][axis] >= 0).sum() > n // 20
    assert np.array_equal(np.ascontiguousarray(hits).view(np.uint32), np.ascontiguousarray(want).view(np.uint32))
    assert np.array_equal(obj, want_obj)
    # and back: the next refit has finite boxes again
    if refit:
        for k in (3, 21):
            tree.SetMeshInstanceTransform(k, finite[k].reshape(-1))
        hits, obj = tree.trace_closest(rays, with_obj=True)
        want, want_obj = _scene(r, finite, -1).trace_closest(rays, with_obj=True)
        assert np.array_equal(np.ascontiguousarray(hits).view(np.uint32), np.ascontiguousarray(want).view(np.uint32))
        assert np.array_equal(obj, want_obj)
