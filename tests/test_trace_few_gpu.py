"""Closest hits where a ray is traced by eight lanes: launches of few rays
(around the edges of a warp's four groups and of one wave of groups) and the
last rays of larger launches, over a single mesh, instances tested in turn and
the instance tree; rays parallel to the axes, whose zero direction components
the node step tests by containment; duplicate instances, whose ties go to the
lower index. The kernel with one thread per ray (set_trace_tuning kernel 1) and
the oracle's brute-force order are the references: every field bit for bit."""
import numpy as np
import pytest

from raydemo_b200 import api, scenes

pytestmark = pytest.mark.gpu

TRIS = scenes.random_triangles(3000, seed=7, mean_edge=0.05)


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _scene(r, xforms, tree):
    attrs, idx = scenes.triangle_soup_mesh(TRIS)
    sc = r.CreateScene()
    m = sc.AddMaterial()
    mesh = sc.AddMesh(attrs, idx, [(m, 0, len(idx))])
    for x in xforms:
        sc.AddMeshInstance(mesh, x)
    sc.set_trace_tuning(instance_tree=tree)
    return sc


def _xforms(n, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        x = np.eye(4, dtype=np.float32)
        x[0, 0] = x[1, 1] = x[2, 2] = rng.uniform(0.3, 0.6)
        x[3, :3] = rng.uniform(0.0, 1.0, 3)
        out.append(x.reshape(-1))
    return out


def _rays(n, seed):
    """Incoherent rays, every third one with one zero direction component,
    every seventh along an axis (with both signs of zero), and some origins on
    vertex coordinates."""
    r = scenes.incoherent_rays(n, seed=seed, tmax=5.0)
    k = np.arange(n)
    r[k % 3 == 0, 4] = 0.0
    r[k % 7 == 0, 4:7] = 0.0
    r[k % 7 == 0, 4 + 2] = np.where(k[k % 7 == 0] % 2 == 0, 1.0, -1.0)
    r[k % 14 == 0, 5] = -0.0
    on = k % 11 == 0
    r[on, 0] = TRIS.reshape(-1, 3)[k[on] % (3 * len(TRIS)), 0]
    return r


@pytest.fixture(scope="module")
def renderer(cuda_device):
    return api.Renderer(16, 16)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 33, 1000, 16575, 16577, 18945, 60001])
@pytest.mark.parametrize("kind", ["mesh", "turn", "tree"])
def test_few_rays_equal_the_one_thread_kernel(renderer, n, kind):
    xf = [np.eye(4, dtype=np.float32).reshape(-1)] if kind == "mesh" else _xforms(19, 3)
    rays = _rays(n, 100 + n)
    sc = _scene(renderer, xf, 1 if kind == "tree" else -1)
    for kernel in (3, 2):
        sc.set_trace_tuning(kernel=kernel, instance_tree=1 if kind == "tree" else -1)
        hits, obj = sc.trace_closest(rays, with_obj=True)
        assert sc.last_trace_info().error_flags == 0
        one = _scene(renderer, xf, -1)
        one.set_trace_tuning(kernel=1, instance_tree=-1)
        ref, ref_obj = one.trace_closest(rays, with_obj=True)
        assert np.array_equal(_bits(hits), _bits(ref)) and np.array_equal(obj, ref_obj)


def test_axis_parallel_rays_equal_the_oracle(renderer, oracle):
    rays = _rays(4000, 5)
    sc = _scene(renderer, [np.eye(4, dtype=np.float32).reshape(-1)], 0)
    hits = sc.trace_closest(rays)
    attrs, idx = scenes.triangle_soup_mesh(TRIS)
    exp = oracle.closest_hit_bvh(oracle.preprocess_tris(attrs[:, :3].copy(), idx), scenes.tri_aabbs(TRIS), rays)
    assert (exp["prim"] >= 0).sum() > 400
    assert np.array_equal(hits["prim"], exp["prim"])
    hit = exp["prim"] >= 0
    assert np.array_equal(_bits(hits[hit]), _bits(exp[hit]))


@pytest.mark.parametrize("n", [500, 50000])
def test_ties_between_instances_go_to_the_lower_index(renderer, n):
    """Every instance twice: each hit is the first of its pair's, in turn and in the tree."""
    xf = [x for x in _xforms(12, 9) for _ in (0, 1)]
    rays = _rays(n, 6)
    out = [_scene(renderer, xf, tree).trace_closest(rays, with_obj=True) for tree in (-1, 1)]
    assert np.array_equal(_bits(out[0][0]), _bits(out[1][0])) and np.array_equal(out[0][1], out[1][1])
    obj = out[1][1]
    assert (obj >= 0).sum() > n // 50 and np.all(obj[obj >= 0] % 2 == 0)
