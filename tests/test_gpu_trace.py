"""Closest hits of the caller's rays: sizes around the limits of the queue walk, own tmin and tmax per ray."""
import numpy as np
import pytest

import mcrt_gb300 as M
from test_gpu_parity import bits, random_scene_rays

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(oracle):
    rng = np.random.default_rng(11)
    spheres = np.zeros(60, M.SPHERE)
    spheres["center_r"][:, :3] = rng.uniform(-3, 3, (60, 3))
    spheres["center_r"][:, 3] = rng.uniform(0.05, 0.4, 60)
    n = 3000
    v = np.zeros(3 * n, M.VERTEX)
    v["position"][:, :3] = (rng.uniform(-3, 3, (n, 1, 3)) + rng.uniform(-0.2, 0.2, (n, 3, 3))).reshape(-1, 3)
    v["position"][:, 3] = 1
    v["normal"][:, 1] = 1
    t = np.zeros(n, M.TRIANGLE)
    t["v"] = np.arange(3 * n).reshape(n, 3)
    md = M.materials([(0, (0.5, 0.5, 0.5), 0, 1)])
    ctx = M.Context(0)
    ctx.upload_scene(spheres=spheres, vertices=v, triangles=t, materials=md)
    yield ctx, oracle.OracleScene(materials=md, spheres=spheres, vertices=v, triangles=t)
    ctx.close()


# a ray per warp, the host's and the kernel's check of tmin (4,096), a queue that fills the grid
# and one of more than eight rays per lane (152 SMs x 12 blocks x 64 lanes)
@pytest.mark.parametrize("n", [1, 2, 33, 4096, 4097, 150001, 8 * 152 * 12 * 64 + 5])
def test_trace_sizes_and_ranges(scene, n):
    ctx, osc = scene
    rng = np.random.default_rng(n)
    rays = random_scene_rays(rng, max(n, 64))[:n]
    rays["tmin"] = rng.choice([1e-3, 0.5, 2.0], n)
    rays["tmax"] = rng.choice([0.7, 3.0, 1e9, np.inf], n)
    got, want = ctx.trace_closest(rays), osc.trace(rays)
    assert np.array_equal(got["prim"], want["prim"])
    assert np.array_equal(bits(got["t"]), bits(want["t"]))
    tri = got["prim"] < 3000
    for f in ("u", "v"):
        assert np.array_equal(bits(got[f][tri]), bits(want[f][tri]))


@pytest.mark.parametrize("n", [5, 4096, 4097, 20000])
@pytest.mark.parametrize("bad", [0.0, -1.0, np.nan])
def test_trace_refuses_a_ray_without_positive_tmin(scene, n, bad):
    ctx, osc = scene
    rays = random_scene_rays(np.random.default_rng(n), max(n, 64))[:n]
    rays["tmin"][n - 2] = bad
    with pytest.raises(M.MCRTError):
        ctx.trace_closest(rays)
    rays["tmin"][n - 2] = 1e-3
    assert np.array_equal(ctx.trace_closest(rays)["prim"], osc.trace(rays)["prim"])


# the host looks at tmin up to 8,192 rays, the kernel above
@pytest.mark.parametrize("layout", [False, True])
@pytest.mark.parametrize("n", [8192, 8193])
def test_trace_checks_tmin_on_both_sides_of_the_limit(scene, n, layout):
    ctx, osc = scene
    rays = random_scene_rays(np.random.default_rng(n), n)
    rays["tmin"][n - 1] = -1e-3
    with pytest.raises(M.MCRTError):
        ctx.trace_closest(rays, reference_layout=layout)
    rays["tmin"][n - 1] = 1e-3
    got, want = ctx.trace_closest(rays, reference_layout=layout), osc.trace(rays)
    assert np.array_equal(got["prim"], want["prim"]) and np.array_equal(bits(got["t"]), bits(want["t"]))


@pytest.mark.parametrize("n", [8, 16, 17])
def test_trace_few_rays(scene, n):
    """A warp to a ray, with late and with early sharing of its subtrees."""
    ctx, osc = scene
    rays = random_scene_rays(np.random.default_rng(n), 64)[:n]
    got, want = ctx.trace_closest(rays), osc.trace(rays)
    assert np.array_equal(got["prim"], want["prim"]) and np.array_equal(bits(got["t"]), bits(want["t"]))


# the kernel without a queue, around its blocks and the limit of the host's check
@pytest.mark.parametrize("n_tri,n_sph", [(1, 0), (4, 4), (0, 3)])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 8192, 8193])
def test_trace_scenes_of_single_leaves(ctx, oracle, n_tri, n_sph, n):
    rng = np.random.default_rng(n + n_tri)
    v, t, s = np.zeros(3 * n_tri, M.VERTEX), np.zeros(n_tri, M.TRIANGLE), np.zeros(n_sph, M.SPHERE)
    v["position"][:, :3], v["position"][:, 3], v["normal"][:, 1] = rng.uniform(-3, 3, (3 * n_tri, 3)), 1, 1
    t["v"] = np.arange(3 * n_tri).reshape(n_tri, 3)
    s["center_r"][:, :3], s["center_r"][:, 3] = rng.uniform(-2, 2, (n_sph, 3)), 0.8
    scene = dict(materials=M.materials([(0, (0.5, 0.5, 0.5), 0, 1)]), vertices=v if n_tri else None,
                 triangles=t if n_tri else None, spheres=s if n_sph else None)
    ctx.upload_scene(**scene)
    rays = random_scene_rays(rng, max(n, 64))[:n]
    for _ in range(2):                              # a second call: nothing left over from the first
        rays["org"] += np.float32(0.01)
        got, want = ctx.trace_closest(rays), oracle.OracleScene(**scene).trace(rays)
        assert np.array_equal(got["prim"], want["prim"]) and np.array_equal(bits(got["t"]), bits(want["t"]))
