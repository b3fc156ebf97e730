"""The GPU builder's trees against the reference builder's (oracle), at shapes where it can go wrong."""
import numpy as np
import pytest

import mcrt_gb300 as M
from test_gpu_parity import bits, leaf_sets

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = M.Context(0)
    yield c
    c.close()


def mesh(points):
    n = len(points)
    v = np.zeros(3 * n, M.VERTEX)
    v["position"][:, :3] = points.reshape(-1, 3)
    v["position"][:, 3] = 1
    v["normal"][:, 1] = 1
    t = np.zeros(n, M.TRIANGLE)
    t["v"] = np.arange(3 * n).reshape(-1, 3)
    return v, t


def build_both(ctx, oracle, points):
    v, t = mesh(points)
    ctx.upload_scene(vertices=v, triangles=t, materials=M.materials([(0, (0.5, 0.5, 0.5), 0, 1)]))
    nodes, order = ctx.mesh_bvh()
    want, _, ids = oracle.build_mesh_bvh(v, t)
    assert len(nodes) == len(want)
    for f in ("right_or_offset", "prim_count"):
        assert np.array_equal(nodes[f], want[f])
    assert leaf_sets(nodes, order) == leaf_sets(want, ids)
    return nodes, want


@pytest.mark.parametrize("n", [7, 40, 300, 4000])
def test_bvh_of_negative_zero_coordinates(ctx, oracle, n):
    """-0 is one of the smallest values a box can have, not the largest integer."""
    p = np.random.default_rng(n).integers(-2, 3, (n, 3, 3)).astype(np.float32)
    p[p == 0] *= np.float32(-1)
    nodes, want = build_both(ctx, oracle, p)
    for f in ("aabb_min", "aabb_max"):       # by value: which zero a box keeps is the order of its primitives
        assert np.array_equal(nodes[f], want[f])


def shape(kind, n, rng):
    if kind == "cloud":                      # balanced splits
        c = rng.uniform(-5, 5, (n, 1, 3))
    elif kind == "chain":                    # a few primitives leave per split: deep trees
        c = np.zeros((n, 1, 3))
        c[:, 0, 0] = 1.2 ** (np.arange(n) % 400)
        c[:, 0, 1] = 4 * (np.arange(n) // 400)
    else:                                    # clusters of equal triangles: leaves above the leaf size
        return rng.integers(0, 3, (max(n // 40, 1), 3, 3)).repeat(40, axis=0)[:n].astype(np.float32)
    return (c + rng.uniform(-0.4, 0.4, (n, 3, 3))).astype(np.float32)


# 4 | 5: leaf and smallest subtree; up to 8, 16, 32: tasks of a part of a warp; 256: of a warp; 1024: of one block;
# 2049 and above: two levels and more above the subtrees
@pytest.mark.parametrize("kind", ["cloud", "chain", "equal"])
@pytest.mark.parametrize("n", [4, 5, 8, 9, 16, 17, 32, 33, 128, 129, 257, 1023, 1024, 1025, 2049, 5000])
def test_bvh_sizes_around_the_subtree_limits(ctx, oracle, n, kind):
    nodes, want = build_both(ctx, oracle, shape(kind, n, np.random.default_rng(n)))
    for f in ("aabb_min", "aabb_max"):
        assert np.array_equal(bits(nodes[f]), bits(want[f]))


def test_triangles_in_one_place_take_two_levels(ctx, oracle):
    """No split of the root: a leaf of any size, found after the second of the levels (six launches each) that a mesh of
    this size would need."""
    rng = np.random.default_rng(2)
    n = 40000
    build_both(ctx, oracle, np.repeat(rng.uniform(-1, 1, (1, 3, 3)), n, 0).astype(np.float32))
    same = ctx.timings()["build_launches"]
    build_both(ctx, oracle, shape("cloud", n, rng))
    cloud = ctx.timings()["build_launches"]                     # six levels at least, and the subtrees
    assert same + 4 * 6 <= cloud
