"""GPU: the kernels that scenes beyond the path kernel's size run.  The Cornell boxes of the other tests are traced
whole by the path kernel; split into more triangles, the same boxes go through the queue kernels (and their cached and
adjoint forms), against the oracle on the same triangles."""
import numpy as np
import pytest

import mcrt_gb300 as M
from mcrt_gb300 import scenes

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def split(sc):
    """Every triangle cut into four at its edges' midpoints (flat shading: the corners' normals are equal)."""
    P, F = sc["vertices"], sc["triangles"]["v"].astype(np.int64)
    c = [P[F[:, k]] for k in range(3)]

    def mid(a, b):
        m = a.copy()
        m["position"][:, :3] = 0.5 * (a["position"][:, :3] + b["position"][:, :3])
        return m

    m01, m12, m20 = mid(c[0], c[1]), mid(c[1], c[2]), mid(c[2], c[0])
    parts = [(c[0], m01, m20), (m01, c[1], m12), (m20, m12, c[2]), (m01, m12, m20)]
    V = np.concatenate([np.stack(p, 1).reshape(-1) for p in parts])
    T = np.tile(sc["triangles"], 4)
    T["v"] = np.arange(len(V)).reshape(-1, 3)
    assert len(T) > 64
    return dict(vertices=V, triangles=T, materials=sc["materials"], env=M.gradient_env_map())


def camera(sc, w, h):
    c = sc["camera"]
    return M.compute_camera(w, h, c["look_from"], c["look_at"], c["vfov"], 0.0)


def constant_cache(ctx, value):
    p = np.zeros(ctx.cache_params().size, np.float32)
    p[-16:-13] = value                              # output bias
    ctx.cache_set_params(p)


@pytest.mark.parametrize("nee", [False, True])
def test_cache_stop_bit_exact(ctx, oracle, nee):
    """Paths stopped at their second vertex into a cache that predicts a constant, one path in seven traced in full."""
    sc = scenes.cornell_box(5)
    s, cam = split(sc), camera(sc, 48, 40)
    ctx.upload_scene(**s)
    ctx.cache_config(query_vertex=1, train_stride=7, train_steps=0, lr=0.0)
    const = np.array([0.3, 0.2, 0.1], np.float32)
    constant_cache(ctx, const)
    r = ctx.render(cam, 48, 40, 6, max_depth=8, nee=nee, spp_per_pass=3, cache=True)
    assert ctx.timings()["shade_ms"] > 0.0
    o = oracle.OracleScene(**s).render_cache_const(cam, 48, 40, 6, const, 3, 7, 1, max_depth=8, nee=nee)
    assert np.array_equal(bits(r["rgba"]), bits(o["rgba"]))
    assert np.array_equal(r["sum"].view(np.uint64), o["sum"].view(np.uint64))


@pytest.mark.parametrize("train_steps", [0, 3])
def test_cached_render_and_training_records_of_both_forms(ctx, train_steps):
    """One scene through the path kernel and, with a named variant, through the queue kernels: the same image, and the
    same training samples as the bias judge sums them up (in another order: float sums of 32 terms of one sign, five
    roundings each, above and below the quotient; doubles above them)."""
    sc = scenes.cornell_box(1234)
    cam = camera(sc, 64, 48)
    ctx.upload_scene(vertices=sc["vertices"], triangles=sc["triangles"], materials=sc["materials"], env=M.gradient_env_map())
    out = []
    for variant in (None, 0):
        ctx.cache_config(query_vertex=2, train_stride=5, train_steps=train_steps, train_batch=2048, lr=0.0)
        constant_cache(ctx, 20.0)                   # far above the scene's radiance: differences of one sign
        r = ctx.render(cam, 64, 48, 8, max_depth=8, nee=True, spp_per_pass=4, cache=True, variant=variant)
        assert (ctx.timings()["shade_ms"] > 0.0) == (variant is not None)
        out.append((r, ctx.cache_stats()))
    (a, sa), (b, sb) = out
    assert np.array_equal(bits(a["rgba"]), bits(b["rgba"])) and np.array_equal(a["sum"], b["sum"])
    assert sa["samples"] == sb["samples"] > 1000 and sa["stopped"] and sb["stopped"]
    assert np.allclose(sa["bias"], sb["bias"], rtol=16 * 2.0 ** -24, atol=0)


@pytest.mark.parametrize("name,nee", [("cornell", True), ("cornell_ggx", True), ("cornell_ggx", False)])
def test_adjoint_matches_bruteforce_gradient(ctx, oracle, name, nee):
    """The queue kernels' replay against forward-mode differentiation of the same sampled paths in double precision,
    within the bounds of the smaller scenes' test (test_gpu_adjoint.py: the same estimator on the same surfaces)."""
    sc = scenes.cornell_box(7) if name == "cornell" else scenes.cornell_box_ggx(1234)
    s, w, h, spp = split(sc), 40, 32, 6
    cam = camera(sc, w, h)
    ctx.upload_scene(**s)
    d = np.random.default_rng(2).standard_normal((h, w, 4)).astype(np.float32)
    g, img = ctx.adjoint(cam, w, h, spp, d, first_frame=11, max_depth=8, nee=nee, with_image=True)
    assert ctx.timings()["render_launches"] > 8     # three kernels and more per bounce
    osc = oracle.OracleScene(**s)
    want, _ = osc.adjoint(cam, w, h, spp, d, first_frame=11, max_depth=8, nee=nee)
    assert np.array_equal(bits(img), bits(osc.render(cam, w, h, spp, first_frame=11, max_depth=8, nee=nee)["rgba"]))
    scale = np.abs(want).max()
    assert scale > 0
    assert np.all(np.abs(g - want) <= 2e-4 * scale + 2e-3 * np.abs(want)), np.abs(g - want).max() / scale
    assert np.array_equal(g != 0, want != 0)


def test_sharing_does_little_useless_work(ctx):
    """Idle lanes take over subtrees of busy rays.  In a voxel world most of those lie behind the ray's hit: a frame of
    few paths, whose queues are shared, may visit at most a quarter more nodes per ray than a frame of many."""
    sc = scenes.voxel_world(3, 256, 128, 256)
    ctx.world_generate(sc["params"])
    ctx.world_mesh(sc["block_material"], sc["voxel_size"], greedy=False)
    ctx.upload_scene(materials=sc["materials"], env=M.gradient_env_map(), sun_dir=sc["sun_dir"],
                     sun_irradiance=sc["sun_irradiance"], world_mesh=True)
    cam = camera(sc, 320, 180)

    def nodes_per_ray(spp):
        ctx.render(cam, 320, 180, spp, max_depth=6, nee=True, outputs=(), count=True)
        t = ctx.timings()
        return t["node_fetches"] / t["rays"]

    assert nodes_per_ray(2) <= 1.25 * nodes_per_ray(64)
