"""GPU: scenes of at most 64 triangles and 16 spheres take the path kernel; it
returns the queue kernels' images bit for bit (a render that names a
closest-hit variant runs those) and their adjoint within the rounding of sums
in another order."""
import numpy as np
import pytest

import mcrt_gb300 as M

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def soup(n_tri, n_sph, seed, scale=1.0, shift=0.0):
    """Triangles of sizes from 0.02 to 2 and spheres in a cube, with every material; slot 4 emits."""
    rng = np.random.default_rng(seed)
    md = M.materials([(0, (0.7, 0.6, 0.5), 0, 1), (1, (0.8, 0.8, 0.9), 0.2, 1), (2, (1, 1, 1), 0, 1.5),
                      (4, (0.9, 0.7, 0.4), 0.3, 1), (3, (4, 3, 2), 0, 1.0)])
    V = np.zeros(3 * n_tri, M.VERTEX)
    T = np.zeros(n_tri, M.TRIANGLE)
    c = rng.uniform(-1, 1, (n_tri, 1, 3))
    e = rng.standard_normal((n_tri, 3, 3)) * (0.02 * 100 ** rng.random((n_tri, 1, 1)))
    P = ((c + e) * scale + shift).astype(np.float32)
    N = np.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
    N /= np.maximum(np.linalg.norm(N, axis=1, keepdims=True), 1e-20)
    V["position"][:, :3], V["position"][:, 3] = P.reshape(-1, 3), 1.0
    V["normal"][:, :3] = np.repeat(N, 3, 0)
    T["v"] = np.arange(3 * n_tri).reshape(-1, 3)
    T["mat_idx"] = rng.integers(0, 5, n_tri) | (rng.integers(0, 2, n_tri).astype(np.uint32) << 31)
    S = np.zeros(n_sph, M.SPHERE)
    for k in range(n_sph):
        S[k]["center_r"] = (*(rng.uniform(-1, 1, 3) * scale + shift), rng.uniform(0.05, 0.4) * scale)
        S[k]["mat_and_pad"][0] = k % 5
    return dict(materials=md, vertices=V if n_tri else None, triangles=T if n_tri else None, spheres=S if n_sph else None)


def camera(w, h, scale=1.0, shift=0.0):
    return M.compute_camera(w, h, np.float32([0.3, 0.4, 3.5]) * scale + np.float32(shift), np.float32([0, 0, 0]) + np.float32(shift),
                            45.0, 0.02 * scale, 3.0 * scale)


@pytest.mark.parametrize("n_tri,n_sph", [(0, 0), (0, 3), (1, 0), (2, 1), (31, 0), (32, 2), (33, 0), (63, 16), (64, 0), (65, 1), (20, 17)])
@pytest.mark.parametrize("nee", [False, True])
def test_images_equal_the_queue_kernels(ctx, n_tri, n_sph, nee):
    ctx.upload_scene(env=M.gradient_env_map(), **soup(n_tri, n_sph, 100 + n_tri))
    for w, h, spp, graph in ((1, 1, 1, False), (37, 23, 5, True), (97, 61, 3, False)):
        got = ctx.render(camera(w, h), w, h, spp, max_depth=9, nee=nee, spp_per_pass=2, graph=graph)
        assert ctx.timings()["shade_ms"] == 0.0 or n_tri > 64 or n_sph > 16
        want = ctx.render(camera(w, h), w, h, spp, max_depth=9, nee=nee, spp_per_pass=2, variant=0)
        for k in ("rgba", "sum", "gbuf"):
            assert np.array_equal(bits(got[k]), bits(want[k])), (k, w, h)


@pytest.mark.parametrize("scale,shift", [(1e-3, 0.0), (1e4, 0.0), (1.0, 3000.0)])
def test_scales_and_places(ctx, scale, shift):
    """The conservative test's tolerance follows the scene's size and its distance from the origin."""
    ctx.upload_scene(env=M.gradient_env_map(), sun_dir=[0.3, 0.8, 0.2], sun_irradiance=[2, 2, 2], **soup(50, 0, 7, scale, shift))
    cam = camera(400, 300, scale, shift)
    got = ctx.render(cam, 400, 300, 1, max_depth=6, nee=True)
    want = ctx.render(cam, 400, 300, 1, max_depth=6, nee=True, variant=0)
    assert np.array_equal(bits(got["rgba"]), bits(want["rgba"]))


def test_large_pass_and_views(ctx):
    """A pass of the one-block-per-SM form, with views of uneven sizes."""
    ctx.upload_scene(env=M.gradient_env_map(), **soup(40, 0, 3))
    views = [(camera(w, h), w, h) for w, h in ((301, 207), (17, 430), (256, 256))]
    got = ctx.render_views(views, 4, max_depth=7, nee=True)
    for (cam, w, h), img in zip(views, got):
        want = ctx.render(cam, w, h, 4, max_depth=7, nee=True, variant=0)["rgba"]
        assert np.array_equal(bits(img), bits(want))


def test_degenerate_triangle_and_inflated_boxes_keep_the_tree(ctx):
    """A triangle of no area, and a given BVH whose child boxes reach beyond their parent's."""
    s = soup(12, 0, 5)
    s["vertices"]["position"][3:6] = s["vertices"]["position"][3]
    ctx.upload_scene(env=M.gradient_env_map(), **s)
    got = ctx.render(camera(64, 48), 64, 48, 4, nee=True)
    assert np.array_equal(bits(got["rgba"]), bits(ctx.render(camera(64, 48), 64, 48, 4, nee=True, variant=0)["rgba"]))
    s = soup(12, 0, 6)
    ctx.upload_scene(env=M.gradient_env_map(), **s)
    nodes, order = ctx.mesh_bvh()
    nodes["aabb_max"][0, 0] -= np.float32(0.7)
    ctx.upload_scene(env=M.gradient_env_map(), materials=s["materials"], vertices=s["vertices"], triangles=s["triangles"][order],
                     mesh_bvh=nodes, triangle_order=order)
    got = ctx.render(camera(64, 48), 64, 48, 4, nee=True)
    assert ctx.timings()["shade_ms"] > 0.0
    assert np.array_equal(bits(got["rgba"]), bits(ctx.render(camera(64, 48), 64, 48, 4, nee=True, variant=0)["rgba"]))


@pytest.mark.parametrize("n_tri,n_sph,w,h", [(33, 2, 31, 17), (64, 0, 200, 150)])
def test_adjoint_equals_the_queue_kernels(ctx, n_tri, n_sph, w, h):
    """Float sums over 32 lanes and doubles above them on both sides: 1e-5 of the largest component."""
    ctx.upload_scene(env=M.gradient_env_map(), **soup(n_tri, n_sph, 11))
    d = np.random.default_rng(1).standard_normal((h, w, 4)).astype(np.float32)
    ref = dict(max_depth=6, nee=True)
    got, img = ctx.adjoint(camera(w, h), w, h, 16, d, with_image=True, **ref)
    o = M._native.RenderOpts(max_depth=6, flags=M._native.RENDER_NEE, variant=1)
    import ctypes
    want = np.zeros(256, np.float64)
    want_img = np.zeros((h, w, 4), np.float32)
    cam = camera(w, h)
    M.check(M.lib().mcrt_adjoint(ctx._h, M.ptr(cam), w, h, 16, 0, ctypes.byref(o), M.ptr(d), M.ptr(want), M.ptr(want_img)), ctx._h)
    want = want.reshape(64, 4)
    assert np.array_equal(bits(img), bits(want_img))
    assert np.array_equal(got != 0, want != 0)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


def queue_adjoint(ctx, cam, w, h, spp, d, **kw):
    """The adjoint with a named closest-hit variant: the queue kernels."""
    import ctypes
    o = M._native.RenderOpts(max_depth=kw["max_depth"], flags=M._native.RENDER_NEE if kw["nee"] else 0, variant=1)
    grad, img = np.zeros(256, np.float64), np.zeros((h, w, 4), np.float32)
    M.check(M.lib().mcrt_adjoint(ctx._h, M.ptr(cam), w, h, spp, 0, ctypes.byref(o), M.ptr(d), M.ptr(grad), M.ptr(img)), ctx._h)
    return grad.reshape(64, 4), img


# passes of 272,384 paths (two rounds of 896 per SM) and fewer take the small blocks and more scenes
@pytest.mark.parametrize("n_tri,n_sph,w,h,spp,nee", [(64, 0, 100, 75, 16, True), (20, 16, 100, 75, 16, False),
                                                    (40, 0, 256, 256, 8, True), (1, 0, 256, 200, 8, False)])
def test_adjoint_of_both_path_kernel_forms(ctx, n_tri, n_sph, w, h, spp, nee):
    """Sums of at most 2^13 float terms per block and parameter, of either sign, in another order (the queue kernels'
    blocks): a random walk of 2^-24 of the partial sums, 2^6.5 x 2^-24 = 5e-6 of the result; doubles above them."""
    ctx.upload_scene(env=M.gradient_env_map(), **soup(n_tri, n_sph, 11))
    d = np.random.default_rng(1).standard_normal((h, w, 4)).astype(np.float32)
    cam = camera(w, h)
    got, img = ctx.adjoint(cam, w, h, spp, d, max_depth=6, nee=nee, with_image=True)
    assert ctx.timings()["render_launches"] == 3               # paths, resolve, replay
    want, want_img = queue_adjoint(ctx, cam, w, h, spp, d, max_depth=6, nee=nee)
    assert ctx.timings()["render_launches"] > 12
    assert np.array_equal(bits(img), bits(want_img))
    assert np.array_equal(got != 0, want != 0)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("depth,nee,path", [(1, False, False), (1, True, False), (2, False, True), (2, True, False), (3, True, True)])
def test_large_passes_of_short_paths(ctx, depth, nee, path):
    """Paths of one segment (two with next-event estimation) go through the queue kernels when there are many."""
    from mcrt_gb300 import scenes
    sc = scenes.cornell_box(3)
    c = sc["camera"]
    ctx.upload_scene(vertices=sc["vertices"], triangles=sc["triangles"], materials=sc["materials"], env=M.gradient_env_map())
    for spp in (1, 16):
        cam = M.compute_camera(160, 120, c["look_from"], c["look_at"], c["vfov"], 0.0)
        got = ctx.render(cam, 160, 120, spp, max_depth=depth, nee=nee)
        assert (ctx.timings()["shade_ms"] == 0.0) == (path or spp == 1)
        want = ctx.render(cam, 160, 120, spp, max_depth=depth, nee=nee, variant=0)
        for k in ("rgba", "sum", "gbuf"):
            assert np.array_equal(bits(got[k]), bits(want[k])), k


def test_table_follows_the_geometry(ctx):
    """The path kernel's table after new vertices: refused beyond coordinates of 1e9, taken again after them; a scene
    without triangles, from one graph to the other."""
    s = soup(20, 0, 9)
    ctx.upload_scene(env=M.gradient_env_map(), **s)
    far = s["vertices"].copy()
    far["position"][:3, :3] *= np.float32(4e9)
    for v, path in ((None, True), (far, False), (s["vertices"], True)):
        if v is not None:
            ctx.update_vertices(v)
        got = ctx.render(camera(40, 30), 40, 30, 2, nee=True)["rgba"]
        assert (ctx.timings()["shade_ms"] == 0.0) == path
        assert np.array_equal(bits(got), bits(ctx.render(camera(40, 30), 40, 30, 2, nee=True, variant=0)["rgba"]))
    ctx.upload_scene(env=M.gradient_env_map(), **soup(0, 3, 9))
    imgs = [ctx.render(camera(40, 30), 40, 30, 4, nee=True, spp_per_pass=2, graph=True, variant=v)["rgba"] for v in (None, 0, None)]
    assert np.array_equal(bits(imgs[0]), bits(imgs[1])) and np.array_equal(bits(imgs[0]), bits(imgs[2]))
