"""Where the kernels change path or tile: ray queries at the sizes around the switch from one
ray per lane to the ray stream, the denoiser on images smaller than its tiles and taps,
wavefront renders over pool sizes, graph lengths and outputs, and transfers around the
pinned ring's chunk size."""
import numpy as np
import pytest

import fumeng_b200 as fb
from fumeng_b200 import synth

LANES = 148 * 1024   # rays in flight of a query that keeps one ray per lane


def _query_rays(n):
    """Random rays with every main axis the triangle test can choose (axis-aligned unit and
    longer directions), a t_min above 0 and a finite t_max among them."""
    rng = np.random.default_rng(9)
    r = synth.random_rays(rng, n, (-1.5, -1.5, -1.5), (1.5, 1.5, 1.5))
    k = np.arange(n)
    r[k % 7 == 0, 4:7] = np.eye(3, dtype=np.float32)[k[k % 7 == 0] % 3]
    r[k % 11 == 0, 4:7] *= 3.0
    r[k % 5 == 0, 3] = 0.3
    r[k % 3 == 0, 7] = 1.2
    return r


@pytest.fixture(scope="module")
def hit_scene(ctx):
    sc = ctx.create_scene(synth.hit_scene(5, level=4, spheres=6).to_desc())
    yield sc
    sc.destroy()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 4735, 4737, LANES - 1, LANES, LANES + 1, 2 * LANES + 77])
def test_queries_do_not_depend_on_the_batch(hit_scene, n):
    """The same rays one batch at a time and in pieces of 1000 give the same hits, bit for bit."""
    rays = _query_rays(n)
    obj, t = hit_scene.trace_closest(rays)
    occ = hit_scene.trace_any(rays)
    pieces = [rays[i:i + 1000] for i in range(0, n, 1000)]
    ref = [hit_scene.trace_closest(p) for p in pieces]
    assert np.array_equal(obj, np.concatenate([o for o, _ in ref]))
    assert np.array_equal(t, np.concatenate([x for _, x in ref]))
    assert np.array_equal(occ, np.concatenate([hit_scene.trace_any(p) for p in pieces]))
    if n <= 262144:
        o2, t2 = hit_scene.trace_closest_noalloc(rays)
        assert np.array_equal(obj, o2) and np.array_equal(t, t2)
    # an occlusion query sees a hit in the open range wherever the closest hit lies in it
    assert np.all(occ[(obj >= 0) & (t < rays[:, 7])] == 1)


def _denoise64(rgb, alb, nrm):
    rgb, alb, nrm = (np.asarray(a, np.float64) for a in (rgb, alb, nrm))
    h, w, _ = rgb.shape
    ln = np.linalg.norm(nrm, axis=-1, keepdims=True)
    nrm = np.where(ln > 0, nrm / np.where(ln > 0, ln, 1), nrm)
    k5 = np.array([1, 4, 6, 4, 1]) / 16.0
    for level in range(5):
        step, sc = 1 << level, 0.5 / (1 << level)
        t = rgb / (1 + np.maximum(rgb, 0))
        out = np.empty_like(rgb)
        for y in range(h):
            for x in range(w):
                acc, ws = np.zeros(3), 0.0
                for dy in range(-2, 3):
                    for dx in range(-2, 3):
                        yy, xx = y + dy * step, x + dx * step
                        if not (0 <= yy < h and 0 <= xx < w):
                            continue
                        wt = k5[dy + 2] * k5[dx + 2] * np.exp(
                            -np.sum((t[yy, xx] - t[y, x]) ** 2) / sc ** 2
                            - max(0.0, 1 - nrm[y, x] @ nrm[yy, xx]) / 0.35 ** 2
                            - np.sum((alb[yy, xx] - alb[y, x]) ** 2) / 0.1 ** 2)
                        acc += wt * rgb[yy, xx]
                        ws += wt
                out[y, x] = acc / ws
        rgb = out
    return rgb


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (1, 40), (40, 1), (5, 3), (31, 9), (33, 8), (64, 17)])
def test_denoise_small_and_ragged_images(ctx, w, h):
    """Against the filter in 64 bits.  A weight's exponent is at most about 300 here, so its
    float rounding (2^-24 each for some ten operations) moves a weight by 2e-4 at worst where
    the weight itself is negligible, and by 1e-5 where it counts; five passes of weighted
    means stay within 1e-4."""
    rng = np.random.default_rng(w * 100 + h)
    rgb = rng.gamma(2.0, 0.3, (h, w, 3)).astype(np.float32)
    alb = rng.uniform(0.4, 0.6, (h, w, 3)).astype(np.float32)
    nrm = (rng.normal(size=(h, w, 3)) * 0.2 + np.array([0, 0, 1.0])).astype(np.float32)
    nrm[0, 0] = 0.0
    out = ctx.postprocess([(fb.FM_POST_DENOISE, 0.0)], rgb, alb, nrm)[0]
    np.testing.assert_allclose(out, _denoise64(rgb, alb, nrm), rtol=1e-4, atol=1e-6)


@pytest.mark.gpu
def test_denoise_leaves_non_finite_pixels_out_of_their_neighbours(ctx):
    rgb = np.full((12, 40, 3), 0.5, np.float32)
    rgb[3, 4] = (np.inf, 1.0, 1.0)
    rgb[5, 20] = (np.nan, 0.0, 0.0)
    rgb[9, 30] = (3e38, 3e38, 3e38)   # finite channels, an infinite sum
    alb = np.full_like(rgb, 0.5)
    nrm = np.dstack([np.zeros((12, 40, 2)), np.ones((12, 40, 1))]).astype(np.float32)
    out = ctx.postprocess([(fb.FM_POST_DENOISE, 0.0)], rgb, alb, nrm)[0]
    ok = np.ones((12, 40), bool)
    ok[3, 4] = ok[5, 20] = ok[9, 30] = False
    np.testing.assert_allclose(out[ok], 0.5, rtol=1e-6)
    assert np.isinf(out[3, 4, 0]) and np.isnan(out[5, 20, 0])


@pytest.mark.gpu
@pytest.mark.parametrize("pool,iters,block", [(1024, 1, 32), (1023 * 8, 3, 64), (40000, 8, 128), (148 * 4096, 2, 256),
                                              (1 << 20, 7, 256)])
def test_wavefront_images_do_not_depend_on_the_tuning(ctx, pool, iters, block):
    """Slots per thread of the logic kernel (four from 148 * 4096 slots on), odd and even graph
    lengths, samples per work item, and kept or skipped albedo / normal sums change only the
    order in which a pixel's float contributions are added: a few tens of additions, so
    well within 1e-5 of the pixel's value (1e-6 for near-black ones)."""
    specs = [synth.material_scene(3, res=96), synth.cornell(res=100, spp=9)]
    scenes = ctx.create_scenes([s.to_desc() for s in specs])
    try:
        cams = [s.camera_struct() for s in specs]
        params = [s.render_params(spp=70, seed=5) for s in specs]
        ref = ctx.render_batch(scenes, cams, params, want_aov=True, tuning=fb.Tuning(1 << 21, 128, 128, 8, 0, 0))
        tun = fb.Tuning(pool, block, block, iters, 0, 0)
        for aov in (True, False):
            got = ctx.render_batch(scenes, cams, params, want_aov=aov, tuning=tun)
            assert got[3].paths == ref[3].paths and got[3].closest_rays == ref[3].closest_rays
            assert got[3].shadow_rays == ref[3].shadow_rays and got[3].bounces == ref[3].bounces
            for a, b in zip(got[0], ref[0]):
                np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6)
            if aov:
                for k in (1, 2):
                    for a, b in zip(got[k], ref[k]):
                        np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6)
    finally:
        for s in scenes:
            s.destroy()


@pytest.mark.gpu
def test_render_with_more_slots_is_the_mean_of_its_halves(ctx):
    """6.8 M samples (1.5 per slot of 2^22) in one render against two renders of half the
    samples, which keep the default slots."""
    spec = synth.cornell(res=512)
    scene = ctx.create_scene(spec.to_desc())
    try:
        cam = spec.camera_struct()
        whole = scene.render(cam, spec.render_params(spp=26, seed=2), want_aov=False)[0]
        a = scene.render(cam, spec.render_params(spp=13, seed=2), want_aov=False)[0]
        b = scene.render(cam, spec.render_params(spp=13, seed=2, sample_offset=13), want_aov=False)[0]
    finally:
        scene.destroy()
    np.testing.assert_allclose(whole, 0.5 * (a.astype(np.float64) + b), rtol=1e-5, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(7, 11), (512, 1365), (512, 1366), (700, 1999)])
def test_postprocess_around_the_ring_size(ctx, h, w):
    """Per-pixel steps of a large image (through the pinned ring from 8 MiB on) equal those of
    its rows in pieces, floats and bytes."""
    rng = np.random.default_rng(h)
    rgb = rng.gamma(1.0, 1.0, (h, w, 3)).astype(np.float32)
    alb = rng.random((h, w, 3)).astype(np.float32)
    chain = [(fb.FM_POST_TONEMAP, 1.1), (fb.FM_POST_LINEAR_TO_SRGB, 0.0)]
    out, c8, a8, _ = ctx.postprocess(chain, rgb, alb)
    cut = max(1, h // 5)
    for y in range(0, h, cut):
        o, c, a, _ = ctx.postprocess(chain, rgb[y:y + cut], alb[y:y + cut])
        assert np.array_equal(out[y:y + cut], o) and np.array_equal(c8[y:y + cut], c)
        assert np.array_equal(a8[y:y + cut], a)


@pytest.mark.gpu
def test_gradients_are_added_through_the_ring_and_beside_it(ctx):
    """Texture gradients of 12.6 MB (pinned ring) and 96 B: added to what the buffers hold, and
    the same on a second call up to the float-atomic order of the accumulators."""
    import ctypes as C
    for tex in (512, 2):
        spec = synth.inverse_scene(tex_res=tex, plane_n=8, sphere_nu=16, sphere_nv=8, res=24, spp=8, depth=3, target=False)
        holder = spec.to_desc()
        scene = ctx.create_scene(holder)
        try:
            ti = holder.texture_index
            p = spec.render_params(seed=1)
            d = [np.ones((24, 24, 3), np.float32)]
            shapes = {ti["basecolor"]: (tex, tex), ti["rm"]: (tex, tex)}
            g = scene.render_adjoint([spec.camera_struct()], [p], d, shapes)[0]
            buf = {k: np.full(s + (3,), 2.0) for k, s in shapes.items()}
            arr = (C.c_void_p * len(ti))(*[buf[k].ctypes.data if k in buf else None for k in range(len(ti))])
            gd = fb.GradDesc(arr, None)
            cam = (fb.Camera * 1)(spec.camera_struct())
            dp = (C.c_void_p * 1)(d[0].ctypes.data)
            ctx.check(ctx.lib.fm_render_adjoint(ctx.h, scene.h, 1, cam, (fb.RenderParams * 1)(p), dp, None, C.byref(gd), 0, None))
        finally:
            scene.destroy()
        for k in shapes:
            assert np.abs(g[k]).max() > 0
            np.testing.assert_allclose(buf[k] - 2.0, g[k], rtol=1e-4, atol=1e-5 * np.abs(g[k]).max())
