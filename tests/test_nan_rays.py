"""Rays that hold a NaN hit nothing, cost nothing and leave the rays beside them alone, in the
three kernels that trace: one ray per lane, the ray stream, and the wavefront's."""
import time

import numpy as np
import pytest

import fumeng_b200 as fb
from fumeng_b200 import synth

NAN = np.float32(np.nan)
NEG_NAN = np.array([0xFFC00000], np.uint32).view(np.float32)[0]
# field of the ray and its value: origin and direction in each component, t_min, t_max
# (an upper bound that is NaN ends the ray only with its sign set, a lower one with it clear)
FIELDS = [(c, NAN) for c in (0, 1, 2, 4, 5, 6, 3)] + [(0, NEG_NAN), (5, NEG_NAN), (7, NEG_NAN)]


@pytest.fixture(scope="module")
def hit_scene(ctx):
    sc = ctx.create_scene(synth.hit_scene(5, level=4, spheres=6).to_desc())
    yield sc
    sc.destroy()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [300, 40000, 200000])   # one ray per lane, the same at full warps, the stream
def test_rays_with_a_nan_miss_among_others(hit_scene, n):
    rng = np.random.default_rng(n)
    good = synth.random_rays(rng, n, (-1.5, -1.5, -1.5), (1.5, 1.5, 1.5))
    obj, t = hit_scene.trace_closest(good)
    occ = hit_scene.trace_any(good)
    assert (obj >= 0).sum() > n // 4
    rays = good.copy()
    bad = np.arange(0, n, 3)
    for k, i in enumerate(bad):
        c, v = FIELDS[k % len(FIELDS)]
        rays[i, c] = v
    is_bad = np.zeros(n, bool)
    is_bad[bad] = True
    obj2, t2 = hit_scene.trace_closest(rays)
    occ2 = hit_scene.trace_any(rays)
    assert np.all(obj2[is_bad] == -1) and np.all(np.isposinf(t2[is_bad])) and not occ2[is_bad].any()
    assert np.array_equal(obj2[~is_bad], obj[~is_bad]) and np.array_equal(t2[~is_bad], t[~is_bad])
    assert np.array_equal(occ2[~is_bad], occ[~is_bad])
    obj3, t3 = hit_scene.trace_closest_noalloc(rays)
    assert np.array_equal(obj3, obj2) and np.array_equal(t3, t2)


@pytest.mark.gpu
def test_rays_with_a_nan_do_not_visit_the_mesh(ctx):
    """327,680 triangles: a ray that visited all of them would take thousands of times an
    ordinary ray's few dozen tests."""
    scene = ctx.create_scene(synth.single_mesh_hit_scene(level=7).to_desc())
    try:
        def best(rays):
            times = []
            for _ in range(4):
                t0 = time.perf_counter()
                scene.trace_closest(rays)
                times.append(time.perf_counter() - t0)
            return min(times)
        for n in (256, 200000):
            good = synth.random_rays(np.random.default_rng(n), n, (-1.5, -1.5, -1.5), (1.5, 1.5, 1.5))
            bad = good.copy()
            bad[:, 4:7] = np.nan
            assert best(bad) < 5 * best(good)
    finally:
        scene.destroy()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [fb.FM_MODE_WAVEFRONT, fb.FM_MODE_MEGAKERNEL])
def test_camera_at_nan_renders_black(ctx, mode):
    spec = synth.cornell(res=24)
    scene = ctx.create_scene(spec.to_desc())
    try:
        cam = spec.camera_struct()
        cam.pos[0] = float("nan")
        rgb, _, _, st = scene.render(cam, spec.render_params(spp=4, seed=1, mode=mode))
        assert st.paths == 24 * 24 * 4 and st.closest_rays == st.paths and st.shadow_rays == 0 and st.bounces == 0
        assert not rgb.any()
    finally:
        scene.destroy()
