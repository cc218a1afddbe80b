"""Renders on a device that is short of memory: an allocation refused at each place where the
wavefront workspace grows is an error or a smaller workspace, never a broken context.  The
refusals come from a bound on what a context's workspace may hold, not from a full device."""
import ctypes as C

import numpy as np
import pytest

import fumeng_b200 as fb
from fumeng_b200 import synth

SPECS = [synth.material_scene(3, res=96), synth.cornell(res=100, spp=9)]


class _Ctx:
    """A context of its own, with the bound and what the workspace holds."""

    def __enter__(self):
        self.ctx = fb.Context(0)
        self.scenes = []
        return self

    def __exit__(self, *a):
        for s in self.scenes:
            s.destroy()
        self.ctx.close()

    def scene(self, spec):
        self.scenes.append(self.ctx.create_scene(spec.to_desc()))
        return self.scenes[-1]

    def limit(self, nbytes):
        self.ctx.lib.fm_internal_limit_workspace(self.ctx.h, C.c_int64(nbytes))

    def workspace(self):
        """(device bytes, times the state was allocated, second set of ray records)."""
        out = (C.c_int64 * 3)()
        self.ctx.lib.fm_internal_workspace(self.ctx.h, out)
        return tuple(out)

    def batch(self, pool=1 << 16, spp=20):
        if not self.scenes:
            for s in SPECS:
                self.scene(s)
        return self.ctx.render_batch(self.scenes, [s.camera_struct() for s in SPECS],
                                     [s.render_params(spp=spp, seed=5) for s in SPECS], want_aov=True,
                                     tuning=fb.Tuning(pool, 128, 128, 4, 0, 0))


def _counts(stats):
    return stats.paths, stats.closest_rays, stats.shadow_rays, stats.bounces


def _same(a, b):
    """Images that differ only in the order of float additions, and equal ray counts."""
    assert _counts(a[3]) == _counts(b[3])
    for x, y in zip(a[:3], b[:3]):
        for p, q in zip(x, y):
            np.testing.assert_allclose(p, q, rtol=1e-5, atol=1e-6)


@pytest.fixture(scope="module")
def unlimited(fm_lib):
    with _Ctx() as c:
        images = c.batch()
        return images, c.workspace()


@pytest.mark.gpu
def test_a_workspace_that_could_not_be_made_is_made_later(unlimited):
    with _Ctx() as c:
        c.limit(1)
        for _ in range(2):
            with pytest.raises(fb.FumengError) as e:
                c.batch()
            assert e.value.status == fb.FM_ERR_OOM
            assert c.workspace() == (0, 0, 0)
        c.limit(0)
        _same(c.batch(), unlimited[0])


@pytest.mark.gpu
def test_a_refused_larger_pool_leaves_the_context_usable(unlimited):
    with _Ctx() as c:
        c.batch(pool=1 << 15)
        c.limit(2 * c.workspace()[0])
        for _ in range(2):
            with pytest.raises(fb.FumengError) as e:
                c.batch(pool=1 << 18, spp=80)
            assert e.value.status == fb.FM_ERR_OOM
        _same(c.batch(pool=1 << 15), unlimited[0])
        c.limit(0)
        _same(c.batch(), unlimited[0])


@pytest.mark.gpu
def test_renders_with_one_set_of_ray_records(unlimited):
    """Without room for the second set, the MIS and shadow rays of an iteration are resolved
    before shading queues the next ones into the same records."""
    images, (held, builds, second) = unlimited
    assert (builds, second) == (1, 1)
    with _Ctx() as c:
        c.limit(held - 1)
        got = c.batch()
        assert c.workspace()[1:] == (1, 0) and c.workspace()[0] < held
        _same(got, images)
        _same(c.batch(), images)
        assert c.workspace()[1:] == (1, 0)


@pytest.mark.gpu
def test_direct_lighting_rounds_count_towards_the_bound_of_a_wide_pool(fm_lib):
    """13.6 M samples would have 2^23 slots, whose ray records for six rounds take 12.5 GB."""
    with _Ctx() as c:
        spec = synth.cornell(res=1024)
        sc = c.scene(spec)
        p = spec.render_params(spp=13, seed=1)
        p.depth, p.direct_loop = 1, 6
        st = sc.render(spec.camera_struct(), p, want_aov=False)[3]
        assert st.paths == 1024 * 1024 * 13
        held = c.workspace()[0]
        assert 6e9 < held <= 8e9   # 2^22 slots


@pytest.mark.gpu
def test_a_wide_pool_that_does_not_fit_is_tried_once(fm_lib):
    """7.3 M samples have 2^22 slots.  Where those are refused, the render runs with the default
    ones, reports no error, and later renders keep the workspace (and its graph)."""
    spec = synth.cornell(res=1024)
    cam = spec.camera_struct()
    few, many = spec.render_params(spp=3, seed=1), spec.render_params(spp=7, seed=2)
    with _Ctx() as c:
        sc = c.scene(spec)
        want = sc.render(cam, many, want_aov=False)
        wide = c.workspace()
        for _ in range(2):
            sc.render(cam, many, want_aov=False)
            sc.render(cam, few, want_aov=False)
        assert c.workspace() == wide and wide[1] == 1
    with _Ctx() as c:
        sc = c.scene(spec)
        sc.render(cam, few, want_aov=False)
        narrow = c.workspace()
        assert narrow[0] < 0.6 * wide[0]
        c.limit(int(1.3 * narrow[0]))
        got = sc.render(cam, many, want_aov=False)
        assert c.ctx.lib.fm_last_error(c.ctx.h) == b""
        assert _counts(got[3]) == _counts(want[3])
        np.testing.assert_allclose(got[0], want[0], rtol=1e-5, atol=1e-6)
        after = c.workspace()
        assert after[1:] == (2, 1)
        for _ in range(2):
            sc.render(cam, many, want_aov=False)
            sc.render(cam, few, want_aov=False)
        assert c.workspace() == after
        c.limit(0)
        sc.render(cam, many, want_aov=False)
        assert c.workspace()[0] > 0.9 * wide[0]


@pytest.mark.gpu
def test_albedo_and_normal_sums_are_held_once_they_are_asked_for(fm_lib):
    spec = synth.material_scene(3, res=96)
    cam, p = spec.camera_struct(), spec.render_params(spp=20, seed=3)
    slots = 96 * 96 * 20
    with _Ctx() as c, _Ctx() as fresh:
        sc = c.scene(spec)
        plain = sc.render(cam, p, want_aov=False)
        lean, builds, _ = c.workspace()
        got = sc.render(cam, p, want_aov=True)
        full = c.workspace()
        assert builds == full[1] == 1   # beside the state, which stays
        # 32 B of sums per slot, and 32 B of partial sums per work item (four or more per slot,
        # or one per sample)
        assert full[0] - lean >= 64 * slots
        again = sc.render(cam, p, want_aov=False)
        assert c.workspace() == full
        want = fresh.scene(spec).render(cam, p, want_aov=True)
        for x in (plain, got, again):
            assert _counts(x[3]) == _counts(want[3])
            np.testing.assert_allclose(x[0], want[0], rtol=1e-5, atol=1e-6)
        for k in (1, 2):
            np.testing.assert_allclose(got[k], want[k], rtol=1e-5, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (40, 3), (3, 200), (513, 129), (1100, 140), (600, 300)])
def test_denoiser_in_tiles_gives_the_same_image(w, h, fm_lib):
    """Where 80 B per pixel are refused, the filter runs tile by tile (512 x 128)."""
    rng = np.random.default_rng(w + h)
    rgb = rng.gamma(2.0, 0.3, (h, w, 3)).astype(np.float32)
    rgb[h // 2, w // 2, 0] = np.inf
    alb = rng.uniform(0.4, 0.6, (h, w, 3)).astype(np.float32)
    nrm = (rng.normal(size=(h, w, 3)) * 0.2 + np.array([0, 0, 1.0])).astype(np.float32)
    chain = [(fb.FM_POST_TONEMAP, 1.1), (fb.FM_POST_DENOISE, 0.0), (fb.FM_POST_DENOISE, 0.0)]
    with _Ctx() as c:
        want = c.ctx.postprocess(chain, rgb, alb, nrm)
        c.limit(79)
        got = c.ctx.postprocess(chain, rgb, alb, nrm)
    for a, b in zip(want, got):
        assert np.array_equal(a, b, equal_nan=a.dtype == np.float32)
