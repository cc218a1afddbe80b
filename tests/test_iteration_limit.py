"""max_iterations stops a render after whole runs of iters_per_graph iterations, whatever the
number of iterations a graph body holds."""
import pytest

import fumeng_b200 as fb
from fumeng_b200 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("profile", [False, True])
def test_limit_is_counted_in_runs_of_the_given_length(ctx, profile):
    spec = synth.cornell(res=32)
    scene = ctx.create_scene(spec.to_desc())

    def passes(iters, limit):
        try:
            ctx.render_batch([scene], [spec.camera_struct()], [spec.render_params(spp=2, seed=4)], profile=profile,
                             tuning=fb.Tuning(1 << 12, 128, 128, iters, limit, 0))
            return True
        except fb.FumengError as e:
            assert e.status == fb.FM_ERR_TIMEOUT
            return False
    try:
        # runs a limit allows: timed renders have always had one more
        extra = 1 if profile else 0
        need = next(n for n in range(1, 64) if passes(1, n)) + extra   # iterations the render takes
        assert 4 <= need <= 12   # a sample's start, at most five bounces of 2048 samples in 2048 slots, its end
        for iters in (2, 3, 4, 5, 7):
            for limit in range(1, need + 3):
                runs = (limit + iters - 1) // iters + extra
                assert passes(iters, limit) == (runs * iters >= need), (iters, limit, need)
    finally:
        scene.destroy()
