"""A path tracer's queues across frames of growing and shrinking size and changes between the
host-driven loop and the graphs: the second shadow queue of the forked graph is as large as the
first queue, whichever frame made it."""
import numpy as np
import pytest

from tests.test_pt import small_mixed_scene


@pytest.mark.gpu
@pytest.mark.parametrize("frames", [((96, 64, 0), (17, 9, 2), (64, 48, 2)), ((17, 9, 2), (96, 64, 2), (64, 48, 0)),
                                    ((96, 64, 2), (1, 1, 1), (33, 31, 2))])
def test_queues_fit_every_frame(cuda, frames):
    from imbatracer_b200 import native as N
    from imbatracer_b200.integrators import GpuScene, PathTracer
    gs = GpuScene(small_mixed_scene())
    kept = PathTracer(gs, max_path_len=5)
    for k, (w, h, graphs) in enumerate(frames):
        N.check(N.load().imbart_pt_set_graphs(kept.ctx, graphs), "imbart_pt_set_graphs")
        got = kept.render(2, 40 + k, w, h).cpu().numpy().astype(np.float64)
        new = PathTracer(gs, max_path_len=5, graphs=0)
        ref = new.render(2, 40 + k, w, h).cpu().numpy().astype(np.float64)
        assert np.array_equal(kept.last_stats[:2], new.last_stats[:2])
        # At most 2 samples * 5 bounces * 2 float32 terms a pixel, in another order: each sum is off
        # by 2^-24 of the pixel a term.
        assert (np.abs(got - ref) <= 20 * 2.0 ** -23 * np.maximum(got, ref)).all()
        new.close()
    kept.close()
