"""Served frames, whose captured waves fork a second stream in some of their bounces, equal the frames rendered directly:
waves small and large, one bounce and many, several samples a wave."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from renderer2_b200 import raytracer as R  # noqa: E402
from renderer2_b200 import render_scenes as RS  # noqa: E402
from renderer2_b200 import serving as S  # noqa: E402


@pytest.mark.parametrize("width,height,spp,depth", [(64, 48, 4, 1), (64, 48, 4, 60), (512, 512, 1, 1), (512, 512, 2, 8),
                                                    (512, 512, 2, 9), (640, 500, 3, 60), (1600, 1400, 4, 5)])
def test_served_frames_equal_rendered_ones(width, height, spp, depth):
    desc, _ = RS.icosphere_grid_scene()
    sc = RS.build_scene(desc)
    cam = R.camera(width, height, 45.0, (0, 0, 24), (0, 0, 0), (0, 1, 0))
    prms = [R.params(spp, depth, k) for k in range(3)]
    srv = S.Server(2, 8 << 30)
    jobs = [srv.submit_render(sc, cam, p) for p in prms]
    for j in jobs:
        srv.wait(j)
    srv.close()
    for j, p in zip(jobs, prms):
        assert np.array_equal(j.out, sc.render(cam, p))
    sc.close()


def test_many_bounces_of_a_small_frame_are_served_as_fast():
    """50 bounces of 64x64: a graph that forked in each of them took five times the direct frame, one without forks takes
    1.6 times it."""
    import time
    desc, _ = RS.icosphere_grid_scene()
    sc = RS.build_scene(desc)
    cam, prm = R.camera(64, 64, 45.0, (0, 0, 24), (0, 0, 0), (0, 1, 0)), R.params(4, 50, 1)
    srv = S.Server(1, 8 << 30)

    def best(run):
        times = []
        for _ in range(12):
            t = time.perf_counter()
            run()
            times.append(time.perf_counter() - t)
        return min(times)

    served, direct = best(lambda: srv.wait(srv.submit_render(sc, cam, prm))), best(lambda: sc.render(cam, prm))
    srv.close()
    sc.close()
    assert served <= 3.0 * direct, (served, direct)
