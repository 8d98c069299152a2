"""Device memory that scenes keep: buffers that stay where they are between builds, and the state of large waves, which a
frame takes only while it is a small part of what is free and of the device."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import wide_probe  # noqa: E402
from renderer2_b200 import raytracer as R  # noqa: E402
from renderer2_b200 import render_scenes as RS  # noqa: E402

GB = 1 << 30


@pytest.mark.parametrize("large,more", [(1000, 10), (1000, 1000), (1000, 5000)])
def test_buffers_of_one_allocation_stay_in_place(large, more):
    """A builder that builds triangles and boxes by turns allocates in the first turn alone."""
    assert wide_probe.lib().probe_reserve_moves(large, more, 4) == 0


def _scene():
    desc, _ = RS.icosphere_grid_scene()
    return RS.build_scene(desc), R.camera(1024, 1024, 45.0, (0, 0, 24), (0, 0, 0), (0, 1, 0)), R.params(16, 4, 1)


def _render(sc, cam, prm):
    frame = torch.empty((cam.height, cam.width, 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    sc.render_device(cam, prm, frame.data_ptr())
    torch.cuda.synchronize()
    return frame, before - torch.cuda.mem_get_info()[0]


def test_large_waves_leave_a_nearly_full_device_alone():
    """16M paths take 3.6 GB; with 20 GB free a frame keeps to waves of 4M (0.9 GB), frame after frame, and the tuner
    too.  The frame is the same bit for bit."""
    sc, cam, prm = _scene()
    want, large = _render(sc, cam, prm)
    assert large > 2 * GB and sc.wave_samples(cam, prm) == 16
    sc.close()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - 20 * GB, dtype=torch.uint8, device="cuda")
    try:
        sc, cam, prm = _scene()
        got, small = _render(sc, cam, prm)
        assert small < 2 * GB and torch.equal(got, want)
        assert sc.wave_samples(cam, prm) == 4
        again, more = _render(sc, cam, prm)
        assert more <= 0 and torch.equal(again, want)
        before = torch.cuda.mem_get_info()[0]
        sc.autotune(cam, prm)
        tuned, _ = _render(sc, cam, prm)
        assert before - torch.cuda.mem_get_info()[0] < GB and torch.equal(tuned, want)
        sc.close()
    finally:
        del held
        torch.cuda.empty_cache()


def test_scenes_together_are_bounded():
    """However many scenes are rendered, their large waves take no more than an eighth of the device beyond what waves
    of 4M paths take, and a scene that is closed gives its share back."""
    total = torch.cuda.mem_get_info()[1]
    scenes, grew = [], []
    for _ in range(12):
        sc, cam, prm = _scene()
        grew.append(_render(sc, cam, prm)[1])
        scenes.append(sc)
    extra = sum(max(0, g - 1.1 * GB) for g in grew)
    assert max(grew) > 2 * GB and grew[-1] < 2 * GB and extra <= total / 8
    for sc in scenes:
        sc.close()
    sc, cam, prm = _scene()
    assert _render(sc, cam, prm)[1] > 2 * GB
    sc.close()


def test_a_failed_allocation_fails_one_call():
    """A frame whose smallest wave does not fit is refused for its memory; the next call is not."""
    from renderer2_b200 import _native as N
    sc, cam, prm = _scene()
    small = R.camera(64, 64, 45.0, (0, 0, 24), (0, 0, 0), (0, 1, 0))
    want, _ = _render(sc, small, prm)
    huge = R.camera(20000, 20000, 45.0, (0, 0, 24), (0, 0, 0), (0, 1, 0))  # 400M paths at one sample: 90 GB
    held = torch.empty(torch.cuda.mem_get_info()[0] - 20 * GB, dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(N.R2Error) as e:
            sc.render_device(huge, R.params(1, 2, 0), held.data_ptr())
        assert e.value.name == "R2_ERR_OUT_OF_MEMORY"
        got, _ = _render(sc, small, prm)
        assert torch.equal(got, want)
    finally:
        del held
        torch.cuda.empty_cache()
        sc.close()


def test_a_filter_job_is_admitted_with_the_work_space_it_takes():
    """A job of few voxels takes 256 KB to work in: a budget without room for that does not admit it."""
    from renderer2_b200 import _native as N
    from renderer2_b200 import filter as F
    from renderer2_b200 import scenes
    from renderer2_b200 import serving as S
    mesh = scenes.icosphere(2, 0.05, 1)
    sc = F.FilterScene(mesh, F.material())
    g = sc.grid(scenes.voxel_size_for(mesh, 8))
    nvox = int(np.prod(np.array(g.num_voxels[:], np.int64)))
    out = 32 * (1 << (nvox - 1).bit_length())
    for budget, fits in ((out + (1 << 18) + 64, True), (out + (1 << 17), False)):
        srv = S.Server(1, budget)
        if fits:
            srv.wait(srv.submit_filter(sc, g, F.params(samples_per_voxel=8, iterations=2)))
        else:
            with pytest.raises(N.R2Error) as e:
                srv.submit_filter(sc, g, F.params(samples_per_voxel=8, iterations=2))
            assert e.value.name == "R2_ERR_ADMISSION_REJECTED"
        srv.close()
    sc.close()


def test_a_served_frame_keeps_to_the_budget():
    """A scene tuned to large waves is served in waves of 4M paths where the budget has no room for them, with the same
    frame."""
    from renderer2_b200 import serving as S
    sc, cam, prm = _scene()
    want = _render(sc, cam, prm)[0].cpu().numpy()
    sc.set_tuning(R.tuning(wave_paths=1 << 24))
    assert S.Server.render_bytes(sc, cam, prm) > 2 * GB
    srv = S.Server(1, 2 * GB)
    job = srv.submit_render(sc, cam, prm)
    srv.wait(job)
    srv.close()
    sc.close()
    assert np.array_equal(job.out, want)


@pytest.mark.parametrize("spare", [1 << 30, 1 << 18], ids=["room", "tight"])
def test_a_served_filter_equals_a_direct_one(spare):
    """With the work space that suits the grid, and with the least, where the grid takes several parts."""
    from renderer2_b200 import _native as N
    from renderer2_b200 import filter as F
    from renderer2_b200 import scenes
    from renderer2_b200 import serving as S
    mesh = scenes.foliage(8000, 6, 0.7, 5)
    sc = F.FilterScene(mesh, F.material())
    g, prm = sc.grid(scenes.voxel_size_for(mesh, 37)), F.params(samples_per_voxel=32, iterations=3)
    nvox = int(np.prod(np.array(g.num_voxels[:], np.int64)))
    want = torch.empty(nvox * 32, dtype=torch.uint8, device="cuda")
    sc.run(g, prm, want.data_ptr())
    srv = S.Server(1, 32 * (1 << (nvox - 1).bit_length()) + spare + 64)
    job = srv.submit_filter(sc, g, prm)
    srv.wait(job)
    srv.close()
    sc.close()
    assert np.array_equal(job.out.view(np.uint8), want.cpu().numpy()) and job.out.dtype == N.VOXEL_DTYPE
