"""The autotuner's choice renders a frame no slower than the defaults do, also where the frame's first sample says little
about the others."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from renderer2_b200 import raytracer as R  # noqa: E402
from renderer2_b200 import render_scenes as RS  # noqa: E402


def _ms(sc, cam, prm):
    frame = torch.empty((cam.height, cam.width, 3), dtype=torch.float32, device="cuda")
    return min(sc.render_device(cam, prm, frame.data_ptr())[1] for _ in range(5))


@pytest.mark.parametrize("width,height,spp", [(96, 80, 2), (512, 512, 12), (1024, 768, 9)])
def test_tuned_frames_are_no_slower(width, height, spp):
    """By more than a quarter: runs of one setting differ by less."""
    desc, _ = RS.icosphere_grid_scene()
    sc = RS.build_scene(desc)
    cam, prm = R.camera(width, height, 45.0, (0, 0, 24), (0, 0, 0), (0, 1, 0)), R.params(spp, 6, 2)
    before = _ms(sc, cam, prm)
    t = sc.autotune(cam, prm)
    assert t.wave_paths in [1 << k for k in range(20, 25)]
    assert np.isfinite(before) and _ms(sc, cam, prm) <= 1.25 * before
    sc.close()
