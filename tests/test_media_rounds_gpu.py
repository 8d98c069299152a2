"""Medium boundaries in queued rounds (bounces of many paths) and in the persistent walk give the same frame bit for bit:
waves large enough for rounds against waves that have none, over what the walk and the rounds depend on.  The frames
without rounds are compared with the oracle elsewhere."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from renderer2_b200 import filter as F  # noqa: E402
from renderer2_b200 import raytracer as R  # noqa: E402
from renderer2_b200 import render_scenes as RS  # noqa: E402
from renderer2_b200 import scenes  # noqa: E402

W, H, SPP = 512, 384, 4  # 196,608 paths a sample: no rounds in waves of one sample, rounds in waves of four


@pytest.fixture(scope="module")
def desc(tmp_path_factory):
    """Rows of filtered balls, so that rays cross many boxes, one of them with a phase function of its own, a mesh
    between them and a ground disc."""
    mesh = scenes.icosphere(3, 0.08, 4)
    prm = F.params(samples_per_voxel=32, iterations=10, min_voxel_size=scenes.voxel_size_for(mesh, 24), lods=1)
    path = F.run_filtering(mesh, F.material(diffuse=(0.8, 0.5, 0.3), alpha=0.35), prm,
                           tmp_path_factory.mktemp("filtering"), "ball")[0][0]
    media = []
    for k in range(18):
        at = (1.3 * (k % 3) - 1.3, 1.2 * (k // 3 % 2), -1.4 * (k // 6))
        media.append((path, (0.0, 0.0, 0.0), (3.0, 3.0, 3.0), at, (0.0, 1.0, 0.0), (0.5, 0.5, 0.5)))
    media[4] = media[4] + (0.4,)
    return {"media": media, "shapes": [(R.CIRCLE, (0.0, -0.8, 0.0), 40.0, (0, 1, 0), F.material(diffuse=(0.6, 0.6, 0.6)))],
            "meshes": [(scenes.icosphere(2, 0.1, 5), F.material(diffuse=(0.2, 0.4, 0.8), alpha=0.3),
                        RS.trs43((0.0, 0.5, -0.7), scale=(0.4, 0.4, 0.4)))],
            "env": RS.lognormal_env(32, 16, 0.7, 3)}


def _frame(sc, cam, dda, **tuning):
    sc.set_tuning(R.tuning(**tuning))
    return sc.render(cam, R.params(SPP, 7, 3, brick_grid=dda))


@pytest.mark.parametrize("dda", [True, False], ids=["dda", "delta"])
def test_rounds_and_walk_give_the_same_frame(desc, dda):
    sc = RS.build_scene(desc)
    cam = R.camera(W, H, 50.0, (0.4, 0.9, 4.0), (0.0, 0.4, 0.0), (0, 1, 0))
    want = _frame(sc, cam, dda, wave_paths=W * H)
    assert np.isfinite(want).all() and want.std() > 0
    for t in (dict(), dict(media_rounds=1, track_steps=1), dict(media_rounds=2, track_steps=64, track_blocks=1),
              dict(media_rounds=5, track_steps=3, track_blocks=2), dict(media_rounds=32),
              dict(wave_paths=2 * W * H, media_rounds=3)):
        assert np.array_equal(_frame(sc, cam, dda, **t), want), t
    for t in (dict(track_steps=1), dict(track_steps=64, track_blocks=1), dict(track_steps=3, track_blocks=3)):
        assert np.array_equal(_frame(sc, cam, dda, wave_paths=W * H, **t), want), t
    sc.close()


def test_rounds_in_a_captured_batch(desc):
    """The batch's waves of one sample, 300,000 paths each: rounds within the captured graph."""
    cam = R.camera(600, 500, 50.0, (0.4, 0.9, 4.0), (0.0, 0.4, 0.0), (0, 1, 0))
    scs = [RS.build_scene(desc) for _ in range(2)]
    prms = [R.params(2, 7, k, brick_grid=True) for k in range(2)]
    frames = [torch.empty(600 * 500 * 3, dtype=torch.float32, device="cuda") for _ in scs]
    batch = R.RenderBatch(scs, [cam, cam], prms, [f.data_ptr() for f in frames])
    batch.run(0)
    torch.cuda.synchronize()
    got = [f.clone() for f in frames]
    batch.close()
    for sc, prm, g, f in zip(scs, prms, got, frames):
        sc.render_device(cam, prm, f.data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(g, f)
        sc.close()
