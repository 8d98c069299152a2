"""The filter's candidate lists where they can go wrong: triangles that a ball
test may drop wrongly (slivers, huge ones, ones without area, an edge-on
plane), grids that end inside a brick or are one voxel thick, objects far from
the origin and of small scale, and grids worked off in several parts.  Hits
are compared with the oracle, which traces every ray from the BVH's root, bit
for bit; the 1e-4 and one-LSB bounds of the other filter tests hold for the rest."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from renderer2_b200 import _native as N  # noqa: E402
from renderer2_b200 import filter as F  # noqa: E402
from renderer2_b200 import scenes  # noqa: E402
from test_filter_gpu import _compare, _gpu_filter, _oracle  # noqa: E402


def _awkward(seed: int) -> F.Mesh:
    """Random triangles in the unit cube: slivers of aspect up to 1e6, small ones, ones without area, and one that
    covers the whole box."""
    rng = np.random.default_rng(seed)
    a, u, v = rng.random((400, 3)), rng.normal(size=(400, 3)), rng.normal(size=(400, 3))
    length = np.exp(rng.uniform(np.log(1e-3), np.log(0.5), 400))[:, None]
    width = length * np.exp(rng.uniform(np.log(1e-6), 0.0, 400))[:, None]
    width[::29] = 0.0
    tri = np.clip(np.stack([a, a + u * length, a + u * length * 0.4 + v * width], 1), 0.0, 1.0)
    tri = np.concatenate([tri, [[[0.0, 0.0, 0.0], [1.0, 1.0, 0.3], [0.0, 1.0, 1.0]]]]).astype(np.float32)
    n = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]).astype(np.float64)
    ln = np.linalg.norm(n, axis=1, keepdims=True)
    n = np.where(ln > 0, n / np.where(ln > 0, ln, 1.0), [0.0, 1.0, 0.0])
    return F.Mesh(tri.reshape(-1, 3), np.arange(tri.size // 3, dtype=np.uint32).reshape(-1, 3),
                  np.repeat(n, 3, axis=0).astype(np.float32))


def _flat(n: int) -> F.Mesh:
    """A strip of quads in the plane y = x / 8, a grid of which is one or two voxels thick."""
    x = np.linspace(0.0, 1.0, n + 1)
    pos = np.stack([np.repeat(x, 2), np.repeat(x, 2) / 8.0, np.tile([0.0, 0.02], n + 1)], 1).astype(np.float32)
    q = 2 * np.arange(n, dtype=np.uint32)[:, None]
    idx = (q + np.array([0, 1, 3, 0, 3, 2], np.uint32)).reshape(-1, 3)
    nrm = np.tile(np.array([-0.12403473, 0.99227788, 0.0], np.float32), (pos.shape[0], 1))
    return F.Mesh(pos, idx, nrm)


@pytest.mark.parametrize("mesh,n", [(_awkward(1), 13), (_awkward(2), 32), (_flat(40), 17), (_flat(9), 3),
                                    (scenes.foliage(3000, 4, 0.7, 2), 31)],
                         ids=["awkward13", "awkward32", "flat17", "flat3", "leaves31"])
@pytest.mark.parametrize("clip", [True, False], ids=["clip", "fixed"])
@pytest.mark.parametrize("place", [(1.0, 0.0), (0.01, 0.0), (1.0, 50.0)], ids=["unit", "small", "far"])
def test_hits_match_the_oracle(mesh, n, clip, place):
    scale, far = place
    m2w = np.array([scale, 0, 0, 0, scale, 0, 0, 0, scale, far, -far, 0.5 * far], np.float32)
    mat = F.material(diffuse=(0.2, 0.5, 0.1), alpha=0.4)
    prm = F.params(samples_per_voxel=40, iterations=3, clip_rays=clip, seed=3)
    vs = scenes.voxel_size_for(mesh, n) * scale
    g, gc, gw, st = _gpu_filter(mesh, mat, prm, vs, m2w)
    ow, oc = _oracle(mesh, mat, prm, g, m2w)
    assert ow[:, 17].sum() > 0
    _compare(gw, gc, ow, oc)
    assert st[1] >= (ow[:, 17] > 0).sum()


def test_a_grid_in_parts_equals_the_whole():
    """The allocation-free entry point has room for 2^20 / 6 voxels at a time: a 64^3 grid takes two parts, the
    scene's own work space holds it whole."""
    leaves = scenes.foliage(6000, 6, 0.7, 5)
    sc = F.FilterScene(leaves, F.material())
    prm = F.params(samples_per_voxel=33, iterations=4)
    g = sc.grid(scenes.voxel_size_for(leaves, 64))
    nvox = int(np.prod(np.array(g.num_voxels[:], np.int64)))
    assert nvox > (1 << 20) // 6
    whole, parts = (torch.full((nvox * 32,), k, dtype=torch.uint8, device="cuda") for k in (1, 2))
    sc.run(g, prm, whole.data_ptr())
    torch.cuda.synchronize()
    run = N.lib.r2_filter_scene_run_static
    run.restype, run.argtypes = C.c_int, [C.c_void_p] * 7
    N.check(run(sc.handle, C.byref(g), C.byref(prm), C.c_void_p(parts.data_ptr()), None, None, None))
    torch.cuda.synchronize()
    sc.close()
    assert torch.equal(whole, parts)


@pytest.mark.parametrize("scale", [1e-14, 1e-12, 1e-10, 1e-6, 1e6, 1e10, 1e12], ids=str)
def test_hits_match_the_oracle_at_any_scale(scale):
    """Triangles whose edges' fourth powers leave the range of a float."""
    mesh = _awkward(4)
    m2w = np.array([scale, 0, 0, 0, scale, 0, 0, 0, scale, 0, 0, 0], np.float32)
    mat = F.material(diffuse=(0.2, 0.5, 0.1), alpha=0.4)
    prm = F.params(samples_per_voxel=40, iterations=3, seed=3)
    g, gc, gw, st = _gpu_filter(mesh, mat, prm, scenes.voxel_size_for(mesh, 9) * scale, m2w)
    ow, oc = _oracle(mesh, mat, prm, g, m2w)
    assert ow[:, 17].sum() > 0
    assert np.array_equal(gw[:, 17], ow[:, 17])
