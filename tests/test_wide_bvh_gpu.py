"""The path tracer's eight-wide BVH where it can go wrong: trees of one triangle
and of one leaf, nodes without extent along an axis, triangles of very
different size in one node, scenes far from the origin, rays along the axes,
and instances whose leaves share a node.  Frames are compared with the oracle,
which walks the binary tree, with the bound of the other frame tests."""
import numpy as np
import pytest

import oracle_lib as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from renderer2_b200 import filter as F  # noqa: E402
from renderer2_b200 import raytracer as R  # noqa: E402
from renderer2_b200 import render_scenes as RS  # noqa: E402
from renderer2_b200 import scenes  # noqa: E402
from test_render_gpu import PIX_FRAC, _agree, _gpu_frame  # noqa: E402


def _mesh(tri):
    tri = np.asarray(tri, np.float32).reshape(-1, 3, 3)
    n = np.cross((tri[:, 1] - tri[:, 0]).astype(np.float64), (tri[:, 2] - tri[:, 0]).astype(np.float64))
    ln = np.linalg.norm(n, axis=1, keepdims=True)
    n = np.where(ln > 0, n / np.where(ln > 0, ln, 1.0), [0.0, 0.0, 1.0])
    return F.Mesh(tri.reshape(-1, 3), np.arange(tri.size // 3, dtype=np.uint32).reshape(-1, 3),
                  np.repeat(n, 3, axis=0).astype(np.float32))


def _quads(n, z):
    """n x n axis-aligned quads in a plane of constant z, [-1, 1]^2."""
    e = np.linspace(-1.0, 1.0, n + 1)
    out = []
    for i in range(n):
        for j in range(n):
            a, b, c, d = ([e[i], e[j], z], [e[i + 1], e[j], z], [e[i + 1], e[j + 1], z], [e[i], e[j + 1], z])
            out += [[a, b, c], [a, c, d]]
    return np.asarray(out)


def _mixed(seed):
    """Triangles whose sizes span five decades, in one box."""
    rng = np.random.default_rng(seed)
    size = np.exp(rng.uniform(np.log(1e-5), 0.0, 300))[:, None, None]
    return rng.uniform(-1, 1, (300, 1, 3)) + size * rng.normal(size=(300, 3, 3))


CASES = {"one": (_mesh([[[-1, -1, 0], [1, -1, 0], [0, 1, 0]]]), (0, 0, 0)),
         "seven": (_mesh(_mixed(3)[:7]), (0, 0, 0)),
         "flat": (_mesh(_quads(9, 0.0)), (0, 0, 0)),
         "layers": (_mesh(np.concatenate([_quads(5, z) for z in (-0.5, 0.0, 0.25)])), (0, 0, 0)),
         "mixed": (_mesh(_mixed(5)), (0, 0, 0)),
         "far": (scenes.icosphere(3, 0.05, 2), (1000.0, -500.0, 250.0)),
         "ball": (scenes.icosphere(2, 0.1, 4), (0, 0, 0))}


def _close(desc, cam, spp, depth, seed):
    g = _gpu_frame(desc, cam, spp, depth, seed)
    o = O.render(desc, cam, spp, depth, seed)
    assert np.isfinite(g).all() and _agree(g, o) >= PIX_FRAC


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("axis", [False, True], ids=["oblique", "axis"])
def test_frames_match_the_oracle(name, axis):
    mesh, at = CASES[name]
    mat = F.material(diffuse=(0.6, 0.5, 0.4), specular=(1, 1, 1), alpha=0.4, ior=1.5)
    desc = {"meshes": [(mesh, mat, RS.translate43(*at))], "shapes": [], "env": RS.lognormal_env(16, 8, 1.0, 3)}
    eye = np.array(at) + (np.array([0.0, 0.0, 4.0]) if axis else np.array([1.1, 0.7, 3.6]))
    cam = R.camera(48, 40, 45.0, tuple(eye), at, (0, 1, 0))
    _close(desc, cam, 4, 6, 1)


@pytest.mark.parametrize("n", [1, 2, 9, 40])
def test_instances_match_the_oracle(n):
    """n placements of one mesh, so that top-level nodes hold up to eight instances that a ray enters in turn, beside
    a world-space mesh."""
    rng = np.random.default_rng(n)
    ball = scenes.icosphere(2, 0.1, 4)
    mat = F.material(diffuse=(0.6, 0.5, 0.4), specular=(1, 1, 1), alpha=0.4, ior=1.5)
    meshes = [(ball, mat, RS.trs43(tuple(rng.uniform(-1.5, 1.5, 3)), (*rng.normal(size=3), 1.0),
                                   tuple(rng.uniform(0.2, 0.8, 3)))) for _ in range(max(n, 2))]
    meshes.append((_mesh(_quads(3, -2.0)), F.material(diffuse=(0.2, 0.6, 0.8)), RS.translate43(0, 0, 0)))
    desc = {"meshes": meshes, "shapes": [], "env": RS.lognormal_env(16, 8, 1.0, 3)}
    cam = R.camera(48, 40, 50.0, (0.4, 0.9, 5.0), (0, 0, 0), (0, 1, 0))
    _close(desc, cam, 4, 6, 1)
