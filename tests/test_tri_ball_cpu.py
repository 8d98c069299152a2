"""The filter's test of triangles against balls may keep a triangle too many, never one too few: against distances in 64
bits, over slivers, triangles without area, large and tiny ones, every scale, and vertices that are not finite."""
import numpy as np
import pytest

import wide_probe


def _dist(p, tri):
    """Distance of points (n, 3) from triangles (n, 3, 3) in 64 bits."""
    a, b, c = (tri[:, k].astype(np.float64) for k in range(3))
    p = p.astype(np.float64)

    def edge(u, v):
        e = v - u
        ee = (e * e).sum(1)
        t = np.clip(((p - u) * e).sum(1) / np.where(ee > 0, ee, 1.0), 0.0, 1.0)
        return np.linalg.norm(p - u - e * t[:, None], axis=1)

    n = np.cross(b - a, c - a)
    nn = (n * n).sum(1)
    inside = nn > 0
    for u, v in ((a, b), (b, c), (c, a)):
        inside &= (np.cross(v - u, p - u) * n).sum(1) >= 0
    plane = np.abs(((p - a) * n).sum(1)) / np.sqrt(np.where(nn > 0, nn, 1.0))
    return np.where(inside, plane, np.minimum(np.minimum(edge(a, b), edge(b, c)), edge(c, a)))


def _draw(rng, n, scale):
    a, u, v = rng.uniform(-1, 1, (n, 3)), rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    length = np.exp(rng.uniform(np.log(1e-4), np.log(20.0), n))[:, None]
    width = length * np.exp(rng.uniform(np.log(1e-7), 0.0, n))[:, None]
    width[::17] = 0.0
    tri = np.stack([a, a + u * length, a + u * length * rng.uniform(-0.2, 1.2, (n, 1)) + v * width], 1)
    c0 = rng.uniform(-1, 1, (n, 3))
    around = rng.uniform(0.0, 0.1, n)
    d = rng.normal(size=(n, 3))
    c = c0 + d / np.linalg.norm(d, axis=1, keepdims=True) * (0.9 * around)[:, None]
    return [(scale * x).astype(np.float32) for x in (tri, c0, around, c)]


@pytest.mark.parametrize("scale", [1e-9, 1e-4, 1.0, 1e4, 1e9, 1e12], ids=str)
def test_no_touching_triangle_is_dropped(scale):
    rng = np.random.default_rng(5)
    tri, c0, around, c = _draw(rng, 200_000, scale)
    d = _dist(c, tri)
    r = (d * rng.choice([1.0, 1.001, 1.3, 5.0], d.size) * (1 + 1e-7)).astype(np.float32)  # from just touching up
    near = wide_probe.tri_near(tri, c0, around, c, r, 0.1 * scale)
    assert near.all(), (int((~near).sum()), tri[~near][:2], c[~near][:2], r[~near][:2])
    wide = np.linalg.norm(np.cross(*(tri[:, k] - tri[:, 0] for k in (1, 2))) / scale**2, axis=1) > 1e-3
    kept = wide_probe.tri_near(tri, c0, around, c, (0.5 * d).astype(np.float32), 0.1 * scale)
    assert kept[wide].mean() < 0.2, kept[wide].mean()  # and most of the others, but for slivers, are dropped


def test_vertices_that_are_no_numbers_drop_nothing():
    rng = np.random.default_rng(6)
    tri, c0, around, c = _draw(rng, 20_000, 1.0)
    k = np.arange(20_000)
    tri[k, rng.integers(0, 3, k.size), rng.integers(0, 3, k.size)] = np.nan
    tri[::3] = np.nan
    assert wide_probe.tri_near(tri, c0, around, c, np.full(k.size, 0.01, np.float32), 0.1).all()
