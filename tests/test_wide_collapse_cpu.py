"""The room that the eight-wide BVH's builder reserves holds the nodes of any tree, also of boxes whose areas are not
numbers: a mesh or an instance transform need not be finite."""
import numpy as np
import pytest

import wide_probe


def _boxes(n, kind):
    rng = np.random.default_rng(n)
    lo = rng.uniform(-1, 1, (n, 3))
    box = np.concatenate([lo, lo + rng.uniform(0, 0.1, (n, 3))], 1).astype(np.float32)
    if kind == "nan":
        box[:] = np.nan
    elif kind == "some_nan":
        box[rng.random(n) < 0.5] = np.nan
    elif kind == "inf":  # infinite along one axis, flat along another: infinity times zero
        box[:, 0], box[:, 3], box[:, 4] = -np.inf, np.inf, box[:, 1]
    elif kind == "inverted":
        box[:, :3], box[:, 3:] = np.inf, -np.inf
    elif kind == "flat":
        box[:, 3:] = box[:, :3]
    return box


@pytest.mark.parametrize("kind", ["finite", "nan", "some_nan", "inf", "inverted", "flat"])
@pytest.mark.parametrize("skew", [0, 1], ids=["halves", "anywhere"])
def test_nodes_fit_the_room_reserved(kind, skew):
    for n in (2, 3, 8, 9, 16, 17, 64, 1000, 10_000):
        count, room = wide_probe.wide_nodes(_boxes(n, kind), skew)
        assert count <= room, (n, count, room)
