"""The device's binned-SAH build against the CPU specification, byte for byte, where its paths meet:
ranges built without bins (up to 10 items), by a warp (up to 512), by a block (up to 4096) and by many
blocks, leaves larger than any of them, and inputs that split at the middle, peel a few items a level
or hold values that are not numbers."""
import numpy as np
import pytest

import oracle
from slimtracin_b200 import api, structs as S

pytestmark = pytest.mark.gpu


def item_boxes(kind, n):
    rng = np.random.default_rng(n * 7 + len(kind))
    c = rng.uniform(-20, 20, (n, 3))
    e = rng.uniform(0.01, 1.5, (n, 3))
    if kind == "same":                   # equal centroids: every split is at the middle
        c[:] = c[0]
    elif kind == "peel":                 # equal boxes far larger than their spacing: each level loses the first bin
        c = np.linspace(-1, 1, n)[:, None] * [1.0, 0.0, 0.0]
        e[:] = 1e4
    elif kind == "clumps":               # many ties, one flat axis, powers of two apart
        c = np.round(c / 8) * 2.0 ** rng.integers(-12, 12, (n, 1))
        c[:, 2] = 3.0
        e[:] = 0.25
    boxes = np.concatenate([c - e, c + e], 1).astype(np.float32)
    if kind == "odd values":
        boxes[rng.integers(0, n, max(n // 50, 1)), 4] = np.nan
        boxes[rng.integers(0, n, max(n // 50, 1)), 3] = np.inf
        boxes[rng.integers(0, n, max(n // 50, 1)), 0] = -0.0
    return boxes


def check(renderer, boxes, max_leaf):
    n = len(boxes)
    _, order, nodes, count, height = renderer.build_lbvh(boxes, max_leaf, api.ST_BVH_BINNED_SAH)
    oo, on, oi = np.zeros(n, np.uint32), np.zeros(2 * n, dtype=S.BVHNODE_DT), np.zeros(2, np.uint32)
    oracle.restatement().orc_binned_sah(boxes.ctypes.data, n, max_leaf, oo.ctypes.data, on.ctypes.data, oi.ctypes.data)
    assert (count, height) == (int(oi[0]), int(oi[1]))
    assert np.array_equal(order, oo)
    assert nodes.tobytes() == on[:count].tobytes()


@pytest.mark.parametrize("kind", ["spread", "same", "peel", "clumps", "odd values"])
@pytest.mark.parametrize("n", [1, 2, 3, 10, 11, 33, 256, 257, 512, 513, 1100, 4096, 4097, 9000])
def test_binned_sah_equals_specification(renderer, n, kind):
    for max_leaf in (1, 2, 4):
        check(renderer, item_boxes(kind, n), max_leaf)


@pytest.mark.parametrize("n,max_leaf", [(60000, 4), (9000, 5000), (9000, 9000), (30000, 700), (300, 299)])
def test_binned_sah_leaf_sizes(renderer, n, max_leaf):
    check(renderer, item_boxes("spread", n), max_leaf)
