"""Refits of TLASes whose arrays go to the host through page-locked staging (up to 16,384 primitives) and by
copies (more): the host gets the same topology with the moved primitives' boxes, either way."""
import ctypes as C

import numpy as np
import pytest

import oracle
from slimtracin_b200 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16384, 16385, 40000])
def test_refit_reaches_the_host(renderer, n):
    sd, cam = scenes.moving_scene(seed_offset=n, count=n)
    renderer.upload(5, sd, tlas=None)
    renderer.build_tlas(5, sd, api.ST_BVH_LBVH30)
    count = sd.tlas_node_count
    before = sd.tlas_nodes[:count].copy(), sd.tlas_leaf_ids[:n].copy()
    ids = np.arange(0, n, 3).astype(np.uint32)
    sd.primitives["position"][ids] += np.float32(0.3)
    renderer.update_primitives(5, sd.primitives[ids], ids)
    sd.tlas_leaf_ids[:n] = 0xFFFFFFFF                       # (written anew)
    renderer.build_tlas(5, sd, api.ST_BVH_REFIT)
    nodes = sd.tlas_nodes[:count]
    assert sd.tlas_node_count == count and np.array_equal(sd.tlas_leaf_ids[:n], before[1])
    for f in ("first_child_id", "child_count", "depth"):
        assert np.array_equal(nodes[f], before[0][f])
    sc, keep = sd.to_ctypes()
    boxes = np.zeros((n, 6), np.float32)
    oracle.restatement().orc_primitive_aabbs(C.byref(sc), boxes.ctypes.data)
    want = np.zeros((count, 6), np.float32)
    for k in np.argsort(-nodes["depth"].astype(int), kind="stable"):
        f, c = int(nodes["first_child_id"][k]), int(nodes["child_count"][k])
        parts = boxes[sd.tlas_leaf_ids[f:f + c]] if c else want[f:f + 2]
        want[k, :3], want[k, 3:] = parts[:, :3].min(0), parts[:, 3:].max(0)
    assert np.array_equal(nodes["aabb"], want)
