"""TLAS updates where their paths meet: LBVH30 by one block (up to 4096 primitives) and by many, a tree
that is one leaf, trees too deep for the traversal stacks, refits, and what the host gets back."""
import ctypes as C

import numpy as np
import pytest

import oracle
from slimtracin_b200 import api, scenes, structs as S
from tests import helpers as H

pytestmark = pytest.mark.gpu


def lbvh_equals_oracle(renderer, boxes, max_leaf):
    n = len(boxes)
    codes, order, nodes, count, height = renderer.build_lbvh(boxes, max_leaf)
    oc, oo, ol = np.zeros(n, np.uint32), np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    on, oi = np.zeros(2 * n, dtype=S.BVHNODE_DT), np.zeros(2, np.uint32)
    oracle.restatement().orc_lbvh30(boxes.ctypes.data, n, max_leaf, oc.ctypes.data, oo.ctypes.data, on.ctypes.data,
                                    ol.ctypes.data, oi.ctypes.data)
    assert (count, height) == (int(oi[0]), int(oi[1]))
    assert np.array_equal(codes, oc) and np.array_equal(order, oo)
    assert nodes.tobytes() == on[:count].tobytes()


@pytest.mark.parametrize("clumped", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 33, 1023, 1025, 2048, 4095, 4096, 4097])
def test_lbvh_equals_specification(renderer, n, clumped):
    rng = np.random.default_rng(n)
    c = rng.uniform(-9, 9, (n, 3))
    if clumped:                          # equal codes in runs, a flat axis
        c = np.round(c / 6) * 6
        c[:, 1] = -2.0
    e = rng.uniform(0, 1, (n, 3))
    boxes = np.concatenate([c - e, c + e], 1).astype(np.float32)
    for max_leaf in (1, 2, 4, 40):
        lbvh_equals_oracle(renderer, boxes, max_leaf)


@pytest.mark.parametrize("mode", [api.ST_BVH_LBVH30, api.ST_BVH_BINNED_SAH])
@pytest.mark.parametrize("n", [1, 2, 3, 600, 4096, 5000])
def test_tlas_update_and_refit(renderer, n, mode):
    """The host's arrays after a build are the oracle's tree, and after moves and a refit the same
    topology with the boxes of the moved primitives; a render uses them."""
    sd, cam = scenes.moving_scene(seed_offset=n, count=n)
    renderer.upload(5, sd, tlas=None)
    renderer.build_tlas(5, sd, mode)
    want = sd.copy()
    (H.tlas_lbvh if mode == api.ST_BVH_LBVH30 else H.tlas_binned)(want)
    assert H.same_tlas(sd, want)
    ids = np.arange(0, n, 3).astype(np.uint32)
    sd.primitives["position"][ids] += np.float32(0.3)
    renderer.update_primitives(5, sd.primitives[ids], ids)
    topology = [sd.tlas_nodes[f].copy() for f in ("first_child_id", "child_count", "depth")]
    renderer.build_tlas(5, sd, api.ST_BVH_REFIT)
    for before, f in zip(topology, ("first_child_id", "child_count", "depth")):
        assert np.array_equal(before, sd.tlas_nodes[f])
    sc, keep = sd.to_ctypes()
    boxes = np.zeros((n, 6), np.float32)
    oracle.restatement().orc_primitive_aabbs(C.byref(sc), boxes.ctypes.data)
    raw = sd.tlas_nodes[:sd.tlas_node_count].view(np.float32).reshape(-1, 8)[:, :6]
    assert np.array_equal(raw[0, :3], boxes[:, :3].min(0)) and np.array_equal(raw[0, 3:], boxes[:, 3:].max(0))
    for k in range(sd.tlas_node_count):
        node = sd.tlas_nodes[k]
        if node["child_count"]:
            items = boxes[sd.tlas_leaf_ids[node["first_child_id"]:node["first_child_id"] + node["child_count"]]]
            assert np.array_equal(raw[k, :3], items[:, :3].min(0)) and np.array_equal(raw[k, 3:], items[:, 3:].max(0))
    g = H.gpu_frame(renderer, 5, sd, cam, 64, 40, depth=1, mode=S.RM_NORMALS)
    o = H.oracle_frame(sd, cam, 64, 40, depth=1, mode=S.RM_NORMALS)
    assert g.float_pixels.tobytes() == o.float_pixels.tobytes()


@pytest.mark.parametrize("n", [130, 300, 4096, 5000])
def test_too_deep_a_tree_is_refused(n):
    """Thin boxes at a small spacing whose unions all have the same area (2^40, the spacing rounds away): of
    equal costs the first split wins, so a level loses its first bin only and the binned tree is deeper than
    the 62 levels that a walk's stack holds.  The update refuses it, and leaves no TLAS until a build
    succeeds."""
    not_resident = 8
    sd, cam = scenes.moving_scene(count=n)
    sd.primitives["type"] = S.PT_BOX
    sd.primitives["rotation"] = (0, 0, 0, 1)
    sd.primitives["position"] = 0
    sd.primitives["position"][:, 0] = np.linspace(0, 0.01, n)
    sd.primitives["scale"] = (1e-9, 2.0 ** 19, 2.0 ** 19)
    want = sd.copy()
    H.tlas_binned(want)
    assert want.tlas_height > 62
    with api.Renderer(device=0) as r:
        r.upload(0, sd, tlas=None)
        r.build_tlas(0, sd, api.ST_BVH_LBVH30)
        first = H.gpu_frame(r, 0, sd, cam, 64, 40, depth=1)
        sc, keep = sd.to_ctypes()
        nodes, ids = sd.tlas_nodes.tobytes(), sd.tlas_leaf_ids.tobytes()
        assert r.L.st_update_scene_bvh(r.ctx, 0, C.byref(sc), api.ST_BVH_BINNED_SAH) == api.ST_ERR_BAD_SCENE
        assert sd.tlas_nodes.tobytes() == nodes and sd.tlas_leaf_ids.tobytes() == ids
        assert r.L.st_update_scene_bvh(r.ctx, 0, None, api.ST_BVH_REFIT) == not_resident
        with pytest.raises(api.STError) as e:
            H.gpu_frame(r, 0, sd, cam, 64, 40, depth=1)
        assert e.value.status == not_resident
        r.build_tlas(0, sd, api.ST_BVH_LBVH30)
        assert H.gpu_frame(r, 0, sd, cam, 64, 40, depth=1).float_pixels.tobytes() == first.float_pixels.tobytes()
