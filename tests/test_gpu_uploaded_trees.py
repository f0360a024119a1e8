"""Uploaded TLASes whose arrays hold nodes that no other leads to: the walk never sees them, and a refit,
which goes over the whole array, neither follows nor changes what they stand beside."""
import numpy as np
import pytest

from slimtracin_b200 import api, scenes, structs as S
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", ["leaf", "leaf out of range", "inner", "inner out of range", "inner claiming the root's children"])
def test_refit_of_a_tree_with_unreached_nodes(renderer, extra):
    sd, cam = scenes.moving_scene(count=300)
    H.tlas_binned(sd)
    plain = sd.copy()
    n, count = len(sd.primitives), sd.tlas_node_count
    assert count + 4 <= 2 * n
    more = sd.tlas_nodes[count:count + 4]
    more["child_count"] = 2 if "leaf" in extra else 0
    more["first_child_id"] = {"leaf": 5, "leaf out of range": n - 1, "inner": count + 4 - (count + 1) % 2, "inner out of range": 2 ** 31 + 1,
                              "inner claiming the root's children": 1}[extra]
    more["aabb"] = sd.tlas_nodes["aabb"][0]
    sd.tlas_node_count = count + 4
    frames = []
    for slot, scene in ((1, plain), (2, sd)):
        renderer.upload(slot, scene)
        ids = np.arange(0, n, 3).astype(np.uint32)
        moved = scene.primitives[ids].copy()
        moved["position"] += np.float32(0.3)
        renderer.update_primitives(slot, moved, ids)
        frames.append(H.gpu_frame(renderer, slot, scene, cam, 64, 40, depth=1, mode=S.RM_NORMALS))
        renderer.build_tlas(slot, scene, api.ST_BVH_REFIT)
        frames.append(H.gpu_frame(renderer, slot, scene, cam, 64, 40, depth=1, mode=S.RM_NORMALS))
    assert sd.tlas_nodes[:count].tobytes() == plain.tlas_nodes[:count].tobytes()
    assert frames[2].float_pixels.tobytes() == frames[0].float_pixels.tobytes()
    assert frames[3].float_pixels.tobytes() == frames[1].float_pixels.tobytes()
