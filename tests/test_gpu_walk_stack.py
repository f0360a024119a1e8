"""The walk's one stack where its parts meet: pending TLAS pairs, the frame of the instance the ray is in,
and pending BLAS pairs, in local memory or with the first 32 words in shared memory.  Both trees are
chains whose boxes all hold the whole scene, so that a pair stays pending at every level."""
import numpy as np
import pytest

from slimtracin_b200 import api, scenes, structs as S
from tests import helpers as H
from tests.test_gpu_walk import instanced_scene

pytestmark = pytest.mark.gpu


def chain(levels, items, box):
    """A tree of `levels` levels: at each the left child goes on, the right one has two leaves; the last left
    child is a leaf.  Of `items` items, each leaf gets its share in order.  All boxes are `box`."""
    nodes = np.zeros(1 + 4 * levels, dtype=S.BVHNODE_DT)
    nodes["aabb"] = box
    cuts = np.linspace(0, items, 2 * levels + 2).astype(int)
    leaves = iter(zip(cuts[:-1], np.diff(cuts)))

    def leaf(k):
        nodes["first_child_id"][k], nodes["child_count"][k] = next(leaves)

    at = 0
    for d in range(levels):
        f = 1 + 4 * d
        nodes["first_child_id"][at] = f
        nodes["first_child_id"][f + 1] = f + 2
        leaf(f + 2)
        leaf(f + 3)
        nodes["depth"][f:f + 2], nodes["depth"][f + 2:f + 4] = d + 1, d + 2
        at = f
    leaf(at)
    return nodes


def deep_scene(tlas_levels, blas_levels):
    sd, cam = instanced_scene(320, 4 * tlas_levels + 2, 2)
    md = sd.meshes[0]
    H.blas_sah(md, "binned")
    md.node_count, md.height = 1 + 4 * blas_levels, blas_levels + 1
    md.nodes[:md.node_count] = chain(blas_levels, md.triangle_count, md.nodes["aabb"][0])
    H.tlas_binned(sd)
    nodes = chain(tlas_levels, len(sd.primitives), sd.tlas_nodes["aabb"][0])
    sd.tlas_nodes[:len(nodes)] = nodes
    sd.tlas_leaf_ids[:len(sd.primitives)] = np.random.default_rng(tlas_levels).permutation(len(sd.primitives))
    sd.tlas_node_count, sd.tlas_height = len(nodes), tlas_levels + 1
    return sd, cam


@pytest.mark.parametrize("tlas_levels,blas_levels", [(16, 12), (20, 9)] + [(d, 20) for d in range(25, 35)] + [(31, 1), (61, 61)])
def test_deep_trees_over_deep_trees(renderer, tlas_levels, blas_levels):
    sd, cam = deep_scene(tlas_levels, blas_levels)
    renderer.upload(3, sd)
    g = H.gpu_frame(renderer, 3, sd, cam, 61, 43, depth=1, mode=S.RM_NORMALS)
    o = H.oracle_frame(sd, cam, 61, 43, depth=1, mode=S.RM_NORMALS)
    assert g.float_pixels.tobytes() == o.float_pixels.tobytes()
    one = H.gpu_frame(renderer, 3, sd, cam, 61, 43, depth=3, counters=True)
    o = H.oracle_frame(sd, cam, 61, 43, depth=3)
    same = [0, 1, 2, 7, 8] if len(sd.primitives) > 64 else list(range(11))
    assert np.array_equal(one.counters[same], o.counters[same]), (one.counters[:11], o.counters[:11])
    for stack_placement in (0, 1):
        fr = scenes.Frame(61, 43, cam, depth=3)
        api.render_batch(renderer, [(3, sd, fr)], tile_shape=0, chunk=1, stack_placement=stack_placement, launch_mode=api.LAUNCH_PERSISTENT)
        assert fr.float_pixels.tobytes() == one.float_pixels.tobytes(), stack_placement
