"""Instances flattened by a zero scale: their object-space rays hold values that are not numbers, and no
triangle of them is ever hit.  The walk spends on them no more box and triangle tests than the reference's
box test (render/AABB.h:6) gives it there: none at all once a ray has hit something."""
import numpy as np
import pytest

from slimtracin_b200 import api, scenes, structs as S
from tests import helpers as H
from tests.test_gpu_walk import instanced_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axes", [(0,), (1,), (2,), (0, 1), (1, 2), (0, 2), (0, 1, 2)])
@pytest.mark.parametrize("turned", [False, True])
def test_flat_instances_cost_what_the_specification_gives(renderer, turned, axes):
    sd, cam = instanced_scene(320, 48, 2)
    for i in range(0, 48, 3):            # (instances and boxes among them)
        sd.primitives["scale"][i, list(axes)] = 0
        if not turned:
            sd.primitives["rotation"][i] = (0, 0, 0, 1)
    renderer.build_blas(sd.meshes[0], api.ST_BVH_BINNED_SAH)
    renderer.upload(3, sd, tlas=None)
    renderer.build_tlas(3, sd, api.ST_BVH_BINNED_SAH)
    g = H.gpu_frame(renderer, 3, sd, cam, 97, 61, depth=1, mode=S.RM_NORMALS)
    o = H.oracle_frame(sd, cam, 97, 61, depth=1, mode=S.RM_NORMALS)
    assert g.float_pixels.tobytes() == o.float_pixels.tobytes()
    g = H.gpu_frame(renderer, 3, sd, cam, 97, 61, depth=4, counters=True)
    o = H.oracle_frame(sd, cam, 97, 61, depth=4)
    # hits, rays and candidates are the specification's; box and triangle tests at most its
    same = [k for k in range(11) if k not in (3, 4)]
    assert np.array_equal(g.counters[same], o.counters[same]), (g.counters[:11], o.counters[:11])
    assert (g.counters[3:5] <= o.counters[3:5]).all(), (g.counters[:11], o.counters[:11])
