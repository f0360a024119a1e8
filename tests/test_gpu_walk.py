"""The two-level walk at the shapes where its bookkeeping can go wrong: meshes whose BLAS is one leaf
or a few nodes, scenes that test every primitive and scenes that walk the TLAS, instances that follow
one another in a leaf, shadow and bounce rays; against the oracle, which nests the walks."""
import numpy as np
import pytest

import oracle  # noqa: F401
from slimtracin_b200 import api, scenes, structs as S
from tests import helpers as H

pytestmark = pytest.mark.gpu


def instanced_scene(triangles, count, lights, nan_vertex=False):
    """`count` primitives, two of three of them instances of one open mesh of `triangles` faces, some
    mirrors and some glass, in a cloud the camera looks at."""
    md = scenes.displaced_icosphere(2, seed=11, radius=1.0)
    md.indices = np.ascontiguousarray(md.indices[:triangles])
    if nan_vertex:
        md.positions[md.indices[triangles // 2, 1]] = np.nan
    rng = np.random.default_rng(triangles * 1000 + count)
    prims = scenes.default_primitives(count)
    kinds = (S.PT_MESH, S.PT_MESH, S.PT_BOX, S.PT_MESH, S.PT_MESH, S.PT_SPHERE)
    for i in range(count):
        prims["type"][i] = kinds[i % 6]
        prims["id"][i] = 0
        prims["position"][i] = rng.uniform(-3, 3, 3)
        q = rng.normal(size=4)
        prims["rotation"][i] = q / np.linalg.norm(q)
        prims["scale"][i] = rng.uniform(0.4, 1.2, 3)
        prims["material_id"][i] = i % 3
    mats = scenes.default_materials(3)
    mats["brdf"] = S.BRDF_LAMBERT
    mats["is_"][1], mats["is_"][2] = S.REFLECTIVE, S.REFRACTIVE
    mats["reflectivity"][1] = 0.8
    mats["n1_over_n2"][2], mats["n2_over_n1"][2] = np.float32(1 / 1.5), np.float32(1.5)
    lt = scenes.default_lights(lights)
    for k in range(lights):
        lt["position_or_direction"][k] = (4.0 - 3 * k, 6.0, -5.0)
        lt["intensity"][k] = 20
    sd = scenes.SceneData(prims, mats, lt, ambient=(0.01, 0.01, 0.02), meshes=[md])
    return sd, scenes.look_at((0.7, 1.0, -9.0), (0.1, 0.0, 0.0))


@pytest.mark.parametrize("lights", [0, 2])
@pytest.mark.parametrize("count", [1, 2, 3, 64, 65, 130])
@pytest.mark.parametrize("triangles", [1, 4, 5, 9, 320])
def test_walk_equals_oracle(renderer, triangles, count, lights):
    """Same hits byte for byte (normals mode takes no libm call) and, over shading, shadow and bounce
    rays, the same work."""
    sd, cam = instanced_scene(triangles, count, lights)
    renderer.build_blas(sd.meshes[0], api.ST_BVH_BINNED_SAH)
    renderer.upload(3, sd, tlas=None)
    renderer.build_tlas(3, sd, api.ST_BVH_BINNED_SAH)
    g = H.gpu_frame(renderer, 3, sd, cam, 97, 61, depth=1, mode=S.RM_NORMALS)
    o = H.oracle_frame(sd, cam, 97, 61, depth=1, mode=S.RM_NORMALS)
    assert g.float_pixels.tobytes() == o.float_pixels.tobytes()
    g = H.gpu_frame(renderer, 3, sd, cam, 97, 61, depth=4, counters=True)
    o = H.oracle_frame(sd, cam, 97, 61, depth=4)
    # box tests and leaf reads of primary rays that walk the TLAS differ by design (screen-space cull)
    same = [0, 1, 2, 7, 8] if count > 64 else list(range(11))
    assert np.array_equal(g.counters[same], o.counters[same]), (g.counters[:11], o.counters[:11])


@pytest.mark.parametrize("stack_placement", [0, 1])
def test_batched_walk_equals_per_frame(renderer, stack_placement):
    """The persistent kernel, its stack in local or partly in shared memory, writes the same bytes."""
    sd, cam = instanced_scene(320, 130, 2)
    renderer.build_blas(sd.meshes[0], api.ST_BVH_BINNED_SAH)
    renderer.upload(3, sd, tlas=None)
    renderer.build_tlas(3, sd, api.ST_BVH_BINNED_SAH)
    one = H.gpu_frame(renderer, 3, sd, cam, 97, 61, depth=4)
    fr = scenes.Frame(97, 61, cam, depth=4)
    api.render_batch(renderer, [(3, sd, fr)], tile_shape=0, chunk=1, stack_placement=stack_placement,
                     launch_mode=api.LAUNCH_PERSISTENT)
    assert fr.float_pixels.tobytes() == one.float_pixels.tobytes()


@pytest.mark.parametrize("mode", [api.ST_BVH_BINNED_SAH, api.ST_BVH_LBVH30])
def test_mesh_with_a_nan_vertex(renderer, mode):
    """Boxes with NaN bounds leave that axis out: the triangles that are numbers are hit as before."""
    sd, cam = instanced_scene(320, 6, 0, nan_vertex=True)
    renderer.build_blas(sd.meshes[0], mode)
    renderer.upload(3, sd, tlas=None)
    renderer.build_tlas(3, sd, api.ST_BVH_BINNED_SAH)
    g = H.gpu_frame(renderer, 3, sd, cam, 97, 61, depth=1, mode=S.RM_NORMALS)
    o = H.oracle_frame(sd, cam, 97, 61, depth=1, mode=S.RM_NORMALS)
    assert g.float_pixels.tobytes() == o.float_pixels.tobytes()
    assert np.isfinite(g.float_pixels["depth"]).any()
