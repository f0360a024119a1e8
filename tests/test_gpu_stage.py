"""Large pageable copies of the ingestion calls: the plain way at first, then through page-locked slots
by several threads, and straight into page-locked destinations; the bytes are the same each time."""
import ctypes as C

import numpy as np
import pytest

from slimtracin_b200 import api, scenes, structs as S

pytestmark = pytest.mark.gpu


def bake(r, image, memory):
    h, w, _ = image.shape
    tex = S.Texture()
    assert r.L.st_bake_texture(r.ctx, image.ctypes.data, w, h, 24, 1, 1, C.byref(tex), memory.ctypes.data, memory.nbytes) == 0
    return memory[(C.sizeof(S.TextureMip) * tex.mip_count + 15) & ~15:].copy()


@pytest.mark.parametrize("size", [(1024, 1024), (1021, 700), (487, 491)])
def test_repeated_bakes_are_the_same_bytes(size):
    """487 x 491 is just above the staged size (a few slots, the last one partial)."""
    import torch
    w, h = size
    image = np.random.default_rng(w).integers(0, 256, (h, w, 3), dtype=np.uint8)
    want = scenes.bake_texture(image, True, True)
    want = np.concatenate([q.view(np.uint8).ravel() for _, _, q in want.mips])
    with api.Renderer(device=0) as r:
        need = r.L.st_texture_bytes(w, h, 1)
        for k in range(int((96 << 20) / need) + 3):
            assert np.array_equal(bake(r, image, np.zeros(need, np.uint8)), want), k
        locked = torch.zeros(need, dtype=torch.uint8, pin_memory=True).numpy()
        assert np.array_equal(bake(r, image, locked), want)


def test_repeated_mesh_builds_are_the_same_bytes():
    md = scenes.displaced_icosphere(6, seed=3)
    bad = scenes.displaced_icosphere(6, seed=3)
    bad.indices = bad.indices.copy()
    bad.indices[-1, 2] = len(bad.positions)
    with api.Renderer(device=0) as r:
        first = None
        for k in range(8):
            for mode in (api.ST_BVH_BINNED_SAH, api.ST_BVH_LBVH30):
                r.build_blas(md, mode)
            got = (md.node_count, md.nodes.tobytes(), md.leaf_ids.tobytes(), md.triangles.tobytes())
            first = first or got
            assert got == first, k
            # a vertex index out of range is refused, whatever way it was copied
            with pytest.raises(api.STError) as e:
                r.build_blas(bad, api.ST_BVH_BINNED_SAH)
            assert e.value.status == api.ST_ERR_BAD_SCENE
