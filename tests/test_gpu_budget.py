"""What the ingestion calls take of the device for their own time counts against the context's budget, and
so does what the context keeps of it for the next call."""
import numpy as np
import pytest

from slimtracin_b200 import api, scenes
from tests import helpers as H

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_builds_and_what_is_kept_of_them_stay_within_the_budget():
    md = scenes.displaced_icosphere(6, seed=3)           # 81,920 triangles: 19 MB, and 15 of scratch for the binned builder
    with api.Renderer(device=0, memory_budget=30 * MB) as r:
        held = lambda: int(r.L.st_device_bytes_in_use(r.ctx))
        with pytest.raises(api.STError) as e:
            r.build_blas(md, api.ST_BVH_BINNED_SAH)
        assert e.value.status == api.ST_ERR_BUDGET
        r.build_blas(md, api.ST_BVH_LBVH30)
        assert held() <= 30 * MB
        sd, cam = scenes.moving_scene(count=4096)
        r.upload(0, sd, tlas="lbvh")
        g = H.gpu_frame(r, 0, sd, cam, 640, 360, depth=1)
        assert np.isfinite(g.float_pixels["depth"]).any() and held() <= 30 * MB
        r.build_blas(md, api.ST_BVH_LBVH30)
        assert held() <= 30 * MB
    with api.Renderer(device=0) as r:                    # room enough: the pool keeps its memory, and says so
        before = int(r.L.st_device_bytes_in_use(r.ctx))
        r.build_blas(md, api.ST_BVH_BINNED_SAH)
        assert 34 * MB <= int(r.L.st_device_bytes_in_use(r.ctx)) - before <= 512 * MB
