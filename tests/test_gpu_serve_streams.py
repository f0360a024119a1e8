"""Scene updates of the serving loop on their own stream, beside batches that still read the scene's
earlier versions: every frame is the one its own sequence of updates gives."""
import numpy as np
import pytest

from slimtracin_b200 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("in_flight", [1, 3])
@pytest.mark.parametrize("launch_mode", [api.LAUNCH_PER_VIEW, api.LAUNCH_PERSISTENT])
def test_updates_beside_batches_in_flight(launch_mode, in_flight):
    """Views of a scene that every request moves, refits and rebuilds in turn, large enough that the
    next update is made while the last frame is traced.  refit_fraction 0.25 of 400."""
    sd, cam = scenes.moving_scene(count=400)
    motion = sd.copy()
    rng = np.random.default_rng(11)
    served, alone = api.Renderer(device=0), api.Renderer(device=0)
    try:
        served.upload(0, sd.copy(), tlas="lbvh")
        alone.upload(0, sd.copy(), tlas="lbvh")
        srv = api.Server(served, max_in_flight=in_flight, refit_fraction=0.25, launch_mode=launch_mode)
        tickets, frames, updates = [], [], []
        try:
            for k in range(12):
                scenes.advance_moving_scene(motion, 1)
                ids = np.sort(rng.choice(400, 150 if k % 3 == 2 else 20, replace=False)).astype(np.uint32)
                updates.append((ids, motion.primitives[ids].copy()))
                frames.append(scenes.Frame(640, 360, cam, depth=2))
                tickets.append(srv.submit(0, sd, frames[-1], moved=updates[-1][1], moved_ids=ids))
            results = [srv.wait(t, timeout=60) for t in tickets]
        finally:
            srv.stop()
        assert all(r.status == api.ST_OK for r in results)
        moved = 0
        for (ids, records), frame in zip(updates, frames):
            alone.update_primitives(0, records, ids)
            moved += len(ids)
            refit = moved < 0.25 * 400
            moved = moved if refit else 0
            alone.build_tlas(0, sd.copy(), api.ST_BVH_REFIT if refit else api.ST_BVH_LBVH30)
            ref = scenes.Frame(640, 360, cam, depth=2)
            alone.render(0, sd, ref)
            assert np.array_equal(frame.float_pixels.view(np.uint8), ref.float_pixels.view(np.uint8))
            assert np.array_equal(frame.pixels.view(np.uint8), ref.pixels.view(np.uint8))
    finally:
        served.close()
        alone.close()
