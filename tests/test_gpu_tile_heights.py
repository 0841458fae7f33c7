"""Both tile heights of the sweep kernel on either side of the rule that picks
one: a request's own run (small tiles where the rule says so) and the queue of
the batched executor (large tiles always) give the same maps, bit for bit."""
import numpy as np
import pytest

from patchmatch_gb300 import native, scene

pytestmark = pytest.mark.gpu


# 7 sources: small by the warps per SM; 8: only where the fullest SM gets fewer
# rows (256x128 and 448x224 small, 320x160 and 512x256 large)
@pytest.mark.parametrize("W,H,S", [(512, 256, 7), (256, 128, 8), (320, 160, 8), (448, 224, 8), (512, 256, 8)])
@pytest.mark.parametrize("sampler", [native.SAMPLER_TEXTURE, native.SAMPLER_EXACT])
def test_tile_heights_agree(ctx, W, H, S, sampler):
    req = scene.make_request(scene.ROOM_OBJECTS, W, H, S, seed=60 + S)
    r = ctx.request(W, H, S, native.default_params(seed=S, iterations=3, sampler=sampler))
    r.set_views([v.gray_u8 for v in req.views], req.R, req.t)
    want = ("depth", "score", "plane")
    r.run()
    alone = r.read(want=want)
    b = native.Batch(ctx, [r])
    for executor in (native.BATCH_PERSISTENT, native.BATCH_STREAMS):
        b.set_executor(executor, 1)
        b.run()
        got = r.read(want=want)
        assert all(np.array_equal(got[k].view(np.int32), alone[k].view(np.int32)) for k in want), executor
    b.close()
    r.close()
