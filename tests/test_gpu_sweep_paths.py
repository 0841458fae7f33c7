"""The sweep kernel's shortcuts leave every map bit-identical.

Within one call of several half-sweeps a pixel skips propagation candidates
that neither it nor they changed since its last visit; half-sweeps enqueued
one call at a time never skip.  The skip is exact, so the maps are equal bit
for bit (no tolerance)."""
import numpy as np
import pytest

from patchmatch_gb300 import native, scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with native.Context(0) as c:
        yield c


def _request(ctx, W, H, S, seed, **kw):
    req = scene.make_request(scene.ROOM_OBJECTS, W, H, S, seed=seed, bmin=0.1, bmax=0.5)
    r = ctx.request(W, H, S, native.default_params(seed=seed, iterations=5, **kw))
    r.set_views([v.gray_u8 for v in req.views], req.R, req.t)
    return r


# sizes around the 64 x 8 tile and the window (16 is the smallest image)
@pytest.mark.parametrize("W,H,S,kw", [
    (16, 16, 1, dict(patch_half=1)),
    (63, 33, 2, dict(patch_half=1)),
    (64, 40, 3, dict(patch_half=3, combine=native.COMBINE_MAX)),
    (129, 65, 4, dict(combine=native.COMBINE_TOPK)),
    (200, 101, 6, dict(combine=native.COMBINE_FOLD_SEPARATE, sampler=native.SAMPLER_EXACT)),
    (131, 67, 9, dict()),
    (131, 67, 3, dict(propagation=native.PROPAGATION_PLAIN, patch_half=1)),
    (257, 129, 5, dict(propagation=native.PROPAGATION_PLAIN, combine=native.COMBINE_MAX,
                       sampler=native.SAMPLER_EXACT, seam=native.SEAM_ZERO)),
    (640, 320, 2, dict(propagation=native.PROPAGATION_PLAIN)),
    (192, 96, 2, dict(sampler=native.SAMPLER_EXACT, seam=native.SEAM_WRAP)),
])
def test_skipping_unchanged_candidates_is_exact(ctx, W, H, S, kw):
    r = _request(ctx, W, H, S, 7 + S, **kw)
    r.init()
    r.sweep(0, 10)
    whole = r.read(raw=True)
    r.init()
    for h in range(10):
        r.sweep(h, 1)
    single = r.read(raw=True)
    r.close()
    for k in whole:
        assert np.array_equal(whole[k].view(np.int32), single[k].view(np.int32)), k
