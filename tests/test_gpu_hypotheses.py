"""Fixed hypotheses scored by warps whose lanes share the taps: every count
around the warp and block sizes and each window size, bit for bit against the
tile kernel's scores and against the same hypotheses in other company."""
import numpy as np
import pytest

from patchmatch_gb300 import native, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("patch_half", [1, 3, 5])
@pytest.mark.parametrize("n_src", [1, 2, 3, 7, 10])
@pytest.mark.parametrize("sampler,fmt", [(native.SAMPLER_EXACT, native.IMAGE_U8),
                                         (native.SAMPLER_TEXTURE, native.IMAGE_F16)])
def test_hypotheses_share_warps(ctx, patch_half, n_src, sampler, fmt):
    W, H = 161, 80
    req = scene.make_request(scene.ROOM, W, H, n_src, seed=70 + n_src, noise_sigma=2.0)
    r = ctx.request(W, H, n_src, native.default_params(patch_half=patch_half, sampler=sampler, image_format=fmt,
                                                       iterations=0, postprocess=0))
    r.set_views([v.gray.astype(np.float16) if fmt == native.IMAGE_F16 else v.gray_u8 for v in req.views], req.R, req.t)
    r.init()
    g = r.read(raw=True)
    ii, jj = (a.ravel() for a in np.mgrid[patch_half + 1:H - patch_half, patch_half + 1:W - patch_half])
    ij = np.stack([ii, jj], 1).astype(np.int32)
    planes = np.ascontiguousarray(g["plane"][ii, jj, :3], np.float32)
    full = r.score_hypotheses(ij, planes, per_source=True)
    assert np.array_equal(full[0], g["score"][ii, jj], equal_nan=True)
    assert np.array_equal(full[1], g["best_view"][ii, jj])
    bits = [a.view(np.int32) for a in full]
    for k in (1, 31, 32, 33, 127, 128, 129, 1000):
        part = r.score_hypotheses(ij[-k:], planes[-k:], per_source=True)
        assert all(np.array_equal(a.view(np.int32), b[-k:]) for a, b in zip(part, bits)), k
    spoilt = planes.copy()  # what the neighbouring lanes hold does not matter
    spoilt[1::2] = np.nan
    odd = r.score_hypotheses(ij, spoilt, per_source=True)
    assert all(np.array_equal(a.view(np.int32)[::2], b[::2]) for a, b in zip(odd, bits))
    r.close()
