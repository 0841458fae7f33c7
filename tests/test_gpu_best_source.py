"""The best source and the maximum, which the kernel settles from an
approximate ranking where the lead allows, against the per-source NCCs it
reports: exact, with ties, textureless windows, infinities and NaN."""
import numpy as np
import pytest

from patchmatch_gb300 import native, scene

pytestmark = pytest.mark.gpu


def _first_argmax(ps):
    """Index of the first value no later one exceeds (a NaN in front stays)."""
    b = np.zeros(len(ps), np.int32)
    m = ps[:, 0].copy()
    for r in range(1, ps.shape[1]):
        with np.errstate(invalid="ignore"):
            g = ps[:, r] > m
        b[g] = r
        m = np.where(g, ps[:, r], m)
    return b


@pytest.mark.parametrize("n_src", [1, 2, 3, 6, 8, 9])
@pytest.mark.parametrize("combine", [native.COMBINE_FOLD, native.COMBINE_MAX])
@pytest.mark.parametrize("sampler", [native.SAMPLER_EXACT, native.SAMPLER_TEXTURE])
def test_best_source_matches_per_source(ctx, n_src, combine, sampler):
    W, H = 160, 80
    req = scene.make_request(scene.ROOM_OBJECTS, W, H, n_src, seed=40 + n_src, bmin=0.1, bmax=0.5)
    imgs = [v.gray_u8.astype(np.float16) for v in req.views]
    R, t = np.array(req.R), np.array(req.t)
    if n_src >= 3:  # two sources that tie everywhere
        imgs[3], R[3], t[3] = imgs[1].copy(), R[1], t[1]
    imgs[0][20:34, 30:60] = 7.0                     # textureless reference windows
    imgs[1][40:55, 60:90] = 120.0                   # and source windows
    imgs[n_src][10:12, 100:104] = np.inf
    imgs[1][60, 20:24] = np.nan
    p = native.default_params(combine=combine, sampler=sampler, image_format=native.IMAGE_F16)
    r = ctx.request(W, H, n_src, p)
    r.set_views(imgs, R, t)
    rng = np.random.default_rng(n_src)
    n = 20000
    ij = np.stack([rng.integers(6, H - 6, n), rng.integers(6, W - 6, n)], 1).astype(np.int32)
    d, nrm = req.views[0].depth[ij[:, 0], ij[:, 1]], req.views[0].normal[ij[:, 0], ij[:, 1]]
    lat, lon = -np.pi * (ij[:, 0] / H - 0.5), 2 * np.pi * (ij[:, 1] / W - 0.5)
    b = np.stack([np.cos(lat) * np.sin(lon), -np.sin(lat), np.cos(lat) * np.cos(lon)], 1)
    planes = (nrm / ((nrm * b).sum(1) * d)[:, None] * rng.uniform(0.9, 1.1, (n, 1))).astype(np.float32)
    scores, best, ps = r.score_hypotheses(ij, planes, per_source=True)
    scores2, best2 = r.score_hypotheses(ij, planes)
    r.close()
    assert np.array_equal(best, _first_argmax(ps))
    assert np.array_equal(best, best2) and np.array_equal(scores.view(np.int32), scores2.view(np.int32))
    if combine == native.COMBINE_MAX:
        want = np.fmax.reduce(ps, axis=1)
        assert np.array_equal(np.isnan(scores), np.isnan(want))
        ok = ~np.isnan(want)
        assert np.array_equal(scores[ok], want[ok])
    assert (ps == -1).any()  # the textureless windows were hit
