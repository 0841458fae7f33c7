"""The consistency filter, which leaves a pixel at the view that settles it,
against the votes of each view on its own: exact for every threshold."""
import numpy as np
import pytest

from patchmatch_gb300 import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 5, 8])
@pytest.mark.parametrize("reproj_px", [0.0, 1.0])
def test_filter_counts_votes(ctx, n, reproj_px):
    W, H = 131, 66
    sc = scene.Scene(scene.ROOM_OBJECTS, 5)
    R, t = sc.poses(n, 5, 0.1, 0.4, 15.0)
    rng = np.random.default_rng(n)
    maps = []
    for v in range(n):
        d = sc.render(R[v], t[v], W, H).depth
        d = d * (1 + 0.006 * rng.standard_normal((H, W))).astype(np.float32)
        d[rng.random((H, W)) < 0.05] = 0
        maps.append(np.ascontiguousarray(d))
    d0 = maps[0]
    votes = (d0 > 1e-6).astype(int)
    for k in range(1, n):
        pair = ctx.filter_consistency([d0, maps[k]], R[[0, k]], t[[0, k]], 0, 0.01, min_consistent=2,
                                      reproj_px=reproj_px)
        votes += pair != 0
    assert len(np.unique(votes)) > 2
    for m in range(0, n + 2):
        out = ctx.filter_consistency(maps, R, t, 0, 0.01, min_consistent=m, reproj_px=reproj_px)
        assert np.array_equal(out, np.where((votes >= m) & (d0 > 1e-6), d0, 0)), m
