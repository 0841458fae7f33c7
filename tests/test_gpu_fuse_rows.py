"""Fusion at the edges of its vector kernels: widths and pixel counts that are
no multiple of 4 or 16, more compaction blocks than one step of the scan holds,
maps off a 16-byte boundary and on both sides of the size from which a thread
takes four pixels, against the sequential oracle and the aligned call."""
import numpy as np
import pytest

from oracle import oracle as O
from patchmatch_gb300 import native, scene

pytestmark = pytest.mark.gpu


def _holed(rng, W, H, drop=0.1):
    d = rng.uniform(0.5, 9.0, (H, W)).astype(np.float32)
    d[rng.random((H, W)) < drop] = 0
    return d


def _views(W, H, n, seed):
    req = scene.make_request(scene.ROOM_OBJECTS, W, H, n - 1, seed=seed, bmin=0.1, bmax=0.4)
    rng = np.random.default_rng(seed)
    maps = []
    for v in req.views:
        d = v.depth.copy()
        d[rng.random(d.shape) < 0.05] = 0
        maps.append(d)
    return req, maps


# One view: which pixels are kept takes no arithmetic, so pixels, order, colours
# and maps are the oracle's exactly; the points are those of the FP64 oracle
# within the FP32 rounding of coordinates up to 10 m (1e-5).  The last three
# have 4,104, 7,206 and 7,200 blocks of 1,024 pixels (the scan takes 4,096 a step).
@pytest.mark.parametrize("W,H", [(2, 2), (3, 2), (5, 3), (7, 7), (33, 31), (131, 67), (1025, 4), (2050, 2050),
                                 (3841, 1921), (3840, 1920)])
def test_one_view_is_exact(ctx, W, H):
    rng = np.random.default_rng(W + H)
    d = _holed(rng, W, H, 0.02)
    bgr = rng.integers(0, 256, (H, W, 3), dtype=np.uint8)
    R, t = np.eye(3)[None], np.array([[0.1, -0.2, 0.3]])
    gp, gx, gc, gij, gm = ctx.fuse([d], R, t, bgr, 0.02)
    op, ox, oc, oij, om = O.prune([d], R, t, bgr, 0.02)
    assert np.array_equal(gp, op) and np.array_equal(gm[0], om[0])
    assert np.array_equal(gij, oij) and np.array_equal(gc, oc)
    assert np.array_equal(gij, np.argwhere(gp != 0))
    assert np.allclose(gx, ox, rtol=0, atol=1e-5)


# Several views, one pixel per thread and (the last, above 700,000 pixels) four:
# keep decisions as far from the oracle as the other fusion tests allow (99.9 %),
# the list in raster order.
@pytest.mark.parametrize("W,H,n", [(131, 67, 5), (333, 166, 4), (642, 321, 3), (1240, 600, 3)])
def test_views_match_the_oracle(ctx, W, H, n):
    req, maps = _views(W, H, n, 11 + n)
    bgr = req.views[0].rgb
    gp, gx, gc, gij, gm = ctx.fuse(maps, req.R, req.t, bgr, 0.02)
    op, ox, oc, oij, om = O.prune(maps, req.R, req.t, bgr, 0.02)
    assert ((gp > 0) == (op > 0)).mean() >= 0.999
    for a, b in zip(gm[1:], om[1:]):
        assert ((a == 0) == (b == 0)).mean() >= 0.999
    assert np.array_equal(gij, np.argwhere(gp != 0))
    assert np.array_equal(gc, bgr[gij[:, 0], gij[:, 1]])
    assert 0 < len(gx) < W * H


# The same maps on and off a 16-byte boundary: from 700,000 pixels, four pixels
# or one per thread.
@pytest.mark.parametrize("W,H,n", [(132, 67, 5), (4, 5, 2), (1168, 600, 2), (1240, 600, 5)])
@pytest.mark.parametrize("moved", ["first", "others", "pruned"])
def test_unaligned_maps_give_the_same_bits(ctx, W, H, n, moved):
    import torch
    req, maps = _views(W, H, n, 21 + n) if W > 16 else (None, None)
    if req is None:
        rng = np.random.default_rng(3)
        maps = [_holed(rng, W, H) for _ in range(n)]
        R, t = np.eye(3)[None].repeat(n, 0), 0.01 * np.arange(3 * n).reshape(n, 3)
    else:
        R, t = np.array(req.R), np.array(req.t)
    ws_bytes = native.fuse_workspace_bytes(W, H)
    out = []
    for off in (0, 1):
        def place(a, by):
            buf = torch.zeros(W * H + 8, device="cuda")
            v = buf[by:by + W * H].view(H, W)
            v.copy_(torch.from_numpy(a))
            return v
        dev = [place(m, off if moved == ("first" if k == 0 else "others") else 0) for k, m in enumerate(maps)]
        pruned = place(np.full((H, W), -5.0, np.float32), off if moved == "pruned" else 0)
        ws = torch.empty(ws_bytes + 256, dtype=torch.uint8, device="cuda")
        xyz = torch.zeros((H * W, 3), device="cuda")
        ij = torch.zeros((H * W, 2), dtype=torch.int32, device="cuda")
        count = torch.zeros(1, dtype=torch.int32, device="cuda")
        ctx.fuse_device([d.data_ptr() for d in dev], W, H, R, t, 0.02, pruned.data_ptr(), xyz.data_ptr(),
                        count.data_ptr(), (ws.data_ptr() + 255) & ~255, ws_bytes, ij_ptr=ij.data_ptr(),
                        stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        out.append([a.cpu().numpy() for a in (pruned, xyz, ij, count, *dev)])
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.int32), b.view(np.int32))
