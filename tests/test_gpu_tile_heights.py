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


@pytest.mark.parametrize("n_src", [2, 8])
def test_height_follows_what_is_in_flight(ctx, n_src):
    """Requests run without waiting for each other take large tiles once the
    device is shared, and small ones again when they run alone: one after the
    other, in flight together (in both orders), and alone again give the same
    maps; a request destroyed with others in flight is no longer looked at."""
    W, H, n = 320, 160, 8
    want = ("depth", "score", "plane")
    rs = []
    for k in range(n):
        req = scene.make_request(scene.ROOM_OBJECTS, W, H, n_src, seed=80 + k)
        r = ctx.request(W, H, n_src, native.default_params(seed=k, iterations=3))
        r.set_views([v.gray_u8 for v in req.views], req.R, req.t)
        rs.append(r)
    alone = []
    for r in rs:
        r.run()
        alone.append(r.read(want=want))

    def same(r, a):
        got = r.read(want=want)
        return all(np.array_equal(got[k].view(np.int32), a[k].view(np.int32)) for k in want)

    for order in (range(n), range(n - 1, -1, -1)):
        for k in order:
            rs[k].run()
        assert all(same(r, a) for r, a in zip(rs, alone))
    for r in rs:
        r.init()
        r.sweep(0, 6)
        r.postprocess()
    assert all(same(r, a) for r, a in zip(rs, alone))
    for r in rs:
        r.run()
    rs.pop().close()
    rs[0].run()
    assert all(same(r, a) for r, a in zip(rs, alone))
    rs[0].synchronize()
    rs[0].run()
    assert same(rs[0], alone[0])
    for r in rs:
        r.close()


def test_running_leaves_an_open_capture_alone(ctx):
    """pm_request_run with other requests in flight, inside a capture that the
    caller has open on another stream: the launches of a captured run are legal
    there, and looking at what is in flight must stay so."""
    import torch
    rs = []
    for k in range(3):
        req = scene.make_request(scene.ROOM_OBJECTS, 192, 96, 2, seed=90 + k)
        r = ctx.request(192, 96, 2, native.default_params(seed=k, iterations=2))
        r.set_views([v.gray_u8 for v in req.views], req.R, req.t)
        r.run()
        r.synchronize()
        rs.append(r)
    for r in rs[:2]:  # the graph of either height
        for q in rs:
            q.run()
        for q in rs:
            q.synchronize()
    want = rs[0].read(want=("depth",))["depth"]
    x = torch.zeros(1000, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x += 1
        rs[1].run()
        rs[0].run()
    g.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 1000.0
    assert np.array_equal(rs[0].read(want=("depth",))["depth"], want)
    for r in rs:
        r.close()
