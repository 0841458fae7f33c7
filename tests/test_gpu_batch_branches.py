"""Batches whose groups run on parallel graph branches: an error in the middle
of a capture, and more groups in a level than branches."""
import numpy as np
import pytest

from patchmatch_gb300 import native, scene

pytestmark = pytest.mark.gpu

EXECUTORS = [native.BATCH_PERSISTENT, native.BATCH_LAUNCHES, native.BATCH_STREAMS, native.BATCH_MIXED]


def _request(ctx, W, H, S, seed, **kw):
    req = scene.make_request(scene.ROOM_OBJECTS, W, H, S, seed=seed)
    r = ctx.request(W, H, S, native.default_params(seed=seed, keyframe_id=seed, **{"iterations": 2, **kw}))
    imgs = [v.gray.astype(np.float16) if kw.get("image_format") == native.IMAGE_F16 else v.gray_u8 for v in req.views]
    r.set_views(imgs, req.R, req.t)
    return r


def _maps(r):
    return r.read(want=("depth", "score", "plane"))


def _same(a, b):
    return all(np.array_equal(a[k].view(np.int32), b[k].view(np.int32)) for k in a)


@pytest.mark.parametrize("executor", EXECUTORS)
def test_error_inside_a_capture_stays_with_its_batch(ctx, executor):
    """A prior that never ran is refused (PM_EINVAL); the next valid call of the
    context and the batch itself, once the prior has run, are not affected."""
    prior = _request(ctx, 96, 48, 2, 1)
    # two groups for every executor: the kinds of sampling differ
    rs = [_request(ctx, 96, 48, 2, 2), _request(ctx, 96, 48, 3, 3, sampler=native.SAMPLER_EXACT),
          _request(ctx, 96, 48, 4, 4)]
    rs[1].set_prior(prior)
    b = native.Batch(ctx, rs)
    b.set_executor(executor, 1)
    for _ in range(2):
        with pytest.raises(native.PmError) as e:
            b.run()
        assert e.value.status == native.PM_EINVAL
        other = _request(ctx, 96, 48, 2, 5)
        other.run()
        assert (other.read(want=("depth",))["depth"] > 0).any()
        other.close()
    prior.run()
    alone = []
    for r in rs:
        r.run()
        alone.append(_maps(r))
    b.run()
    for r, a in zip(rs, alone):
        assert _same(_maps(r), a)
    b.close()
    for r in rs + [prior]:
        r.close()


@pytest.mark.parametrize("executor", EXECUTORS)
def test_more_groups_than_branches(ctx, executor):
    kinds = [dict(), dict(sampler=native.SAMPLER_EXACT), dict(image_format=native.IMAGE_F16),
             dict(sampler=native.SAMPLER_EXACT, image_format=native.IMAGE_F16)]
    rs = [_request(ctx, 64 + 8 * S, 40, S, S) for S in range(1, 11)]  # ten groups by source count
    rs += [_request(ctx, 72, 36, 2 + q, 20 + q, iterations=1 + q % 3, **kinds[q % 4])  # twelve by the rest
           for q in range(8)]
    rs += [_request(ctx, 72, 36, 2, 30 + q, propagation=native.PROPAGATION_PLAIN, **kinds[q]) for q in range(4)]
    alone = []
    for r in rs:
        r.run()
        alone.append(_maps(r))
    b = native.Batch(ctx, rs)
    b.set_executor(executor, 1)
    for _ in range(2):
        b.run()
        for r, a in zip(rs, alone):
            assert _same(_maps(r), a), (r.W, r.S)
    b.close()
    for r in rs:
        r.close()
