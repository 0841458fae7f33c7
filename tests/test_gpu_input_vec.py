"""Input preparation at the edges of its 16-byte kernels: tails, padded and
unaligned rows, odd heights and the half-size resize, bit-exact against the
oracle's restatements."""
import numpy as np
import pytest

from oracle import oracle as O
from patchmatch_gb300 import native

pytestmark = pytest.mark.gpu


def _padded(torch, img, pitch, offset):
    """img's rows at `pitch` bytes from `offset` bytes into a fresh device buffer."""
    H, row = img.shape[0], int(np.prod(img.shape[1:])) * img.itemsize
    buf = torch.zeros(offset + pitch * H + 64, dtype=torch.uint8, device="cuda")
    v = buf[offset:offset + pitch * H].view(H, pitch)
    v[:, :row] = torch.from_numpy(np.ascontiguousarray(img).view(np.uint8).reshape(H, row)).cuda()
    torch.cuda.synchronize()
    return buf, buf.data_ptr() + offset


# packed (one long row, with and without a tail), padded aligned rows, rows off the boundary
@pytest.mark.parametrize("W,H,pad,offset", [(16, 1, 0, 0), (7, 3, 0, 0), (64, 5, 0, 0), (33, 9, 15, 0), (40, 6, 8, 0),
                                            (40, 6, 0, 4)])
@pytest.mark.parametrize("ch", [1, 3, 4])
def test_gray_rows(ctx, W, H, pad, offset, ch):
    import torch
    rng = np.random.default_rng(W + ch)
    img = rng.integers(0, 256, (H, W, ch) if ch > 1 else (H, W), dtype=np.uint8)
    pitch, dpitch = W * ch + pad * ch, W + pad
    src, sp = _padded(torch, img, pitch, offset)
    dst, dp = _padded(torch, np.zeros((H, W), np.uint8), dpitch, offset)
    assert native.lib().pm_image_to_gray(ctx.h, sp, W, H, pitch, ch, native.ORDER_BGR, dp, dpitch) == 0
    torch.cuda.synchronize()
    got = dst[offset:offset + dpitch * H].view(H, dpitch).cpu().numpy()
    assert np.array_equal(got[:, :W], O.to_gray(img[..., :3] if ch == 4 else img, rgb=False))
    assert not got[:, W:].any() and not dst[offset + dpitch * H:].any()


@pytest.mark.parametrize("dw,dh,pad", [(8, 1, 0), (16, 5, 0), (11, 3, 10), (24, 4, 16), (13, 7, 0)])
@pytest.mark.parametrize("ch", [1, 2, 3, 4])
def test_half_size(ctx, dw, dh, pad, ch):
    import torch
    rng = np.random.default_rng(dw + ch)
    img = rng.integers(0, 256, (2 * dh, 2 * dw, ch), dtype=np.uint8)
    img[0, 0] = 255
    src, sp = _padded(torch, img, 2 * dw * ch + pad * ch, 0)
    dpitch = (dw * ch + 7) // 8 * 8 if pad else dw * ch
    dst, dp = _padded(torch, np.zeros((dh, dw, ch), np.uint8), dpitch, 0)
    rc = native.lib().pm_image_resize(ctx.h, sp, 2 * dw, 2 * dh, 2 * dw * ch + pad * ch, ch, dp, dw, dh, dpitch)
    assert rc == 0
    torch.cuda.synchronize()
    got = dst[:dpitch * dh].view(dh, dpitch).cpu().numpy()
    want = np.stack([O.resize_linear(np.ascontiguousarray(img[..., c]), dw, dh) for c in range(ch)], -1)
    assert np.array_equal(got[:, :dw * ch].reshape(dh, dw, ch), want)
    assert not got[:, dw * ch:].any() and not dst[dpitch * dh:].any()


@pytest.mark.parametrize("W,H,levels", [(16, 8, 4), (24, 7, 3), (40, 5, 4), (33, 3, 3), (1, 1, 2), (8, 1, 3)])
@pytest.mark.parametrize("f16", [False, True])
def test_pyramid_rows(ctx, W, H, levels, f16):
    import torch
    rng = np.random.default_rng(W * H)
    img = rng.integers(0, 256, (H, W), dtype=np.uint8)
    src = torch.from_numpy(img.astype(np.float16) if f16 else img).cuda()
    got = [t.cpu().numpy() for t in ctx.pyramid_f16(src, levels)]
    for a, b in zip(got, O.pyramid_f16(img, levels)):
        assert a.shape == b.shape and np.array_equal(a.view(np.uint16), b.view(np.uint16))
