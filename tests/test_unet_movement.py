"""The network's data movement in 16-byte vectors against the element-wise kernels, bit for bit.  Tensors that
do not start on a 16-byte boundary go element by element, so the same call on shifted copies is the reference."""
import pytest

from test_unet_conv import L  # noqa: F401 - fixture

pytestmark = pytest.mark.gpu


def _at(t, shift):
    """A copy of t that starts `shift` elements after a 16-byte boundary."""
    import torch
    b = torch.zeros(t.numel() + 16, dtype=t.dtype, device="cuda")
    v = b[shift:shift + t.numel()].view(t.shape)
    v.copy_(t)
    return v


def _both(t):
    return _at(t, 0), _at(t, 1)


@pytest.mark.parametrize("B,h,w,C,ld,c0", [(1, 1, 1, 8, 8, 0), (2, 3, 5, 8, 24, 8), (1, 7, 4, 32, 96, 64), (3, 4, 4, 16, 24, 0),
                                           (2, 5, 3, 12, 28, 16), (1, 6, 2, 4, 4, 0), (2, 2, 2, 5, 9, 3)])
def test_movement_kernels(L, B, h, w, C, ld, c0):  # noqa: F811
    import torch
    g = torch.Generator(device="cuda").manual_seed(C + ld)
    H, W = 2 * h, 2 * w
    bf = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    f32 = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    fine, coarse, wide = bf(B * H * W, C), bf(B * h * w, C), bf(B * H * W, ld)
    ffine, fcoarse, fwide = f32(B * H * W, C), f32(B * h * w, C), f32(B * H * W, ld)
    p = lambda t: t.data_ptr()  # noqa: E731
    calls = [
        (fine, torch.zeros_like(coarse), lambda x, y: L.unet_pool_fwd(p(x), B, H, W, C, p(y), None)),
        (coarse, wide, lambda x, y: L.unet_up_fwd(p(x), B, h, w, C, p(y), ld, c0, None)),
        (fine, wide, lambda x, y: L.unet_copy_channels(p(x), B * H * W, C, p(y), ld, c0, None)),
        (fwide, torch.zeros_like(fcoarse), lambda x, y: L.unet_up_bwd(p(x), ld, c0, B, h, w, C, p(y), None)),
    ]
    for acc in (0, 1):
        calls.append((fcoarse, ffine, lambda x, y, acc=acc: L.unet_pool_bwd(p(x), B, H, W, C, p(y), acc, None)))
        calls.append((fwide, ffine, lambda x, y, acc=acc: L.unet_take_channels(p(x), ld, c0, B * H * W, C, p(y), acc, None)))
    for k, (src, dst, call) in enumerate(calls):
        out = []
        for x, y in zip(_both(src), _both(dst)):
            assert call(x, y) == 0
            torch.cuda.synchronize()
            out.append(y.clone())
        assert torch.equal(out[0], out[1]), k


@pytest.mark.parametrize("B,H,W,C", [(1, 1, 1, 8), (2, 5, 7, 11), (1, 6, 3, 3), (3, 4, 5, 16), (1, 9, 9, 1)])
def test_im2col(L, B, H, W, C):  # noqa: F811
    import torch
    kp = (9 * C + 7) // 8 * 8
    X = torch.randn(B * H * W, C, device="cuda").to(torch.bfloat16)
    out = []
    for x, col in zip(_both(X), _both(torch.full((B * H * W, kp), 7.0, device="cuda", dtype=torch.bfloat16))):
        assert L.unet_im2col(x.data_ptr(), B, H, W, C, kp, col.data_ptr(), None) == 0
        torch.cuda.synchronize()
        out.append(col.clone())
    assert torch.equal(out[0], out[1])
