"""The gradients of the window convolutions at the edges of the canvas."""
import pytest

from test_unet_conv import L  # noqa: F401 - fixture

pytestmark = pytest.mark.gpu


SIZES = pytest.mark.parametrize("B,H,W,Cin,Cout", [(1, 20, 20, 32, 32), (2, 18, 13, 11, 16), (1, 16, 16, 64, 8), (1, 33, 9, 136, 144)])


def _places(H, W):
    """Pixels at every edge and corner and inside, and the value to put there."""
    values = (float("inf"), float("-inf"), float("nan"))
    at = [(0, 0), (0, W - 1), (H - 1, 0), (H - 1, W - 1), (H // 2, W - 1), (H - 1, W // 2), (H // 2, W // 2)]
    return [(q, y, x, values[q % 3]) for q, (y, x) in enumerate(at)]


@SIZES
def test_dw_with_infinities_and_nan(L, B, H, W, Cin, Cout):  # noqa: F811
    """An infinite or NaN activation reaches exactly the weight gradients whose sum over the canvas (the
    column of im2col) holds it, also on canvases that tiles reach over."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(W)
    M, kp = B * H * W, (9 * Cin + 7) // 8 * 8
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for q, y, x, v in _places(H, W):
        X = torch.randn(M, Cin, device="cuda", generator=g).to(torch.bfloat16)
        dz = torch.randn(M, Cout, device="cuda", generator=g).to(torch.bfloat16)
        X[y * W + x, q % Cin] = v
        gw = torch.zeros(kp, Cout, device="cuda")
        assert L.unet_conv3x3_dw(X.data_ptr(), dz.data_ptr(), B, H, W, Cin, Cout, gw.data_ptr(), err.data_ptr(), None) == 0
        col = torch.zeros(M, kp, dtype=torch.bfloat16, device="cuda")
        assert L.unet_im2col(X.data_ptr(), B, H, W, Cin, kp, col.data_ptr(), None) == 0
        bad = ~torch.isfinite(col.float()).all(0)
        assert torch.equal(~torch.isfinite(gw), bad[:, None].expand(kp, Cout)), (y, x)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
