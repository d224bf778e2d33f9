"""The gradients of the window convolutions at the edges of the canvas."""
import pytest

from test_unet_conv import L  # noqa: F401 - fixture
from test_unet_kernels import _gemm

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


@SIZES
@pytest.mark.parametrize("where", ["weight", "dz"])
def test_dx_with_infinities_and_nan(L, B, H, W, Cin, Cout, where):  # noqa: F811
    """The same for dX: the values that the GEMM and col2im give."""
    import torch
    if not L.unet_conv3x3_dx_fits(Cin, Cout):
        pytest.skip("dX of these channels goes through col2im")
    g = torch.Generator(device="cuda").manual_seed(W)
    M, kp = B * H * W, (9 * Cin + 7) // 8 * 8
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for q, y, x, v in _places(H, W):
        dz = torch.randn(M, Cout, device="cuda", generator=g).to(torch.bfloat16)
        Wt = torch.randn(kp, Cout, device="cuda", generator=g).to(torch.bfloat16)
        if where == "weight":
            Wt[q * Cin + 1, q % Cout] = v  # of tap q
        else:
            dz[y * W + x, q % Cout] = v
        dcol = torch.zeros(M, kp, device="cuda")
        d0 = torch.zeros(M, Cin, device="cuda")
        d1 = torch.zeros_like(d0)
        assert _gemm(L, dz, Wt, M, kp, Cout, 0, Cbuf=dcol) == 0
        assert L.unet_col2im(dcol.data_ptr(), B, H, W, Cin, kp, d0.data_ptr(), None) == 0
        assert L.unet_conv3x3_dx(dz.data_ptr(), Wt.data_ptr(), B, H, W, Cin, Cout, d1.data_ptr(), err.data_ptr(), None) == 0
        assert torch.equal(torch.isfinite(d0), torch.isfinite(d1)), (y, x)
        assert torch.equal(torch.nan_to_num(d0), torch.nan_to_num(d1)), (y, x)
    torch.cuda.synchronize()
    assert int(err.item()) == 0


@pytest.mark.parametrize("where", ["x", "weight"])
@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1, 20, 20, 32, 40), (2, 18, 13, 11, 16), (1, 33, 9, 144, 136)])
def test_forward_with_infinities_and_nan(L, B, H, W, Cin, Cout, where):  # noqa: F811
    """The same for the convolution itself (window and gathering kernel): the values of im2col and the GEMM."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(W)
    M, kp = B * H * W, (9 * Cin + 7) // 8 * 8
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for q, y, x, v in _places(H, W):
        X = torch.randn(M, Cin, device="cuda", generator=g).to(torch.bfloat16)
        Wt = torch.randn(Cout, kp, device="cuda", generator=g).to(torch.bfloat16)
        Wt[:, 9 * Cin:] = 0.0
        if where == "x":
            X[y * W + x, q % Cin] = v
        else:
            Wt[q % Cout, q * Cin + 1] = v  # of tap q
        col = torch.zeros(M, kp, dtype=torch.bfloat16, device="cuda")
        y0 = torch.zeros(M, Cout, dtype=torch.bfloat16, device="cuda")
        y1 = torch.zeros_like(y0)
        assert L.unet_im2col(X.data_ptr(), B, H, W, Cin, kp, col.data_ptr(), None) == 0
        assert _gemm(L, col, Wt, M, Cout, kp, 2, Y=y0) == 0
        if Cin % 16 == 0:
            assert L.unet_conv3x3(X.data_ptr(), B, H, W, Cin, Wt.data_ptr(), kp, Cout, 2, None, y1.data_ptr(), Cout, None, 0,
                                  err.data_ptr(), None) == 0
        else:
            assert L.unet_conv3x3_gather(X.data_ptr(), B, H, W, Cin, Wt.data_ptr(), kp, kp, Cout, y1.data_ptr(), Cout, None, 0,
                                         err.data_ptr(), None) == 0
        assert torch.equal(torch.isfinite(y0), torch.isfinite(y1)), (y, x)
        assert torch.equal(torch.nan_to_num(y0.float()), torch.nan_to_num(y1.float())), (y, x)
    torch.cuda.synchronize()
    assert int(err.item()) == 0


@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (3, 1, 2), (2, 2, 1), (1, 17, 9), (70, 3, 5)])
@pytest.mark.parametrize("Cin,Cout", [(16, 8), (11, 16), (32, 32), (3, 64)])
def test_tiny_canvases(L, B, H, W, Cin, Cout):  # noqa: F811
    """Canvases smaller than a tile, and just larger: the convolution and dX bit-identical to im2col, GEMM and
    col2im, dW within 2e-6 of the FP64 product's norm (at most 1050 products per sum, FP32)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(H * W + Cin)
    M, kp = B * H * W, (9 * Cin + 7) // 8 * 8
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    X = torch.randn(M, Cin, device="cuda", generator=g).to(torch.bfloat16)
    dz = torch.randn(M, Cout, device="cuda", generator=g).to(torch.bfloat16)
    Wt = torch.randn(Cout, kp, device="cuda", generator=g).to(torch.bfloat16)
    Wt[:, 9 * Cin:] = 0.0
    wt = Wt.t().contiguous()
    col = torch.zeros(M, kp, dtype=torch.bfloat16, device="cuda")
    y0 = torch.zeros(M, Cout, dtype=torch.bfloat16, device="cuda")
    y1 = torch.zeros_like(y0)
    assert L.unet_im2col(X.data_ptr(), B, H, W, Cin, kp, col.data_ptr(), None) == 0
    assert _gemm(L, col, Wt, M, Cout, kp, 2, Y=y0) == 0
    if Cin % 16 == 0:
        assert L.unet_conv3x3(X.data_ptr(), B, H, W, Cin, Wt.data_ptr(), kp, Cout, 2, None, y1.data_ptr(), Cout, None, 0,
                              err.data_ptr(), None) == 0
    else:
        assert L.unet_conv3x3_gather(X.data_ptr(), B, H, W, Cin, Wt.data_ptr(), kp, kp, Cout, y1.data_ptr(), Cout, None, 0,
                                     err.data_ptr(), None) == 0
    assert torch.equal(y0, y1)
    gw = torch.zeros(kp, Cout, device="cuda")
    assert L.unet_conv3x3_dw(X.data_ptr(), dz.data_ptr(), B, H, W, Cin, Cout, gw.data_ptr(), err.data_ptr(), None) == 0
    ref = col.double().t() @ dz.double()
    assert float((gw.double() - ref).norm()) <= 2e-6 * float(ref.norm())
    dcol = torch.zeros(M, kp, device="cuda")
    d0 = torch.zeros(M, Cin, device="cuda")
    d1 = torch.full((M, Cin), float("nan"), device="cuda")
    assert _gemm(L, dz, wt, M, kp, Cout, 0, Cbuf=dcol) == 0
    assert L.unet_col2im(dcol.data_ptr(), B, H, W, Cin, kp, d0.data_ptr(), None) == 0
    assert L.unet_conv3x3_dx(dz.data_ptr(), wt.data_ptr(), B, H, W, Cin, Cout, d1.data_ptr(), err.data_ptr(), None) == 0
    assert torch.equal(d0, d1)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
