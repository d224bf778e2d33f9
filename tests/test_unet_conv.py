"""The window convolutions against im2col + GEMM, bit for bit (same K order)."""
import pytest

from test_unet_kernels import _gemm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L(gpu):
    import importlib
    return importlib.import_module("solver_cfd_b200.unet").kernels()


@pytest.mark.parametrize("B,H,W,Cc,Cout", [(1, 8, 8, 16, 8), (1, 33, 17, 48, 40), (3, 16, 24, 112, 128),
                                            (1, 20, 20, 384, 128), (2, 40, 20, 256, 256), (40, 64, 40, 64, 64)])
def test_window_conv_sizes(L, B, H, W, Cc, Cout):
    """The window kernel at partial tiles, K tails, one and two tiles per CTA and its largest window
    against im2col + GEMM, bit for bit (same K order)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(Cc + Cout)
    M, K = B * H * W, 9 * Cc
    X = torch.randn(M, Cc, device="cuda", generator=g).to(torch.bfloat16)
    Wt = torch.randn(Cout, K, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(Cout, device="cuda", generator=g)
    col = torch.zeros(M, K, dtype=torch.bfloat16, device="cuda")
    y0 = torch.zeros(M, Cout, device="cuda")
    y1 = torch.zeros_like(y0)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert L.unet_im2col(X.data_ptr(), B, H, W, Cc, K, col.data_ptr(), None) == 0
    assert _gemm(L, col, Wt, M, Cout, K, 3, Cbuf=y0, bias=bias) == 0
    assert L.unet_conv3x3(X.data_ptr(), B, H, W, Cc, Wt.data_ptr(), K, Cout, 3, y1.data_ptr(), None, Cout,
                          bias.data_ptr(), 0, err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and torch.equal(y0, y1)


@pytest.mark.parametrize("B,H,W,Cc,Cout", [(1, 8, 8, 11, 32), (2, 33, 20, 11, 48), (1, 16, 16, 3, 64), (1, 9, 7, 1, 5)])
def test_gathering_conv_equals_im2col_gemm(L, B, H, W, Cc, Cout):
    import torch
    g = torch.Generator(device="cuda").manual_seed(Cc + Cout)
    M, K = B * H * W, (9 * Cc + 7) // 8 * 8
    X = torch.randn(M, Cc, device="cuda", generator=g).to(torch.bfloat16)
    Wt = torch.randn(Cout, K, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(Cout, device="cuda", generator=g)
    col = torch.zeros(M, K, dtype=torch.bfloat16, device="cuda")
    y0 = torch.zeros(M, Cout, dtype=torch.bfloat16, device="cuda")
    y1 = torch.zeros_like(y0)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert L.unet_im2col(X.data_ptr(), B, H, W, Cc, K, col.data_ptr(), None) == 0
    assert _gemm(L, col, Wt, M, Cout, K, 2, Y=y0, bias=bias, relu=1) == 0
    assert L.unet_conv3x3_gather(X.data_ptr(), B, H, W, Cc, Wt.data_ptr(), K, K, Cout, y1.data_ptr(), Cout,
                                 bias.data_ptr(), 1, err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and torch.equal(y0, y1)


@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1, 16, 8, 32, 32), (2, 33, 20, 11, 32), (1, 20, 20, 32, 8), (3, 24, 16, 96, 32),
                                            (1, 40, 40, 384, 128), (2, 20, 20, 256, 256), (14, 32, 32, 64, 64)])
def test_window_conv_gradients(L, B, H, W, Cin, Cout):
    """dX bit-identical to GEMM + col2im; dW against an FP64 product within 2e-6 of its norm: at most
    1536 products of 16 per sum in tensor memory, the rest FP32 atomics (unit roundoff 6e-8, error growth
    with the square root of the number of terms)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(Cin + Cout)
    M, kp = B * H * W, (9 * Cin + 7) // 8 * 8
    X = torch.randn(M, Cin, device="cuda", generator=g).to(torch.bfloat16)
    dz = torch.randn(M, Cout, device="cuda", generator=g).to(torch.bfloat16)
    Wt = torch.randn(kp, Cout, device="cuda", generator=g).to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    gw = torch.zeros(kp, Cout, device="cuda")
    assert L.unet_conv3x3_dw(X.data_ptr(), dz.data_ptr(), B, H, W, Cin, Cout, gw.data_ptr(), err.data_ptr(), None) == 0
    col = torch.zeros(M, kp, dtype=torch.bfloat16, device="cuda")
    assert L.unet_im2col(X.data_ptr(), B, H, W, Cin, kp, col.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = col.double().t() @ dz.double()
    assert float((gw.double() - ref).norm() / ref.norm()) < 2e-6
    if L.unet_conv3x3_dx_fits(Cin, Cout):
        dcol = torch.zeros(M, kp, device="cuda")
        d0 = torch.zeros(M, Cin, device="cuda")
        d1 = torch.full((M, Cin), float("nan"), device="cuda")
        assert _gemm(L, dz, Wt, M, kp, Cout, 0, Cbuf=dcol) == 0
        assert L.unet_col2im(dcol.data_ptr(), B, H, W, Cin, kp, d0.data_ptr(), None) == 0
        assert L.unet_conv3x3_dx(dz.data_ptr(), Wt.data_ptr(), B, H, W, Cin, Cout, d1.data_ptr(), err.data_ptr(), None) == 0
        torch.cuda.synchronize()
        assert int(err.item()) == 0 and torch.equal(d0, d1)


@pytest.mark.parametrize("M,Cc,relu", [(1000, 8, 0), (777, 32, 1), (64, 96, 1), (130, 256, 1)])
def test_activation_and_bias_gradient_in_one_pass(L, M, Cc, relu):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M)
    dy = torch.randn(M, Cc, device="cuda", generator=g)
    y = torch.randn(M, Cc, device="cuda", generator=g).to(torch.bfloat16)
    z0 = torch.zeros(M, Cc, dtype=torch.bfloat16, device="cuda")
    z1 = torch.zeros_like(z0)
    db = torch.zeros(Cc, device="cuda")
    assert L.unet_act_bwd(dy.data_ptr(), y.data_ptr(), M * Cc, relu, z0.data_ptr(), None) == 0
    assert L.unet_act_bias_bwd(dy.data_ptr(), y.data_ptr(), M, Cc, relu, z1.data_ptr(), db.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(z0, z1)
    ref = z0.double().sum(0)
    assert float((db.double() - ref).abs().max()) < 1e-5 * float(z0.double().abs().sum(0).max())
