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
