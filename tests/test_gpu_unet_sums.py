"""The weight gradient on both sides of the line between its kernels, with every size of the ring
of positions; against float64 sums by torch of the same bf16 values."""
import pytest

from test_gpu_unet_tiles import _p, _taps

pytestmark = pytest.mark.gpu


# the kernel that stages each tap: one position to just below the line, channel remainders; the
# ring: 256, 512 and 1024 positions (413 pixels a row the last that fits), remainders, and a
# gradient that is not 8-byte aligned
@pytest.mark.parametrize("cin,cout,B,H,W,shift", [(8, 8, 1, 1, 1, 0), (16, 32, 3, 7, 5, 0), (32, 32, 128, 8, 8, 0),
                                                  (24, 40, 13, 17, 33, 0), (128, 256, 1, 32, 32, 1),
                                                  (32, 32, 170, 8, 8, 0), (16, 32, 500, 3, 5, 0),
                                                  (24, 40, 20, 17, 33, 0), (64, 16, 6, 9, 200, 0),
                                                  (8, 8, 6, 4, 413, 0), (96, 136, 4, 20, 30, 0),
                                                  (32, 64, 32, 16, 16, 1)])
def test_weight_gradient(cin, cout, B, H, W, shift):
    import torch
    from mumax2 import _native as nat
    g = torch.Generator(device="cuda").manual_seed(cin * cout + W)
    x = torch.randn(B * H * W, cin, device="cuda", generator=g).bfloat16()
    dy = torch.randn(B * H * W, cout, device="cuda", generator=g).bfloat16()
    buf = torch.zeros(cout * 9 * cin + shift, device="cuda")
    dw = buf[shift:]
    nat.check(nat.lib().mm_nn_conv3x3_wgrad(_p(dy), cout, 0, cout, _p(x), cin, 0, cin, _p(dw), B, H, W, None))
    ref = torch.stack([dy.double().t() @ v for v in _taps(x, B, H, W, cin)], 1).reshape(-1)
    # FP32 sums of P products in a few hundred partial sums: eps * sqrt(P) of the norm and more
    assert float((dw.double() - ref).norm() / ref.norm()) < 1e-5
