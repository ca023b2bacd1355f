"""The tcgen05 convolution with several position tiles per block, the weight gradient's ring of
positions, and the whole-network optimiser step, at the sizes where their tiles change; against
float64 sums by torch of the same bf16 values."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _taps(x, B, H, W, c):
    """[9][B*H*W][c] float64: x at every tap, zero outside the image."""
    import torch
    xp = torch.nn.functional.pad(x.double().reshape(B, H, W, c), (0, 0, 1, 1, 1, 1))
    return [xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(B * H * W, c) for t in range(9)]


# enough positions for two blocks per SM of the widest tile; ragged widths; every tile of Cout
@pytest.mark.parametrize("cin,cout,B,H,W", [(16, 16, 45, 64, 64), (32, 32, 40, 64, 64), (96, 32, 61, 41, 63),
                                            (32, 48, 40, 40, 50), (64, 64, 20, 64, 64), (32, 96, 20, 64, 64),
                                            (16, 136, 13, 64, 50), (32, 24, 1, 5, 3)])
def test_conv_tiles(cin, cout, B, H, W):
    import torch
    from mumax2 import _native as nat
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.randn(B * H * W, cin, device="cuda", generator=g).bfloat16()
    w = (torch.randn(cout, 9, cin, device="cuda", generator=g) / (9 * cin) ** 0.5).bfloat16()
    b = torch.randn(cout, device="cuda", generator=g)
    out = torch.zeros(B * H * W, cout, device="cuda", dtype=torch.bfloat16)
    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    nat.check(nat.lib().mm_nn_conv3x3_tc(_p(x), cin, 0, cin, _p(w), _p(b), _p(out), cout, 0, cout, B, H, W, 0, _p(err),
                                         None))
    ref = b.double() + sum(v @ w[:, t].double().t() for t, v in enumerate(_taps(x, B, H, W, cin)))
    assert int(err.item()) == 0
    # one bf16 rounding (2^-9 of the value) and FP32 sums of up to 864 products
    assert float(((out.double() - ref).abs() - 2.0 ** -8 * ref.abs()).max()) < 1e-4


# a ring of 256, 512 and 1024 positions, rows too long for it, channel remainders, and a
# gradient that is not 8-byte aligned
@pytest.mark.parametrize("cin,cout,B,H,W,shift", [(16, 32, 1, 3, 5, 0), (32, 32, 70, 8, 8, 0), (24, 40, 3, 17, 33, 0),
                                                  (96, 32, 2, 64, 64, 0), (64, 16, 2, 9, 200, 0), (8, 8, 1, 4, 413, 0),
                                                  (16, 32, 1, 3, 450, 0), (32, 64, 2, 16, 16, 1)])
def test_weight_gradient_ring(cin, cout, B, H, W, shift):
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


def test_network_step_equals_layer_steps():
    """mm_nn_adam_net against mm_nn_adam and mm_nn_flip per layer, bit for bit."""
    import torch
    from mumax2 import _native as nat
    from mumax2 import unet as U
    net = U.UNet(2, H=16, W=16, seed=3)
    g = torch.Generator(device="cuda").manual_seed(1)
    for _ in range(2):
        net.flat["g"].copy_(torch.randn(net.flat["g"].numel(), device="cuda", generator=g))
        want = {}
        for name, _, cin, _, cout, _ in U.CONVS:
            d = net.p[name]
            q = {k: d[k].clone() for k in ("w", "gw", "mw", "vw", "wb", "b", "gb", "mb", "vb", "wt")}
            for k, wb in (("w", _p(q["wb"])), ("b", None)):
                nat.check(nat.lib().mm_nn_adam(_p(q[k]), _p(q["g" + k]), _p(q["m" + k]), _p(q["v" + k]), q[k].numel(),
                                               1e-2, 0.9, 0.999, 1e-8, net.t + 1, wb, None))
            if name == "out":
                q["w"].reshape(cout, -1)[3:].zero_()
                q["wb"].copy_(q["w"].to(torch.bfloat16))
            nat.check(nat.lib().mm_nn_flip(_p(q["wb"]), cout, cin, _p(q["wt"]), d["cin_t"], cin, None))
            want[name] = q
        net.adam(lr=1e-2)
        for name, q in want.items():
            for k, v in q.items():
                assert torch.equal(net.p[name][k], v), (name, k)
