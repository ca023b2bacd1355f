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


# channel groups that are powers of two and not, one pixel, remainders of the pixels in flight and
# of the blocks, channel views; the masked gradient is exact, its sums are of up to 30000 bf16
# values in FP32 (eps * sqrt(P) of their norm and more)
@pytest.mark.parametrize("C,P", [(8, 1), (8, 4099), (24, 777), (32, 30011), (40, 13), (96, 5003), (256, 601), (384, 1999),
                                 (512, 300)])
@pytest.mark.parametrize("relu", [0, 1])
def test_relu_and_bias(C, P, relu):
    import torch
    from mumax2 import _native as nat
    g = torch.Generator(device="cuda").manual_seed(C + P)
    out = torch.randn(P, C + 8, device="cuda", generator=g).bfloat16()
    d = torch.randn(P, C + 16, device="cuda", generator=g).bfloat16()
    db = torch.ones(C, device="cuda")
    want = d.clone()
    if relu:
        want[:, 16:] = torch.where(out[:, 8:] > 0, d[:, 16:], torch.zeros_like(d[:, 16:]))
    nat.check(nat.lib().mm_nn_relu_bias_bwd(_p(out), C + 8, 8, _p(d), C + 16, 16, C, P, relu, _p(db), None))
    assert torch.equal(d, want)
    ref = 1 + want[:, 16:].double().sum(0)
    assert float((db.double() - ref).abs().max()) < 1e-5 * max(1.0, P ** 0.5)


def test_parameters_of_another_network():
    """A network takes another one's device tensors, arrays of any float type and plain lists, and
    refuses layers of other sizes."""
    import numpy as np
    import torch
    from mumax2 import unet as U
    a = U.UNet(1, H=16, W=16, seed=5)
    forms = {"tensors": lambda t: t, "doubles": lambda t: t.cpu().numpy().astype(np.float64), "lists": lambda t: t.tolist()}
    for form in forms.values():
        b = U.UNet(2, H=16, W=16, params={n: (form(d["w"]), form(d["b"])) for n, d in a.p.items()})
        for n, d in a.p.items():
            for k in ("w", "b", "wb", "wt"):
                assert torch.equal(d[k], b.p[n][k]), (n, k)
    b.p["out"]["w"].add_(1.0)   # the copies are the network's own
    assert not torch.equal(a.p["out"]["w"], b.p["out"]["w"])
    short = {n: (d["w"], d["b"]) for n, d in a.p.items()}
    first = next(iter(short))
    short[first] = (short[first][0][:-1], short[first][1])
    with pytest.raises(ValueError, match=first):
        U.UNet(1, H=16, W=16, params=short)
