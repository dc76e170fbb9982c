"""1x1 convolutions of many tiles with the shortcut folded in through shared memory: columns that end inside a tile and inside a slab,
connections of fewer channels and of larger planes, ragged planes, one K block and sixteen; the bits of the convolution and the
shortcut one after the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (B, C, H, W, F, channels of the connection, its plane relative to the output, activation)
CASES = [(32, 32, 28, 28, 256, 256, 1, "relu"), (9, 64, 53, 47, 160, 160, 1, "relu"), (20, 96, 30, 31, 132, 36, 1, "leaky"),
         (24, 512, 28, 28, 200, 100, 2, "relu"), (64, 64, 17, 19, 64, 64, 1, "linear"), (40, 128, 25, 25, 292, 292, 1, "leaky")]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_folded_shortcut(handle, case):
    import torch
    from nebula_b200 import api
    B, C, H, W, F, rc, s, act = case
    g = torch.Generator(device="cuda").manual_seed(F)
    x = torch.randn(B, H, W, C, device="cuda", generator=g)
    w = torch.randn(F, C, 1, 1, device="cuda", generator=g) * (2.0 / C) ** 0.5
    b = torch.randn(F, device="cuda", generator=g)
    bn = (torch.rand(F, device="cuda", generator=g) + 0.5, torch.randn(F, device="cuda", generator=g), torch.rand(F, device="cuda", generator=g) + 0.5)
    r = torch.randn(B, s * H, s * W, rc, device="cuda", generator=g)
    handle.set_math("tf32")
    plan = api.Conv2d(handle, B, C, H, W, F, 1, 1, 0, True, "linear", api.LAYOUT_NHWC)
    plan.set_weights(w, b, bn)
    fused = [plan.forward_fused(x, residual=r, res_act=act) for _ in range(2)]
    y = plan.forward(x)
    handle.synchronize()
    plan.close()
    y[..., :rc] += r[:, ::s, ::s]
    want = {"relu": lambda v: v.clamp(min=0), "linear": lambda v: v, "leaky": lambda v: torch.where(v > 0, v, (0.1 * v.double()).float())}[act](y)
    assert torch.equal(fused[0], want) and torch.equal(fused[1], want)
