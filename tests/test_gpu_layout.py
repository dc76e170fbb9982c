"""Layout passes, pooling and shortcut over whole and ragged quads: the 16-byte paths must give what the general ones give."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _x(shape, seed=0):
    import torch
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def _shifted(x):
    """The same values at an address that is 4 bytes off a 16-byte boundary."""
    import torch
    y = torch.empty(x.numel() + 4, device=x.device)[1:1 + x.numel()].view(x.shape)
    y.copy_(x)
    assert y.data_ptr() % 16 == 4
    return y


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 64, 8, 8), (3, 65, 8, 8), (2, 68, 7, 9), (1, 3, 33, 31), (2, 130, 16, 20)], ids=str)
def test_layout_convert(handle, shape):
    import torch
    from nebula_b200 import api
    B, C, H, W = shape
    x = _x(shape)
    for src in (x, _shifted(x)):
        nhwc = handle.layout_convert(src, B, C, H, W, api.LAYOUT_NCHW)
        assert torch.equal(nhwc, x.permute(0, 2, 3, 1))
        back = handle.layout_convert(_shifted(nhwc) if src is not x else nhwc, B, C, H, W, api.LAYOUT_NHWC)
        assert torch.equal(back, x)


@pytest.mark.parametrize("mode", ["max", "avg"])
@pytest.mark.parametrize("shape", [(1, 3, 2, 4), (2, 5, 6, 8), (2, 5, 7, 8), (2, 4, 6, 10), (3, 2, 56, 56)], ids=str)
def test_pool_nchw_quads(handle, shape, mode):
    import torch
    x = _x(shape)
    y = handle.pool(x, 2, 2, 0, mode)
    assert torch.equal(y, handle.pool(_shifted(x), 2, 2, 0, mode))
    want = (torch.nn.functional.max_pool2d if mode == "max" else torch.nn.functional.avg_pool2d)(x.double(), 2, 2)
    assert torch.allclose(y.double(), want, rtol=4 * 2.0 ** -24, atol=4 * 2.0 ** -24 * 4)


@pytest.mark.parametrize("act", ["linear", "leaky", "tanh"])
@pytest.mark.parametrize("shapes", [((2, 6, 4, 4), (2, 6, 4, 4)), ((2, 6, 4, 4), (2, 3, 4, 4)), ((2, 4, 6, 6), (2, 9, 6, 6)),
                                    ((1, 5, 3, 3), (1, 5, 3, 3)), ((2, 3, 4, 8), (2, 3, 8, 16))], ids=str)
def test_shortcut_nchw_quads(handle, shapes, act):
    import torch
    prev, conn = _x(shapes[0], 1), _x(shapes[1], 2)
    y = handle.shortcut(prev, conn, act)
    assert torch.equal(y, handle.shortcut(_shifted(prev), conn, act))


# (B, C, H, F, k): whole planes, long runs of pixels per image, single pixels of many images, runs of two and four
@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
@pytest.mark.parametrize("case", [(40, 64, 1, 48, 1), (8, 32, 7, 64, 1), (128, 32, 7, 40, 1), (128, 32, 13, 36, 1), (32, 32, 14, 64, 1), (130, 32, 14, 260, 1),
                                  (5, 64, 28, 33, 3), (16, 3, 28, 32, 3)], ids=str)
def test_convolution_to_nchw(handle, case, mode):
    """NCHW written by the epilogue or by a pass behind it: the NHWC result, bit for bit."""
    import torch
    from nebula_b200 import api
    B, C, H, F, k = case
    x, w, b = _x((B, C, H, H), 1), _x((F, C, k, k), 2) / (C * k * k) ** 0.5, _x((F,), 3)
    handle.set_math(mode)
    ys = []
    for layout, xi in ((api.LAYOUT_NCHW, x), (api.LAYOUT_NHWC, x.permute(0, 2, 3, 1).contiguous())):
        plan = api.Conv2d(handle, B, C, H, H, F, k, 1, k // 2, False, "leaky", layout)
        plan.set_weights(w, b)
        ys.append(plan.forward(xi))
        handle.synchronize()
        plan.close()
    assert torch.equal(ys[0], ys[1].permute(0, 3, 1, 2))
