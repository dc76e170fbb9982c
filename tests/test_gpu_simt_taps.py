"""fp32 convolutions on the CUDA cores, whose copies advance from tap to tap: taps of less than a block of 16 columns, of whole
blocks and of a few more, windows that lie outside the plane, ranges of K that begin in the middle of a tap, both layouts.  Against
64-bit products."""
import pytest

pytestmark = pytest.mark.gpu

# (B, C, H, W, F, k, stride, pad)
CASES = [(2, 1, 9, 7, 5, 3, 1, 1), (1, 6, 31, 23, 70, 5, 1, 2), (3, 10, 14, 14, 130, 7, 1, 3), (2, 15, 8, 8, 33, 3, 2, 0), (2, 16, 8, 8, 33, 3, 1, 2),
         (1, 17, 12, 5, 64, 4, 3, 3), (1, 20, 7, 7, 40, 7, 1, 3), (1, 36, 7, 7, 24, 7, 1, 0), (4, 51, 6, 6, 100, 2, 2, 1), (40, 33, 20, 20, 96, 3, 1, 1),
         (1, 3, 4, 4, 8, 9, 1, 6)]


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_taps(handle, layout, case):
    import torch
    from nebula_b200 import api
    B, C, H, W, F, k, s, p = case
    g = torch.Generator(device="cuda").manual_seed(C * k)
    x, w = torch.randn(B, C, H, W, device="cuda", generator=g), torch.randn(F, C, k, k, device="cuda", generator=g)
    b = torch.randn(F, device="cuda", generator=g)
    handle.set_math("fp32")
    plan = api.Conv2d(handle, B, C, H, W, F, k, s, p, False, "linear", api.LAYOUT_NHWC if layout == "nhwc" else api.LAYOUT_NCHW)
    plan.set_weights(w, b)
    y = plan.forward(x.permute(0, 2, 3, 1).contiguous() if layout == "nhwc" else x)
    handle.synchronize()
    plan.close()
    y = y.permute(0, 3, 1, 2) if layout == "nhwc" else y

    def conv(x, w):
        cols = torch.nn.functional.unfold(x.double(), k, padding=p, stride=s)
        return torch.matmul(w.double().reshape(F, -1), cols).reshape(y.shape)
    want, size = conv(x, w) + b.double().reshape(1, -1, 1, 1), conv(x.abs(), w.abs()) + b.double().abs().reshape(1, -1, 1, 1)
    # every addition rounds by 2^-24 of a partial sum, which the sum of the absolute products bounds
    assert bool(((y.double() - want).abs() <= (C * k * k + 2) * 2.0 ** -24 * size).all())
