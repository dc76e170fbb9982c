"""Stand-alone shortcuts of any extents with every activation: relu, leaky and linear are a kernel of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# the sum is one fp32 addition on either side; the double formulas may round to a neighbour
ACTS = ["linear", "relu", "leaky", "relie", "logistic", "loggy", "tanh", "elu", "hardtan", "lhtan", "plse", "ramp", "stair"]


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("act", ACTS)
def test_shortcut_activation(handle, layout, act):
    import torch
    from nebula_b200 import api
    g = torch.Generator(device="cuda").manual_seed(1)
    prev, conn = torch.randn(2, 7, 5, 5, device="cuda", generator=g) * 3, torch.randn(2, 6, 10, 10, device="cuda", generator=g) * 3
    prev[0, 0, 0, :4] = torch.tensor([float("nan"), float("inf"), -float("inf"), -0.0])
    v = prev.clone()
    v[:, :6] += conn[:, :, ::2, ::2]
    want = handle.activation(v.clone(), act)
    nhwc = layout == "nhwc"
    a, b = (t.permute(0, 2, 3, 1).contiguous() if nhwc else t for t in (prev, conn))
    y = handle.shortcut(a, b, act, api.LAYOUT_NHWC if nhwc else api.LAYOUT_NCHW)
    y = y.permute(0, 3, 1, 2) if nhwc else y
    assert np.array_equal(y.cpu().numpy(), want.cpu().numpy(), equal_nan=True)
