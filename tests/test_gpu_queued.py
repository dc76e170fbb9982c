"""Calls and passes queued behind one another, each on new inputs: every one must give what it gives when it is waited for."""
import numpy as np
import pytest

from tests.util import assert_close

pytestmark = pytest.mark.gpu


# (B, C, H, W, F, k, stride, pad): the in-kernel gather with one K block, a full ring, a second pass through it, the largest
# table it holds; one tile and more tiles than SMs; 64- and 128-wide tiles
GATHER_CASES = [(1, 5, 9, 9, 16, 1, 1, 0), (8, 30, 33, 33, 64, 3, 1, 1), (2, 7, 20, 20, 40, 7, 2, 3), (4, 15, 64, 64, 96, 5, 1, 2),
                (8, 28, 57, 57, 128, 3, 1, 1)]


@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("case", GATHER_CASES, ids=str)
def test_gathered_convolutions(handle, mode, layout, case):
    import torch
    from nebula_b200 import api
    from oracle import oracle as O
    B, C, H, W, F, k, s, p = case
    g = torch.Generator(device="cuda").manual_seed(3)
    handle.set_math(mode)
    plan = api.Conv2d(handle, B, C, H, W, F, k, s, p, False, "relu", api.LAYOUT_NCHW if layout == "nchw" else api.LAYOUT_NHWC)
    w = torch.randn(F, C, k, k, device="cuda", generator=g) * (2.0 / (C * k * k)) ** 0.5
    bias = torch.randn(F, device="cuda", generator=g) * 0.1
    plan.set_weights(w, bias)
    shape = (B, C, H, W) if layout == "nchw" else (B, H, W, C)
    xs = [torch.randn(shape, device="cuda", generator=g) for _ in range(6)]
    torch.cuda.synchronize()
    queued = [plan.forward(x) for x in xs]
    handle.synchronize()
    for x, y in zip(xs, queued):
        alone = plan.forward(x)
        handle.synchronize()
        assert torch.equal(alone, y)
    nchw = (lambda t: t) if layout == "nchw" else (lambda t: t.permute(0, 3, 1, 2))
    ref = O.conv_forward(np.ascontiguousarray(nchw(xs[-1]).cpu().numpy()), w.cpu().numpy(), bias.cpu().numpy(), k, s, p, "relu", None)
    assert_close(nchw(queued[-1]).cpu().numpy(), ref, mode, f"gathered conv {case}")
    plan.close()


@pytest.mark.parametrize("mode", ["tf32", "tf32x3", "fp32"])
@pytest.mark.parametrize("name", ["toy_convnet", "tiny_resnet", "mid_vgg", "tiny_lstm", "dbn", "rnn"])
def test_passes_on_other_inputs(handle, name, mode):
    """Passes of a network queued on three inputs in turn, the last one read: a pass that left an earlier one's output would show."""
    import torch
    from nebula_b200 import api, workloads
    from tests import nets
    wl = (workloads.dbn(batch=5, height=32, width=32) if name == "dbn" else
          workloads.rnn2(batch=9, time_steps=5, input_size=40, hidden=72, classes=50) if name == "rnn" else getattr(nets, name)(3))
    handle.set_math(mode)
    net = api.Network(handle, wl.cfg)
    net.load_weights(wl.make_weights(11))
    xs = [torch.from_numpy(wl.make_input(s)).cuda() for s in (1, 2, 3)]
    alone = []
    for x in xs:
        net.forward(x)
        handle.synchronize()
        alone.append(net.logits().copy())
    for last in range(3):
        for k in range(6):
            net.forward(xs[(last + k + 1) % 3])
        handle.synchronize()
        assert (net.logits() == alone[last]).all()
    net.close()
