"""Contractions cut along K (small convolutions, connected layers): one or two slices to sixteen, a shorter last slice, the
layers folded into the reduction, against the CPU oracle; and activations four at a time."""
import numpy as np
import pytest

from tests.util import assert_close

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


# (B, C, H, W, F, k, stride, pad, fold): 32 K blocks and more on few tiles; odd and even slice counts; C off 32
CASES = [(1, 512, 7, 7, 512, 3, 1, 1, ""), (1, 256, 14, 14, 256, 3, 2, 1, ""), (1, 1024, 7, 7, 64, 1, 1, 0, ""), (3, 128, 8, 6, 32, 3, 1, 1, "pool"),
         (2, 160, 10, 12, 100, 3, 1, 1, "pool"), (1, 132, 9, 9, 36, 3, 1, 1, "res"), (2, 256, 7, 7, 96, 3, 1, 1, "res"), (5, 2048, 3, 3, 60, 1, 1, 0, "res")]


@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_split_convolution(handle, mode, case):
    from nebula_b200 import api
    from oracle import oracle as O
    B, C, H, W, F, k, s, p, fold = case
    rng = np.random.default_rng(C + F)
    x = rng.standard_normal((B, C, H, W), dtype=np.float32)
    w = (rng.standard_normal((F, C, k, k)) * np.sqrt(2.0 / (C * k * k))).astype(np.float32)
    b = (0.1 * rng.standard_normal(F)).astype(np.float32)
    act = "linear" if fold == "res" else "leaky"
    ref = O.conv_forward(x, w, b, k, s, p, act)
    handle.set_math(mode)
    plan = api.Conv2d(handle, B, C, H, W, F, k, s, p, False, act, api.LAYOUT_NHWC)
    plan.set_weights(w, b)
    n0 = handle.launch_count()
    xd = _t(x.transpose(0, 2, 3, 1))
    if fold == "pool":
        y = plan.forward_fused(xd, pool=True)
        ref = O.pool_forward(ref, 2, 2, 0, True)
    elif fold == "res":
        rc = F // 2 // 4 * 4
        r = rng.standard_normal((B, rc, 2 * ref.shape[2], 2 * ref.shape[3]), dtype=np.float32)
        y = plan.forward_fused(xd, residual=_t(r.transpose(0, 2, 3, 1)), res_act="relu")
        ref = ref.copy()
        ref[:, :rc] += r[:, :, ::2, ::2]
        ref = np.maximum(ref, 0)
    else:
        y = plan.forward(xd)
    assert handle.launch_count() - n0 == (3 if mode == "tf32" else 2), "a copy or rounding pass, the product and its reduction"
    assert_close(y.cpu().numpy().transpose(0, 3, 1, 2), ref, mode, f"{case}")
    handle.synchronize()
    plan.close()


@pytest.mark.parametrize("mode", ["tf32", "tf32x3"])
@pytest.mark.parametrize("case", [(32, 2000, 1000, "logistic"), (1, 512, 60, "tanh"), (128, 1000, 500, "loggy"), (129, 1000, 500, "relu"), (8, 4100, 132, "leaky")],
                         ids=lambda c: "x".join(map(str, c)))
def test_split_connected(handle, mode, case):
    from nebula_b200 import api
    from oracle import oracle as O
    B, inp, out, act = case
    rng = np.random.default_rng(inp)
    x = rng.standard_normal((B, inp), dtype=np.float32)
    w = (rng.standard_normal((out, inp)) / np.sqrt(inp)).astype(np.float32)
    b = (0.1 * rng.standard_normal(out)).astype(np.float32)
    handle.set_math(mode)
    plan = api.Connected(handle, B, inp, out, False, act)
    plan.set_weights(w, b)
    y = plan.forward(_t(x)).cpu().numpy()
    handle.synchronize()
    plan.close()
    assert_close(y, O.connected_forward(x, w, b, act), mode, f"{case}", factor=3.0 if act in ("tanh", "logistic", "loggy") else 1.0)
