"""The one-kernel recurrence on a cluster (LSTM and RNN), at widths around its tiles and cluster sizes, batches around its
row groups, one and more steps, against the CPU oracle; and a batch against its slices, bit for bit."""
import numpy as np
import pytest

from tests.util import assert_close

pytestmark = pytest.mark.gpu


def _plan(handle, kind, T, B, inp, H, bn, act, w):
    from nebula_b200 import api
    plan = (api.Lstm if kind == "lstm" else api.Rnn)(handle, T, B, inp, H, bn, act)
    plan.set_weights(w)
    return plan


# (kind, T, B, inputs, H, batch-norm, activation)
CASES = [("lstm", 1, 3, 12, 8, False, "linear"), ("lstm", 4, 1, 5, 1, False, "linear"), ("lstm", 5, 9, 40, 33, True, "linear"),
         ("lstm", 3, 20, 64, 300, False, "linear"), ("lstm", 3, 33, 32, 101, False, "tanh"), ("lstm", 2, 100, 36, 420, False, "linear"),
         ("lstm", 6, 2, 64, 64, True, "leaky"), ("rnn", 1, 4, 33, 7, False, "tanh"), ("rnn", 5, 32, 64, 256, False, "tanh"),
         ("rnn", 4, 70, 40, 36, True, "relu"), ("rnn", 3, 5, 64, 500, False, "logistic"), ("rnn", 6, 17, 35, 129, True, "leaky")]


@pytest.mark.parametrize("mode", ["fp32", "tf32", "tf32x3"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_recurrence_on_a_cluster(handle, mode, case):
    import torch
    from nebula_b200.workloads import NetBuilder
    from oracle import oracle as O
    kind, T, B, inp, H, bn, act = case
    b = NetBuilder("r", B, input_size=inp, time_steps=T, bias_init="bias_n01")
    getattr(b, kind)(H, act, bn=bn, bound=1.0 / np.sqrt(H + inp))
    wl = b.build("normal")
    w, x = wl.make_weights(H + T), wl.make_input(B)
    ref = O.forward_network(wl.cfg, w, x)[0]
    handle.set_math(mode)
    plan = _plan(handle, kind, T, B, inp, H, bn, act, w)
    xd = torch.from_numpy(x).cuda()
    out = plan.forward(xd)
    assert_close(out.cpu().numpy(), ref, mode, f"{case}", factor=3.0 if act in ("tanh", "logistic") else 1.0)
    if mode == "fp32" and B > 1:            # the last rows alone
        n = max(1, B // 3)
        part = _plan(handle, kind, T, n, inp, H, bn, act, w)
        assert torch.equal(part.forward(xd[:, B - n:].contiguous()), out[:, B - n:])
        part.close()
    handle.synchronize()
    plan.close()
