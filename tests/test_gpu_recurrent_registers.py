"""The one-kernel recurrence with its weights in registers, at the edges: one column block and all twelve, widths that leave CTAs
of a cluster or rows of a warp without units, every number of batch rows per cluster and ragged ones, one step and many (the
barriers' phases), each activation route, in the mode whose sums are exact fp32, against the CPU oracle."""
import numpy as np
import pytest

from tests.util import assert_close

pytestmark = pytest.mark.gpu

# (kind, T, B, H, batch-norm, activation)
CASES = [("lstm", 9, 1, 33, False, "linear"), ("lstm", 2, 2, 3, False, "linear"), ("lstm", 7, 3, 304, True, "linear"), ("lstm", 4, 21, 161, False, "linear"),
         ("lstm", 3, 55, 97, False, "tanh"), ("lstm", 40, 4, 17, False, "linear"), ("lstm", 3, 28, 300, False, "linear"), ("rnn", 9, 1, 384, False, "relu"),
         ("rnn", 5, 2, 5, False, "tanh"), ("rnn", 33, 3, 31, True, "tanh"), ("rnn", 4, 30, 255, False, "logistic"), ("rnn", 6, 60, 130, False, "leaky"),
         ("rnn", 1, 9, 100, False, "tanh")]


@pytest.mark.parametrize("mode", ["fp32", "tf32x3"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_recurrence(handle, mode, case):
    import torch
    from nebula_b200 import api
    from nebula_b200.workloads import NetBuilder
    from oracle import oracle as O
    kind, T, B, H, bn, act = case
    b = NetBuilder("r", B, input_size=36, time_steps=T, bias_init="bias_n01")
    getattr(b, kind)(H, act, bn=bn, bound=1.0 / np.sqrt(H + 36))
    wl = b.build("normal")
    w, x = wl.make_weights(H + T), wl.make_input(B)
    ref = O.forward_network(wl.cfg, w, x)[0]
    handle.set_math(mode)
    plan = (api.Lstm if kind == "lstm" else api.Rnn)(handle, T, B, 36, H, bn, act)
    plan.set_weights(w)
    xd = torch.from_numpy(x).cuda()
    out = plan.forward(xd)
    again = plan.forward(xd)            # (queued behind it)
    handle.synchronize()
    plan.close()
    assert_close(out.cpu().numpy(), ref, mode, f"{case}", factor=3.0 if act in ("tanh", "logistic") else 1.0)
    assert torch.equal(out, again)
