"""The TF32 LSTM recurrence in one kernel (lstm_persistent.cu) at the edges of its tiles: widths off its 32-unit blocks and
with empty slices of K, batches around the MMA's 16 columns, its groups of rows and
the 128 rows of a chunk, three steps and more.  Against the CPU
oracle, and bit for bit against a launch per step, which adds the same slices of K in the same order."""
import numpy as np
import pytest

from tests.util import assert_close

pytestmark = pytest.mark.gpu

# (T, B, inputs, H)
CASES = [(3, 1, 32, 32), (3, 15, 36, 64), (4, 16, 32, 96), (3, 17, 40, 452), (5, 64, 32, 512), (3, 65, 64, 500), (3, 128, 32, 1020),
         (6, 3, 32, 1024), (3, 127, 32, 288), (3, 33, 32, 1184),
         (3, 129, 32, 512), (3, 200, 32, 576), (3, 251, 32, 64), (4, 1000, 32, 32)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_lstm_in_slices_of_k(handle, case, monkeypatch):
    import torch
    from nebula_b200 import api
    from nebula_b200.workloads import NetBuilder
    from oracle import oracle as O
    T, B, inp, H = case
    b = NetBuilder("l", B, input_size=inp, time_steps=T, bias_init="bias_n01")
    b.lstm(H, bound=1.0 / np.sqrt(H))
    wl = b.build("normal")
    w, x = wl.make_weights(H), wl.make_input(B)
    ref = O.forward_network(wl.cfg, w, x)[0]
    handle.set_math("tf32")
    plan = api.Lstm(handle, T, B, inp, H, False, "linear")
    plan.set_weights(w)
    xd = torch.from_numpy(x).cuda()
    runs = []
    for env in ("1", "0", "1"):                 # (the kernel leaves its counters ready for the next launch)
        monkeypatch.setenv("NEBULA_B200_LSTM_PERSISTENT", env)
        out, cell = plan.forward(xd, want_cell=True)
        runs.append((out.clone(), cell.clone()))
    handle.synchronize()
    plan.close()
    assert_close(runs[0][0].cpu().numpy(), ref, "tf32", f"{case}")
    for out, cell in runs[1:]:
        assert torch.equal(out, runs[0][0]) and torch.equal(cell, runs[0][1])
