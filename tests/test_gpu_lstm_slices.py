"""The TF32 LSTM recurrence in one kernel (lstm_persistent.cu; lstm_wide.cu for what does not fit that) at the edges of its tiles:
widths off its 32-unit blocks and with empty slices of K, batches around the MMA's 16 columns, its groups of rows and the 128 rows
of a chunk.  Against the CPU oracle, and bit for bit against a launch per step, which adds the same slices of K in the same order."""
import numpy as np
import pytest

from tests.util import assert_close

pytestmark = pytest.mark.gpu

# (T, B, inputs, H)
CASES = [(3, 1, 32, 32), (3, 15, 36, 64), (4, 16, 32, 96), (3, 17, 40, 452), (5, 64, 32, 512), (3, 65, 64, 500), (3, 128, 32, 1020),
         (6, 3, 32, 1024), (3, 127, 32, 288), (3, 33, 32, 1184),
         (3, 129, 32, 512), (3, 200, 32, 576), (3, 251, 32, 64), (4, 1000, 32, 32),
         (3, 65, 32, 1056), (5, 128, 32, 1056), (6, 1, 32, 1088), (9, 64, 64, 1088), (3, 100, 32, 1152), (12, 128, 32, 1184), (3, 20, 32, 1216),
         (2, 64, 32, 256), (2, 128, 32, 1056), (2, 65, 32, 416), (2, 20, 32, 1184)]
# launches fewer than a launch per step: step 0 is a kernel of its own in front of lstm_wide.cu
WIDE = {(3, 33, 32, 1184), (3, 65, 32, 1056), (5, 128, 32, 1056), (6, 1, 32, 1088), (9, 64, 64, 1088), (3, 100, 32, 1152), (12, 128, 32, 1184),
        (2, 64, 32, 256), (2, 128, 32, 1056), (2, 65, 32, 416)}
PER_STEP = {(3, 200, 32, 576), (3, 20, 32, 1216), (2, 20, 32, 1184)}       # (more clusters, or weights, than the device holds)


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
    runs, launches = [], []
    for env in ("1", "0", "1"):                 # (the kernel leaves its counters ready for the next launch)
        monkeypatch.setenv("NEBULA_B200_LSTM_PERSISTENT", env)
        n0 = handle.launch_count()
        out, cell = plan.forward(xd, want_cell=True)
        launches.append(handle.launch_count() - n0)
        runs.append((out.clone(), cell.clone()))
    handle.synchronize()
    plan.close()
    assert launches[1] - launches[0] == (0 if case in PER_STEP else T - 2 if case in WIDE else T - 1)
    assert_close(runs[0][0].cpu().numpy(), ref, "tf32", f"{case}")
    for out, cell in runs[1:]:
        assert torch.equal(out, runs[0][0]) and torch.equal(cell, runs[0][1])


@pytest.mark.parametrize("B", [65, 100, 128])
@pytest.mark.parametrize("H", [772, 900, 1024])
def test_slices_of_more_blocks_than_the_ring_has_slots(handle, H, B, monkeypatch):
    """65 rows and more leave six slots to a group of rows, a slice of these widths has seven or eight blocks: two copies of a step
    share a slot.  Many steps, several times, bit for bit what a launch per step gives."""
    import torch
    from nebula_b200 import api
    T = 64
    g = torch.Generator(device="cuda").manual_seed(H + B)
    handle.set_math("tf32")
    plan = api.Lstm(handle, T, B, 32, H, False, "linear")
    plan.set_weights((torch.rand(8 * H + 4 * H * H + 4 * H * 32, device="cuda", generator=g) * 2 - 1) / H ** 0.5)
    x = torch.randn(T, B, 32, device="cuda", generator=g)
    monkeypatch.setenv("NEBULA_B200_LSTM_PERSISTENT", "0")
    n0 = handle.launch_count()
    want = plan.forward(x)
    per_step = handle.launch_count() - n0
    monkeypatch.setenv("NEBULA_B200_LSTM_PERSISTENT", "1")
    n0 = handle.launch_count()
    got = [plan.forward(x) for _ in range(4)]
    assert handle.launch_count() - n0 == 4 * (per_step - T + 1), "all steps in one launch"
    handle.synchronize()
    plan.close()
    assert bool(want.abs().amax() > 0) and all(torch.equal(y, want) for y in got)


@pytest.mark.parametrize("H", [96, 500, 1024, 1056])
def test_the_width_decides_the_order_of_additions(handle, H):
    """A batch that runs a launch per step, its slices in one launch, and its first two steps by themselves: the same bits."""
    import torch
    from nebula_b200 import api
    T, B = 4, 300
    g = torch.Generator(device="cuda").manual_seed(H)
    w = (torch.rand(8 * H + 4 * H * H + 4 * H * 64, device="cuda", generator=g) * 2 - 1) / H ** 0.5
    x = torch.randn(T, B, 64, device="cuda", generator=g)
    handle.set_math("tf32")
    def run(steps, lo, hi):
        plan = api.Lstm(handle, steps, hi - lo, 64, H, False, "linear")
        plan.set_weights(w)
        y = plan.forward(x[:steps, lo:hi].contiguous())
        handle.synchronize()
        plan.close()
        return y
    want = run(T, 0, B)
    assert torch.equal(want, torch.cat([run(T, lo, hi) for lo, hi in ((0, 1), (1, 65), (65, 170), (170, 300))], 1))
    assert torch.equal(want[:2, :64], run(2, 0, 64))


@pytest.mark.parametrize("B,H", [(40, 768), (48, 1024), (63, 1056)])
def test_two_steps_of_fewer_rows(handle, B, H, monkeypatch):
    """From 40 rows on, two steps of wide layers are one launch behind step 0 too: bit for bit the launch per step."""
    import torch
    from nebula_b200 import api
    g = torch.Generator(device="cuda").manual_seed(H)
    handle.set_math("tf32")
    plan = api.Lstm(handle, 2, B, 32, H, False, "linear")
    plan.set_weights((torch.rand(8 * H + 4 * H * H + 4 * H * 32, device="cuda", generator=g) * 2 - 1) / H ** 0.5)
    x = torch.randn(2, B, 32, device="cuda", generator=g)
    got = []
    for env in ("0", "1"):
        monkeypatch.setenv("NEBULA_B200_LSTM_PERSISTENT", env)
        got.append(plan.forward(x))
    handle.synchronize()
    plan.close()
    assert bool(got[0].abs().amax() > 0) and torch.equal(got[0], got[1])
